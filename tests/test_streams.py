"""Order between torch's streams and the library's in the drop-in calls, on
the CPU: the streams are stand-ins that log what is asked of them."""
import numpy as np
import pytest


class _Stream:
    cuda_stream = 0x5150

    def __init__(self, log):
        self.log = log

    def synchronize(self):
        self.log.append("wait")


@pytest.fixture
def log(monkeypatch):
    import torch
    log = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: _Stream(log))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    return log


def test_columns_split_before_they_are_returned(log):
    """Records are taken apart by kernels on torch's current stream; the
    library may read the columns on another one, so they are waited for."""
    import torch
    from ldgpu.lines import device_columns
    x = np.arange(10, dtype=np.float32)
    v = np.rec.fromarrays([x, x + 100, x + 200], names=["demod", "demod_raw", "demod_05"])
    got = device_columns(v, ("demod", "demod_05"), torch.device("cpu"))
    np.testing.assert_array_equal(got["demod_05"].numpy(), x + 200)
    assert log == ["wait"]
