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


@pytest.fixture
def on_cpu(log, monkeypatch):
    """Uploads that stay on the CPU (no device here)."""
    import torch
    empty = torch.empty
    monkeypatch.setattr(torch.Tensor, "to", lambda self, *a, **k: self)
    monkeypatch.setattr(torch, "empty", lambda *a, device=None, **k: empty(*a, **k))
    return log


def test_dropouts_run_where_their_results_are_read(on_cpu, monkeypatch):
    from ldgpu import dropouts
    got = []
    monkeypatch.setattr(dropouts, "run", lambda rf, descs, stream=None, **kw: got.append((stream, kw)) or ["out"])
    x = np.zeros(10, np.float32)
    data = {"video": {k: x for k in ("demod", "demod_05", "demod_raw")}, "rfhpf": x}
    for kw in ({}, {"out_cap": 7}, {"stream": 5}):
        assert dropouts.detect_host_field(None, data, np.arange(4.0), 0, 2, True, 5, **kw) == "out"
    assert got == [(0x5150, {}), (0x5150, {"out_cap": 7}), (5, {})]


def test_rf_tbc_runs_where_its_output_is_read(on_cpu, monkeypatch):
    from ldgpu import field, rftbc
    from ldgpu.rfdecode import RFParams
    rf = RFParams(system="NTSC")
    got = []
    monkeypatch.setattr(rftbc, "run", lambda rf, descs, stream=None: got.append(stream))
    monkeypatch.setattr(field, "tbc_status", lambda rf: None)
    rftbc.rf_tbc_host_field(rf, np.zeros(100, np.int16), np.arange(4.0), 0, 1, 0.0)
    assert got == [0x5150]


def test_process_field_scans_and_refines_on_the_callers_stream(on_cpu, monkeypatch):
    import torch
    from types import SimpleNamespace
    from ldgpu import lib as L
    from ldgpu import lines
    from ldgpu.rfdecode import RFParams

    class Seen(Exception):
        pass

    got = []
    loc = lines.LineLocator.__new__(lines.LineLocator)
    loc.torch, loc.rf, loc.pal, loc.proclines = torch, RFParams(system="NTSC"), False, 273
    loc._rbuf, loc._nruns = None, 0
    loc.sync_runs = lambda ptr, n, stream=None: got.append(stream)
    plan = np.zeros(1, lines.PLAN_DTYPE)
    plan["valid"] = 1
    monkeypatch.setattr(lines, "run_chain", lambda *a, **k: (plan.view(np.recarray), L.LDG_CHAIN_STOP_END, None))

    def refine(arrays, n, plans, pam, stream, **kw):
        got.append(stream)
        raise Seen

    loc._refine = refine
    x = np.zeros(100_000, np.float32)
    f = SimpleNamespace(data={"video": {k: x for k in ("demod", "demod_05", "demod_burst")}, "startloc": 0},
                        prevfield=None, fields_written=0)
    with pytest.raises(Seen):
        loc.process_field(f)
    assert got == [0x5150, 0x5150]


@pytest.mark.parametrize("offsets", [(0, 4), (4, 0), (0, 0), (4, 4), (0, 2), (0, 3)])
def test_columns_are_found_by_their_offset(log, offsets):
    """Records whose fields share bytes, or lie off a multiple of four."""
    import torch
    from ldgpu.lines import device_columns
    dt = np.dtype({"names": ["demod", "demod_05"], "formats": [np.float32] * 2, "offsets": offsets, "itemsize": 8})
    v = np.frombuffer(bytearray(np.arange(40, dtype=np.float32).tobytes()), dt)
    got = device_columns(v, ("demod", "demod_05"), torch.device("cpu"))
    for k in dt.names:
        assert got[k].numpy().tobytes() == np.ascontiguousarray(v[k]).tobytes(), k
