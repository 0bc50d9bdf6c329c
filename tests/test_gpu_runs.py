"""ldg_sync_runs at the ends of its tiles and chunks, against numpy: runs that
start, end or cross there, arrays that start between 16-byte boundaries, the
shortest arrays and more tiles than chunks."""
import ctypes

import numpy as np
import pytest

from ldgpu import lib as L
from ldgpu.lib import LDG_ERR_RANGE

pytestmark = pytest.mark.gpu

TILE, CHUNKS = 2048, 148 * 8
THR = 0.1 + 1e-12  # between two float32 values


def _signal(kind, n, rng):
    edge = np.float32(THR)
    edge = edge if float(edge) <= THR else np.nextafter(edge, np.float32(-1))  # the greatest value at or below it
    above = np.nextafter(edge, np.float32(1))
    if kind == "below":
        return np.full(n, edge, np.float32)
    if kind == "above":
        return np.full(n, above, np.float32)
    if kind == "alternate":
        return np.where(np.arange(n) % 2, above, edge).astype(np.float32)
    if kind == "noise":
        return np.where(rng.random(n) < 0.5, above, edge).astype(np.float32)
    x = rng.normal(0.5, 0.05, n).astype(np.float32)
    pos = 0
    while pos < n:  # pulses of 1 sample to several tiles
        ln = int(rng.choice([1, 3, 4, 32, 128, 190, 1084, 2048, 9000]))
        x[pos:pos + ln] = rng.normal(-0.5, 0.05, len(x[pos:pos + ln]))
        if ln > 2000 and pos + 500 < n:
            x[pos + 500] = np.nan  # a NaN is above: it splits the run
        pos += ln + int(rng.choice([1, 2, 31, 127, 700, 2048, 30000]))
    return x


def _expected(x, min_long, lo, hi):
    below = np.concatenate([[False], x.astype(np.float64) <= THR])
    d = np.diff(below.astype(np.int8))
    st, en = np.nonzero(d == 1)[0], np.nonzero(d == -1)[0]
    st = st[:len(en)]
    ln = en - st
    mean = np.full(len(st), np.nan)
    for k in np.nonzero(ln > min_long)[0]:
        seg = x[st[k] + lo:max(st[k] + ln[k] - hi, 0)]
        if len(seg):
            mean[k] = np.mean(seg, dtype=np.float64)
    return st, ln, mean


@pytest.fixture(scope="module")
def ctx(cuda_ok):
    from ldgpu import RFDecode
    rf = RFDecode(system="NTSC")
    yield rf._ctx
    rf.close()


@pytest.mark.parametrize("n", [2, 127, 129, TILE - 1, TILE, TILE + 1, 40 * TILE, CHUNKS * TILE + 1,
                               2 * CHUNKS * TILE + 5003])
@pytest.mark.parametrize("kind", ["pulses", "noise", "alternate", "below", "above"])
def test_runs_at_tile_edges(ctx, n, kind):
    import torch
    lib = L.load()
    rng = np.random.default_rng(n)
    host = _signal(kind, n, rng)
    for off, min_long in ((0, 400), (1, 400), (2, 2000), (3, -1)):
        if off and n > 40 * TILE and kind != "pulses":
            continue
        if min_long < 400 and n > 40 * TILE:
            min_long = 100
        buf = torch.full((n + off + 4,), -1.0, dtype=torch.float32, device="cuda")  # below on both sides
        buf[off:off + n] = torch.from_numpy(host)
        es, el, em = _expected(host, min_long, 40, 41)
        cap = len(es) + 1
        out = [torch.empty(cap, dtype=dt).pin_memory() for dt in (torch.int64, torch.int64, torch.float64)]
        nr = ctypes.c_int64(0)
        args = (ctx.handle, ctypes.c_void_p(buf.data_ptr() + 4 * off), n, THR, min_long, 40, 41)
        L.check(lib.ldg_sync_runs(*args, *(t.data_ptr() for t in out), cap, ctypes.byref(nr), None))
        assert nr.value == len(es)
        k = nr.value
        np.testing.assert_array_equal(out[0].numpy()[:k], es)
        np.testing.assert_array_equal(out[1].numpy()[:k], el)
        m = out[2].numpy()[:k]
        np.testing.assert_array_equal(np.isnan(m), np.isnan(em))
        # two orders of one sum of up to 9000 float64 terms below 1 in size
        np.testing.assert_allclose(m, em, rtol=0, atol=9000 * 2.0 ** -53 * 2, equal_nan=True)
        if k > 1:
            rc = lib.ldg_sync_runs(*args, *(t.data_ptr() for t in out), k - 1, ctypes.byref(nr), None)
            assert rc == LDG_ERR_RANGE and nr.value == k
