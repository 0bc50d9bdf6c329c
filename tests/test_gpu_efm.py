"""Zero crossings of EFM samples on the GPU (ldg_efm_edges, through
ldgpu.efm.efm_edges) against the same test done sample by sample in numpy
(EFM_PLL.process's detector, efm_pll.py:148-151), on the seeded EFM-like
signals of tests/golden/efm_cases.py and the demodulator's own EFM output;
then the PLL run from the GPU crossings equals the PLL run from the
samples."""

import sys

import numpy as np
import pytest

from conftest import GOLDEN
from helpers import efm_crossings

pytestmark = pytest.mark.gpu

if GOLDEN not in sys.path:
    sys.path.insert(0, GOLDEN)
from efm_cases import EFM_CASES, efm_case  # noqa: E402


@pytest.mark.parametrize("name", [c[0] for c in EFM_CASES])
def test_edges_equal_numpy(cuda_ok, name):
    import torch
    from ldgpu.efm import efm_edges
    x, _ = efm_case(name)
    t = torch.from_numpy(np.ascontiguousarray(x, np.int16)).cuda()
    got = efm_edges(t)
    want = efm_crossings(x)
    assert len(got) == len(want) > 100
    assert got.tobytes() == want.tobytes()
    # a view starting at sample 1000, reading the sample before it, positions kept
    got2 = efm_edges(t[1000:], has_before=True, pos_offset=1000)
    want2 = want[want["pos"] >= 1000]
    assert got2.tobytes() == want2.tobytes()


@pytest.mark.parametrize("n", [1, 7, 8, 31, 32, 33, 4095, 4096, 4097, 4102, 5 * 4096 + 5, 2369 * 4096 - 3])
@pytest.mark.parametrize("off", [0, 1, 3, 7])
def test_edges_tile_edges(cuda_ok, n, off):
    """Lengths around the kernel's words and tiles, starts off a 16-byte
    boundary (their first tile begins before the samples), with and without
    the sample before, and more tiles than chunks."""
    import torch
    from ldgpu.efm import efm_edges
    rng = np.random.default_rng(n + off)
    x = rng.integers(-3, 3, n + off + 1).astype(np.int16)
    x[rng.random(len(x)) < 0.5] = 5
    t = torch.from_numpy(x).cuda()
    want = efm_crossings(x[off:off + n])
    assert efm_edges(t[off:off + n]).tobytes() == want.tobytes()
    if off:
        got = efm_edges(t[off:off + n], has_before=True, pos_offset=off)
        want = efm_crossings(x[:off + n])
        assert got.tobytes() == want[want["pos"] >= off].tobytes()


def test_edges_count_beyond_cap_and_empty(cuda_ok):
    import torch
    from ldgpu import lib as L
    x, _ = efm_case(EFM_CASES[0][0])
    t = torch.from_numpy(np.ascontiguousarray(x, np.int16)).cuda()
    lib = L.load()
    n = t.numel()
    scratch = torch.empty(int(lib.ldg_efm_edges_scratch_bytes(n)), dtype=torch.uint8, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    cap = 10
    out = torch.zeros(cap * 8, dtype=torch.uint8, device="cuda")
    L.check(lib.ldg_efm_edges(t.data_ptr(), n, 0, 0, out.data_ptr(), cap, count.data_ptr(), scratch.data_ptr(),
                              torch.cuda.current_stream().cuda_stream))
    want = efm_crossings(x)
    assert int(count.item()) == len(want)
    assert out.cpu().numpy().view(L.EFM_EDGE_DTYPE).tobytes() == want[:cap].tobytes()
    L.check(lib.ldg_efm_edges(t.data_ptr(), 0, 0, 0, out.data_ptr(), cap, count.data_ptr(), scratch.data_ptr(),
                              torch.cuda.current_stream().cuda_stream))
    assert int(count.item()) == 0
    with pytest.raises(L.LdgError):
        L.check(lib.ldg_efm_edges(t.data_ptr(), n, 0, 2**31 - 10, out.data_ptr(), cap, count.data_ptr(),
                                  scratch.data_ptr(), 0))


def test_pll_from_gpu_edges_of_demodulated_efm(cuda_ok):
    """The demodulator's EFM output of a seeded capture and its located
    fields: each field's EFM slice (Field.downscale's efmout) found on the
    GPU equals the one from the field's line locations, and the PLL fed the
    fields' slices of the samples and the PLL fed the GPU's crossings give
    the same T-values and state."""
    import torch
    from ldgpu import RFDecode
    from ldgpu.efm import EFM_PLL, efm_edges, field_efm_slices
    from ldgpu.fieldread import blocks_in_capture
    from ldgpu.lines import LineLocator
    from ldgpu.synth import synth_capture
    rf = RFDecode(system="NTSC", decode_digital_audio=True)
    cap = synth_capture("NTSC", 4_000_000, seed=11).numpy()
    nb = blocks_in_capture(rf, len(cap))
    U = rf.blocklen - rf.blockcut - rf.blockcut_end
    outs = {k: torch.empty(nb * U, dtype=torch.float32, device="cuda") for k in ("demod", "demod_05", "demod_burst")}
    efm = torch.empty(nb * U, dtype=torch.int16, device="cuda")
    d = torch.from_numpy(cap).cuda()
    torch.cuda.synchronize()
    rf.demod_blocks_device(d.data_ptr(), nb, U, dict({k: v.data_ptr() for k, v in outs.items()}, efm=efm.data_ptr()),
                           mtf_level=1)
    rf.synchronize()
    fields = LineLocator(rf).locate(outs, nb)
    torch.cuda.synchronize()
    assert len(fields) >= 4
    x = efm.cpu().numpy()
    edges = efm_edges(efm)
    assert edges.tobytes() == efm_crossings(x).tobytes()
    bounds, samples = field_efm_slices(fields, efm)
    bounds, samples = bounds.cpu().numpy(), samples.cpu().numpy()
    # into pinned host memory directly, for a range of the fields
    hb = torch.zeros((3, 2), dtype=torch.int64).pin_memory()
    hs = torch.zeros((3, 2), dtype=torch.int16).pin_memory()
    field_efm_slices(fields, efm, 1, 3, bounds=hb, samples=hs)
    torch.cuda.synchronize()
    assert (hb.numpy() == bounds[1:4]).all() and (hs.numpy() == samples[1:4]).all()
    a, b = EFM_PLL(), EFM_PLL()
    total = 0
    for i, fl in enumerate(fields):
        ll = fl.host_linelocs()
        lo = fl.window.startloc + int(ll[1])
        hi = fl.window.startloc + int(ll[fl.linecount + 1])
        assert (bounds[i] == [lo, hi]).all() and (samples[i] == [x[lo], x[hi - 1]]).all()
        ta = a.process(x[lo:hi])
        tb = b.process_edges(edges, lo, hi, samples[i, 0], samples[i, 1])
        np.testing.assert_array_equal(tb, ta)
        total += len(ta)
    assert total > 1000 and a.state() == b.state()
    rf.close()


@pytest.mark.parametrize("every", [1, 2, 3, 5, 6, 7, "noise", "mixed"])
def test_dense_edges(cuda_ok, every):
    """Tiles with more crossings than a thread writes for itself, among tiles
    with fewer, from any alignment of the samples; and room for some of them."""
    import ctypes

    import torch
    from ldgpu import lib as L
    from ldgpu.efm import efm_edges
    n = 3 * 4096 + 77
    rng = np.random.default_rng(1)
    if every == "noise":
        x = rng.integers(-3000, 3000, n + 9)
    elif every == "mixed":
        x = np.where(np.arange(n + 9) // 4096 % 2, (-1) ** np.arange(n + 9), 1) * rng.integers(1, 99, n + 9)
    else:
        x = (-1) ** (np.arange(n + 9) // every) * rng.integers(1, 99, n + 9)
    x = x.astype(np.int16)
    for off in (0, 1, 5, 8):
        t = torch.from_numpy(x).cuda()[off:off + n]
        want = efm_crossings(x[off:off + n])
        assert efm_edges(t).tobytes() == want.tobytes()
    # a cap within a dense tile, a buffer that starts between 8-byte boundaries
    lib, cap = L.load(), len(want) * 2 // 3
    for shift, room in ((0, cap), (4, len(want)), (4, cap)):
        buf = torch.full((8 * len(want) + 32,), 85, dtype=torch.uint8, device="cuda")
        count = torch.zeros(1, dtype=torch.int64, device="cuda")
        scratch = torch.empty(lib.ldg_efm_edges_scratch_bytes(n), dtype=torch.uint8, device="cuda")
        L.check(lib.ldg_efm_edges(t.data_ptr(), n, 0, 0, ctypes.c_void_p(buf.data_ptr() + shift), room, count.data_ptr(),
                                  scratch.data_ptr(), 1))
        got = buf.cpu().numpy().tobytes()
        assert int(count.item()) == len(want)
        assert got[shift:shift + 8 * room] == want[:room].tobytes()
        assert got[:shift] == b"U" * shift and set(got[shift + 8 * room:]) == {85}


def test_noise_takes_no_longer_than_a_pass_and_its_edges(cuda_ok):
    """20 M samples of alternating sign against samples of one sign: the 8
    bytes of every crossing (160 MB) beside the 40 MB of samples, and not
    scattered stores (76 against 28 us; 280 by each thread its own word's)."""
    import torch
    from ldgpu import lib as L
    lib, n = L.load(), 20_000_000
    edges = torch.empty(8 * n + 64, dtype=torch.uint8, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    scratch = torch.empty(lib.ldg_efm_edges_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    took = []
    for noisy in (False, True):
        x = torch.full((n,), 5, dtype=torch.int16, device="cuda")
        if noisy:
            x[::2] = -5
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            L.check(lib.ldg_efm_edges(x.data_ptr(), n, 0, 0, edges.data_ptr(), n, count.data_ptr(), scratch.data_ptr(), 1))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        took.append(float(np.median(times)))
    assert int(count.item()) == n and took[1] < 6 * took[0], took
