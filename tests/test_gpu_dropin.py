"""The drop-in classes (ldgpu.FieldNTSC / FieldPAL, as LDdecode.readfield
uses them) on the GPU: Field.process() runs the GPU line path on each
field's read and Field.downscale() the GPU TBC and analog audio.  Over the
seeded captures of tests/golden/fields_<case>.npz, field after field with
the reference's read offsets, the results equal the batched LineLocator's
(the same kernels over the capture-wide arrays; line locations to 1e-9
samples) and the reference's integers."""

import sys

import numpy as np
import pytest

from conftest import GOLDEN, golden

pytestmark = pytest.mark.gpu

if GOLDEN not in sys.path:
    sys.path.insert(0, GOLDEN)
from field_cases import field_case, field_case_capture  # noqa: E402


@pytest.mark.parametrize("name", ["ntsc_dropouts", "pal_8phase"])
def test_dropin_fields_equal_batched_and_reference(cuda_ok, name):
    import torch
    from ldgpu import RFDecode
    from ldgpu.audio import downscale_audio_located
    from ldgpu.field import FieldNTSC, FieldPAL
    from ldgpu.fieldread import blocks_in_capture, readlen_for
    from ldgpu.lines import LineLocator
    case = field_case(name)
    system = case[1]
    g = golden("fields_" + name)
    rf = RFDecode(system=system, decode_analog_audio=44100)
    try:
        cap, _ = field_case_capture(case, rf.blocklen, readlen_for(rf))
        nb = blocks_in_capture(rf, len(cap))
        U = rf.blocklen - rf.blockcut - rf.blockcut_end
        pb = int(round(U / rf.Filters["audio_fdiv"]))
        keys = ["demod", "demod_05", "demod_burst"] + (["demod_pilot"] if system == "PAL" else [])
        dcap = torch.from_numpy(cap).cuda()
        outs = {k: torch.empty(nb * U, dtype=torch.float32, device="cuda") for k in keys}
        outs["audio_left"] = torch.empty(nb * pb, dtype=torch.float32, device="cuda")
        outs["audio_right"] = torch.empty(nb * pb, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        rf.demod_blocks_device(dcap.data_ptr(), nb, U, {k: v.data_ptr() for k, v in outs.items()}, mtf_level=1)
        rf.synchronize()
        batched = LineLocator(rf).locate({k: outs[k] for k in keys}, nb)
        aud, offs, _, _ = downscale_audio_located(rf, batched, outs["audio_left"], outs["audio_right"], freq=44100)
        torch.cuda.synchronize()
        aud = aud.cpu().numpy()
        host = {k: v.cpu().numpy() for k, v in outs.items()}
        cls = FieldPAL if system == "PAL" else FieldNTSC
        n = int(g["nfields"])
        prev, prev_startloc = None, None
        for i in range(n):
            fl = batched[i]
            w = fl.window
            sl = slice(w.startloc, w.startloc + w.length)
            asl = slice(w.first_block * pb, (w.first_block + w.nblocks) * pb)
            video = np.rec.fromarrays([host[k][sl] for k in keys], names=keys)
            audio = np.rec.fromarrays([host["audio_left"][asl], host["audio_right"][asl]],
                                      names=["audio_left", "audio_right"])
            f = cls(rf, {"video": video, "audio": audio, "startloc": w.startloc}, prevfield=prev,
                    initphase=(i == 0), fields_written=i, readloc=w.startloc)
            f.process()
            assert f.valid
            p = f"f{i}_"
            flags = [int(f.isFirstField), f.linecount, f.lineoffset, f.fieldPhaseID]
            np.testing.assert_array_equal(flags, g[p + "flags"][:4], err_msg=f"{name} field {i}")
            assert flags == [int(fl.isFirstField), fl.linecount, fl.lineoffset, fl.fieldPhaseID]
            # the batched path takes NTSC burst phases from parallel rounds
            # seeded with values equal to the field-by-field ones to the
            # last bits, so its line locations agree to ~1e-11 samples
            np.testing.assert_allclose(np.asarray(f.linelocs), fl.host_linelocs(), rtol=0, atol=1e-9)
            np.testing.assert_array_equal(np.asarray(f.linebad, dtype=bool), fl.linebad)
            assert f.sync_confidence == fl.sync_confidence
            lfw = None if i == 0 else (i, prev_startloc)
            pic, dsaudio, _ = f.downscale(linesout=f.outlinecount, final=True, audio=44100, lastfieldwritten=lfw)
            np.testing.assert_array_equal(dsaudio, aud[offs[i]:offs[i + 1]])
            prev, prev_startloc = f, w.startloc
            print(name, i, "ok", f.fieldPhaseID)
    finally:
        rf.close()


@pytest.mark.parametrize("form", ["records", "view", "dict", "mixed", "read-only"])
def test_video_columns_cross_as_they_are(cuda_ok, form):
    """A field read's video reaches the device column by column whatever
    holds it: records of float32 fields (one copy), a strided part of them,
    arrays by name, records with other types, records that may not be written."""
    import torch
    from ldgpu.lines import device_columns
    names = ["demod", "demod_raw", "demod_05", "demod_burst", "demod_pilot"]
    rng = np.random.default_rng(1)
    cols = {k: rng.normal(size=1003).astype(np.float32) for k in names}
    v = cols
    if form in ("records", "view", "read-only"):
        v = np.rec.fromarrays([cols[k] for k in names], names=names)
    if form == "view":
        v, cols = v[::2], {k: a[::2] for k, a in cols.items()}
    if form == "read-only":
        v.flags.writeable = False
    if form == "mixed":
        v = np.rec.fromarrays([cols[k] for k in names] + [np.arange(1003, dtype=np.float64)], names=names + ["t"])
    for keys in (("demod", "demod_05", "demod_burst"), ("demod_pilot",)):
        got = device_columns(v, keys, torch.device("cuda"))
        for k in keys:
            np.testing.assert_array_equal(got[k].cpu().numpy(), cols[k])
            assert got[k].is_contiguous() and got[k].dtype == torch.float32


@pytest.mark.parametrize("system", ["NTSC", "PAL"])
def test_field_on_a_side_stream_equals_default(cuda_ok, system):
    """A field's calls inside torch.cuda.stream(s), with s and the default
    stream busy as each begins: the results of the default stream alone, and
    the same for a second field's data in the memory the first one left."""
    import torch
    from ldgpu import RFDecode
    from ldgpu.field import FieldNTSC, FieldPAL
    from ldgpu.fieldread import field_window
    from ldgpu.synth import inject_dropouts, synth_capture
    rf = RFDecode(system=system, decode_analog_audio=44100)
    U = rf.blocklen - rf.blockcut - rf.blockcut_end
    w = field_window(rf, 0.0)
    keys = ["demod", "demod_raw", "demod_05", "demod_burst"] + (["demod_pilot"] if system == "PAL" else [])
    reads = []
    for seed in (11, 12):
        frame = 1_334_666 if system == "NTSC" else 1_600_000
        cap = synth_capture(system, (w.nblocks - 1) * U + rf.blocklen, seed=seed, start=frame - 30_000 - 911 * seed).numpy()
        inject_dropouts(cap, seed, 6)
        dcap = torch.from_numpy(cap).cuda()
        outs = {k: torch.empty(w.nblocks * U, dtype=torch.float32, device="cuda") for k in keys + ["rfhpf"]}
        torch.cuda.synchronize()
        rf.demod_blocks_device(dcap.data_ptr(), w.nblocks, U, {k: v.data_ptr() for k, v in outs.items()}, mtf_level=1)
        rf.synchronize()
        host = {k: v.cpu().numpy() for k, v in outs.items()}
        reads.append({"video": np.rec.fromarrays([host[k] for k in keys], names=keys), "rfhpf": host["rfhpf"],
                      "input": cap[rf.blockcut:rf.blockcut + w.length], "startloc": w.startloc})
    cls = FieldPAL if system == "PAL" else FieldNTSC

    def decode(read, before):
        f = cls(rf, read, initphase=True, readloc=w.readloc)
        before()
        f.process()
        assert f.valid
        before()
        pic = f.downscale(linesout=f.outlinecount, final=True)[0]
        before()
        drops = f.dropout_detect()
        before()
        return [np.asarray(f.linelocs), np.asarray(f.linebad), [f.isFirstField, f.fieldPhaseID, f.linecount], pic,
                *map(np.asarray, drops), f.rf_tbc()]

    def busy():
        torch.cuda._sleep(4_000_000)  # a few ms of this stream
        with torch.cuda.stream(torch.cuda.default_stream()):
            torch.cuda._sleep(8_000_000)

    want = [decode(r, lambda: None) for r in reads]
    assert len(want[0][4]) > 0
    with torch.cuda.stream(torch.cuda.Stream()):
        got = [decode(r, busy) for r in reads]
    torch.cuda.synchronize()
    for a, b in zip(want, got):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)
    rf.close()
