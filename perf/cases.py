"""The work a user of ldgpu has it do, as timed cases through the public entry points.

A decode of a LaserDisc capture runs these in order: `.lds` unpack, RF
demodulation (block by block from host buffers, or whole captures on the
device), line locations, time-base correction, analog audio, and beside them
dropout detection, the RF TBC, the EFM zero crossings and the AC3-RF front
end.  Most cases are one of these through its own call; `decode` and `mixed`
are whole calls, and `field` is the per-field drop-in form the decoder's
field loop uses.  Sizes are those of the benchmark and the tests: 40 MSPS
captures of a few blocks to 10 s, single fields to ten-second batches, NTSC
and PAL.

The demodulator's two FFT decompositions are both used: the library's
default ("stockham", what a plain `demodblock` runs) and the one its
autotuner picks for batches on B200 ("in_place").
"""

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ld-decode_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

FS = 40_000_000
FFT = {"stockham": 0, "in_place": 1}
FLOATS = ("demod", "demod_raw", "demod_05", "demod_burst", "demod_pilot", "rfhpf")


def listed():
    return [
        # the decoder's block cache: one block per call, numpy in and out, every output
        {"name": "demodblock_ntsc", "kind": "demodblock", "system": "NTSC", "dtype": "int16", "mtf": 1.0,
         "fft": "stockham"},
        # the read of one PAL field (31 blocks), device buffers, float32 input of a resampled capture
        {"name": "demod_pal_read", "kind": "demod", "system": "PAL", "blocks": 31, "dtype": "float32",
         "digital": True, "fft": "stockham"},
        # a 10 s NTSC capture, every output: the benchmark's demodulation
        {"name": "demod_ntsc_10s", "kind": "demod", "system": "NTSC", "blocks": 12613, "dtype": "int16",
         "digital": True, "fft": "in_place"},
        # a second and a half of NTSC from packed .lds bytes to pictures, audio and EFM crossings
        {"name": "decode_ntsc", "kind": "decode", "system": "NTSC", "samples": 60_000_000, "fft": "in_place"},
        # captures of both systems and uneven length in one work-queue batch
        {"name": "mixed", "kind": "mixed", "captures": 4, "samples": 10_000_000},
        # one field through the drop-in class: process, downscale, dropout_detect, rf_tbc
        {"name": "field_ntsc", "kind": "field", "system": "NTSC", "snr": 38.0},
        # the TBC of a second of PAL fields, and of one NTSC frame with spline wow and level smoothing
        {"name": "tbc_pal_50", "kind": "tbc", "system": "PAL", "fields": 50, "wow": "linear", "smoothing": 0.0},
        {"name": "tbc_ntsc_spline", "kind": "tbc", "system": "NTSC", "fields": 60, "wow": "cubic", "smoothing": 2.0},
        # side outputs of a second of fields
        {"name": "dropouts_ntsc_60", "kind": "dropouts", "system": "NTSC", "fields": 60},
        {"name": "rftbc_pal_50", "kind": "rftbc", "system": "PAL", "fields": 50},
        # the EFM crossings of two seconds, and two seconds of AC3-RF to baseband
        {"name": "efm_2s", "kind": "efm", "samples": 80_000_000},
        {"name": "ac3_2s", "kind": "ac3", "samples": 80_000_000, "dtype": "int16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("demodblock", "demod", "demod", "decode", "mixed", "field", "tbc", "tbc", "dropouts", "rftbc",
                       "efm", "ac3"))
    system = rng.choice(("NTSC", "PAL"))
    fft = rng.choice(("stockham", "in_place"))
    if kind == "demodblock":
        return {"kind": kind, "system": system, "dtype": rng.choice(("int16", "float32")),
                "mtf": round(rng.uniform(0.0, 1.2), 3), "fft": fft}
    if kind == "demod":
        return {"kind": kind, "system": system, "blocks": _log(rng, 1, 9000), "dtype": rng.choice(("int16", "float32")),
                "digital": rng.random() < 0.7, "fft": fft}
    if kind == "decode":
        return {"kind": kind, "system": system, "samples": _log(rng, 5_000_000, 60_000_000) | 1, "fft": fft}
    if kind == "mixed":
        return {"kind": kind, "captures": rng.randint(2, 4), "samples": _log(rng, 4_000_000, 10_000_000)}
    if kind == "field":
        return {"kind": kind, "system": system, "snr": round(rng.uniform(32.0, 46.0), 2)}
    if kind == "tbc":
        return {"kind": kind, "system": system, "fields": _log(rng, 1, 120),
                "wow": rng.choice(("linear", "linear", "quadratic", "cubic")), "smoothing": rng.choice((0.0, 0.0, 2.0))}
    if kind in ("dropouts", "rftbc"):
        return {"kind": kind, "system": system, "fields": _log(rng, 1, 120)}
    if kind == "efm":
        return {"kind": kind, "samples": _log(rng, 500_000, 80_000_000) | 1}
    return {"kind": kind, "samples": _log(rng, 500_000, 80_000_000) | 1, "dtype": rng.choice(("int16", "float32"))}


# ---- handles a program keeps over many captures

_RF = {}
_LOC = {}


def _rf(system, fft="stockham", digital=True):
    """One RFDecode per configuration (filters designed and uploaded, sinc
    table loaded by its first field), kept like a decoder keeps it."""
    key = (system, fft, digital)
    if key not in _RF:
        from ldgpu import RFDecode
        _RF[key] = RFDecode(system=system, decode_analog_audio=44100, decode_digital_audio=digital,
                            fft_variant=FFT[fft])
    return _RF[key]


def _locator(rf):
    from ldgpu.lines import LineLocator
    if id(rf) not in _LOC:
        _LOC[id(rf)] = LineLocator(rf)
    return _LOC[id(rf)]


def _params(system):
    from ldgpu.rfdecode import RFParams
    key = ("params", system)
    if key not in _RF:
        _RF[key] = RFParams(system=system, decode_analog_audio=44100, decode_digital_audio=True)
    return _RF[key]


def _stride(rf):
    return rf.blocklen - rf.blockcut - rf.blockcut_end


# ---- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _capture(system, n, seed, snr=38.0):
    """A seeded synthetic capture (sync, burst, bars, audio carriers, EFM,
    noise) that starts a little before a frame's vertical sync."""
    from ldgpu.synth import synth_capture
    frame = 1_334_666 if system == "NTSC" else 1_600_000
    return synth_capture(system, int(n), seed=int(seed), snr_db=snr, device="cuda",
                         start=frame - 30_000 - int(seed) * 131 % 20_000)


def _long_capture(system, n, seed, dtype):
    """A long capture for the demodulator alone: a synthetic stretch repeated, fresh noise over all of it."""
    base = _capture(system, min(n, 1 << 22), seed)
    cap = base.repeat(-(-n // base.numel()))[:n].contiguous()
    cap += torch.randint(-60, 61, (n,), generator=_gen(seed), device="cuda", dtype=torch.int16)
    return cap if dtype == "int16" else cap.to(torch.float32)


def _block_input(case, seed):
    x = _long_capture(case["system"], 32768, seed, "int16").cpu().numpy()
    return x if case["dtype"] == "int16" else x.astype(np.float32)


def _demod_input(case, rf, seed):
    return _long_capture(case["system"], (case["blocks"] - 1) * _stride(rf) + rf.blocklen, seed, case["dtype"])


def _pack_lds(cap):
    """A capture as 10-bit samples, packed four to five bytes (most significant bits first)."""
    v = ((cap.to(torch.int32) >> 6) + 512).clamp_(0, 1023)
    v = torch.nn.functional.pad(v, (0, -cap.numel() % 4)).view(-1, 4)
    a, b, c, d = v.unbind(1)
    q = torch.stack((a >> 2, ((a & 3) << 6) | (b >> 4), ((b & 15) << 4) | (c >> 6), ((c & 63) << 2) | (d >> 8), d & 255), 1)
    return q.to(torch.uint8).reshape(-1)


def _alloc(rf, nblocks, digital=True):
    U = _stride(rf)
    keys = ["demod", "demod_raw", "demod_05", "demod_burst"] + (["demod_pilot"] if rf.system == "PAL" else []) + ["rfhpf"]
    o = {k: torch.empty(nblocks * U, dtype=torch.float32, device="cuda") for k in keys}
    if digital:
        o["efm"] = torch.empty(nblocks * U, dtype=torch.int16, device="cuda")
    per = rf.output_slices(True)["audio"][1]
    for k in ("audio_left", "audio_right"):
        o[k] = torch.empty(nblocks * per, dtype=torch.float32, device="cuda")
    return o


def _ptrs(o):
    return {k: v.data_ptr() for k, v in o.items()}


def _geometry(rf):
    outw = rf.SysParams["outlinelen"]
    outl = rf.SysParams["frame_lines"] // 2 + 1
    nlines = outl + 10 + (3 if rf.system == "PAL" else 0)
    return outw, outl, nlines


def _lines(rf, nfields, seed, wow_amp=0.6):
    """Line locations of `nfields` field reads (FP64, field-local): the line
    grid with a slow speed error (wow_amp samples), jitter and a few moved lines."""
    _, _, nlines = _geometry(rf)
    rng = np.random.default_rng(int(seed) * 31 + 5)
    true = rf.SysParams["line_period"] * rf.freq
    i = np.arange(nlines)
    out = np.empty((nfields, nlines))
    for f in range(nfields):
        wow = wow_amp * np.sin(2 * np.pi * (i / rng.uniform(90, 400) + rng.random()))
        ll = 3000.0 + i * true + wow + rng.normal(size=nlines) * 0.02
        if wow_amp:
            ll[rng.integers(20, nlines - 2, 2)] += rng.choice((-3.0, 3.0))
        out[f] = ll
    return out


def _baseband(rf, n, seed, nfields):
    """Demodulated video (Hz) of `nfields` reads of n samples: the synthetic raster with noise."""
    from ldgpu.synth import _System, composite_ire
    ire = composite_ire(_System(rf.system), torch.arange(n, device="cuda") - 3000)  # line 0 at sample 3000, as _lines
    hz = (rf.DecoderParams["ire0"] + rf.DecoderParams["hz_ire"] * ire).to(torch.float32)
    noise = torch.randn((nfields, n), generator=_gen(seed), device="cuda")
    return noise.mul_(15e3).add_(hz)


def _read_len(rf):
    from ldgpu.fieldread import field_window
    return field_window(rf, 0.0).length


# ---- prepare

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prep_demodblock(case, seed):
    return {"case": case, "rf": _rf(case["system"], case["fft"]), "x": _block_input(case, seed)}


def _prep_demod(case, seed):
    rf = _rf(case["system"], case["fft"], case["digital"])
    cap = _demod_input(case, rf, seed)
    outs = _alloc(rf, case["blocks"], case["digital"])
    return {"case": case, "rf": rf, "cap": cap, "outs": outs, "ptrs": _ptrs(outs),
            "kind": 0 if case["dtype"] == "int16" else 1, "stream": torch.cuda.current_stream().cuda_stream or 1}


def _prep_decode(case, seed):
    from ldgpu.fieldread import blocks_in_capture
    rf = _rf(case["system"], case["fft"])
    n = case["samples"]
    packed = _pack_lds(_capture(case["system"], n, seed))
    nb = blocks_in_capture(rf, n)
    outw, outl, _ = _geometry(rf)
    most = int(n / (rf.freq_hz / rf.SysParams["FPS"] / 2)) + 4
    return {"case": case, "rf": rf, "loc": _locator(rf), "packed": packed, "n": n, "nb": nb, "outs": _alloc(rf, nb),
            "cap": torch.empty(n + (n & 1), dtype=torch.int16, device="cuda"),
            "pics": torch.zeros((most, outw * outl), dtype=torch.int16, device="cuda"),
            "audio": torch.zeros((most, 2048), dtype=torch.int16, device="cuda"), **_edge_buffers(nb * _stride(rf)),
            "stream": torch.cuda.current_stream().cuda_stream or 1}


def _prep_mixed(case, seed):
    from ldgpu.batch import MixedBatch
    caps = []
    for i in range(case["captures"]):
        system = ("NTSC", "PAL")[i % 2]
        caps.append((system, _capture(system, case["samples"] * (3 + 2 * i) // 9 + 2_500_000, seed * 10 + i)))
    if "mixed" not in _RF:
        _RF["mixed"] = [{s: _new_rf(s) for s in ("NTSC", "PAL")} for _ in range(2)]
    mb = MixedBatch(caps, rfs={s: _rf(s) for s in ("NTSC", "PAL")}, locate_threads=2, locate_rfs=_RF["mixed"])
    return {"case": case, "mb": mb}


def _new_rf(system):
    from ldgpu import RFDecode
    return RFDecode(system=system, decode_analog_audio=44100, decode_digital_audio=True)


def _prep_field(case, seed):
    from ldgpu.fieldread import field_window
    rf = _rf(case["system"])
    w = field_window(rf, 0.0)
    n = (w.nblocks - 1) * _stride(rf) + rf.blocklen
    cap = _capture(case["system"], n, seed, case["snr"])
    from ldgpu.synth import inject_dropouts
    inject_dropouts(cap, int(seed), 6)
    outs = _alloc(rf, w.nblocks)
    torch.cuda.synchronize()
    rf.demod_blocks_device(cap.data_ptr(), w.nblocks, _stride(rf), _ptrs(outs), mtf_level=1)
    rf.synchronize()
    h = {k: v.cpu().numpy() for k, v in outs.items()}
    names = [k for k in FLOATS if k in h and k != "rfhpf"]
    data = {"video": np.rec.fromarrays([h[k] for k in names], names=names), "rfhpf": h["rfhpf"], "efm": h["efm"],
            "audio": np.rec.fromarrays([h["audio_left"], h["audio_right"]], names=["audio_left", "audio_right"]),
            "input": cap[rf.blockcut:rf.blockcut + w.length].cpu().numpy(), "startloc": w.startloc}
    return {"case": case, "rf": rf, "data": data, "readloc": w.readloc}


def _prep_tbc(case, seed):
    from ldgpu import lib as L
    from ldgpu.field import tbc_descriptor
    from ldgpu.lines import field_levels
    rf = _rf(case["system"])
    nf, n = case["fields"], _read_len(rf)
    outw, outl, nlines = _geometry(rf)
    buf = _baseband(rf, n, seed, nf)
    ll = torch.from_numpy(_lines(rf, nf, seed)).cuda()
    f32 = torch.zeros((nf, outw * outl), dtype=torch.float32, device="cuda")
    u16 = torch.zeros((nf, outw * outl), dtype=torch.int16, device="cuda")
    descs = [tbc_descriptor(rf, buf[i].data_ptr(), ll[i].data_ptr(), _offset(rf, i), outw, outl, outl,
                            field_levels(rf), out_u16=u16[i].data_ptr(), out_f32=f32[i].data_ptr(), buf_len=n,
                            nlines=nlines, wow_smoothing=case["smoothing"], wow_interpolation_method=case["wow"])
             for i in range(nf)]
    return {"case": case, "rf": rf, "buf": buf, "ll": ll, "f32": f32, "u16": u16, "descs": (L.TbcField * nf)(*descs)}


def _offset(rf, i):
    return 0 if rf.system == "NTSC" else 2 + i % 2


def _dropout_input(case, rf, seed):
    """demod, demod_05, demod_raw and rfhpf of field reads, the carrier lost
    for a few microseconds four times a field."""
    nf, n = case["fields"], _read_len(rf)
    dm = _baseband(rf, n, seed, nf)
    g = _gen(seed + 1)
    raw = dm + torch.randn((nf, n), generator=g, device="cuda").mul_(8e4)
    d05 = torch.nn.functional.avg_pool1d(dm[:, None], 31, 1, 15)[:, 0].contiguous()
    hp = torch.randn((nf, n), generator=g, device="cuda").mul_(250.0).clamp_(-700.0, 700.0)
    rng = np.random.default_rng(int(seed) * 13 + 1)
    for f in range(nf):
        for s, ln in zip(rng.integers(30_000, n - 60_000, 4), rng.integers(40, 1200, 4)):
            dm[f, s:s + ln] = 3.0e6
            hp[f, s:s + ln:3] = 4000.0
    return dm, d05, raw, hp


def _prep_dropouts(case, seed):
    from ldgpu.dropouts import _field
    rf = _rf(case["system"])
    nf, n = case["fields"], _read_len(rf)
    _, outl, nlines = _geometry(rf)
    dm, d05, raw, hp = _dropout_input(case, rf, seed)
    ll = torch.from_numpy(_lines(rf, nf, seed, 0.0)).cuda()
    hsync = int((rf.SysParams["hsyncPulseUS"] + 0.7) * rf.freq)
    descs = [_field(dm[i].data_ptr(), d05[i].data_ptr(), raw[i].data_ptr(), hp[i].data_ptr(), n, ll[i].data_ptr(),
                    nlines, _offset(rf, i), outl - 1, i % 2 == 0, hsync) for i in range(nf)]
    return {"case": case, "rf": rf, "keep": (dm, d05, raw, hp, ll), "descs": descs}


def _prep_rftbc(case, seed):
    from ldgpu.rftbc import descriptor, line_samples
    rf = _rf(case["system"])
    nf, n = case["fields"], _read_len(rf)
    _, outl, nlines = _geometry(rf)
    cap = _long_capture(case["system"], nf * n, seed, "int16").view(nf, n)
    ll = torch.from_numpy(_lines(rf, nf, seed)).cuda()
    out = torch.zeros((nf, (outl - 1) * line_samples(rf)), dtype=torch.int16, device="cuda")
    descs = [descriptor(rf, cap[i].data_ptr(), n, ll[i].data_ptr(), nlines, _offset(rf, i), outl - 1,
                        out[i].data_ptr()) for i in range(nf)]
    return {"case": case, "rf": rf, "keep": (cap, ll), "out": out, "descs": descs}


def _prep_efm(case, seed):
    from ldgpu.synth import _efm_wave
    n, g = case["samples"], _gen(seed)
    m = min(n, 1 << 22)
    w = torch.nn.functional.avg_pool1d(_efm_wave(g, 0, m, torch.device("cuda"))[None, None], 13, 1, 6)[0, 0]
    x = (w * 900).to(torch.int16).repeat(-(-n // m))[:n].contiguous()
    x += torch.randint(-25, 26, (n,), generator=g, device="cuda", dtype=torch.int16)
    return {"case": case, "efm": x, **_edge_buffers(n), "stream": torch.cuda.current_stream().cuda_stream or 1}


def _edge_buffers(n):
    """Device buffers of ldg_efm_edges over n samples: crossings, their count, scratch."""
    from ldgpu import lib as L
    return {"edges": torch.zeros((n // 12 + 1024, 4), dtype=torch.int16, device="cuda"),
            "count": torch.zeros(1, dtype=torch.int64, device="cuda"),
            "scratch": torch.empty(L.load().ldg_efm_edges_scratch_bytes(n), dtype=torch.uint8, device="cuda")}


def _edges(s, efm):
    from ldgpu import lib as L
    L.check(L.load().ldg_efm_edges(efm.data_ptr(), efm.numel(), 0, 0, s["edges"].data_ptr(), s["edges"].shape[0],
                                   s["count"].data_ptr(), s["scratch"].data_ptr(), s["stream"]))


def _prep_ac3(case, seed):
    from ldgpu.ac3 import Ac3Frontend
    if "ac3" not in _RF:
        _RF["ac3"] = Ac3Frontend(float(FS))
    x = _ac3_input(case, seed)
    m = (case["samples"] + 15) // 16
    return {"case": case, "fe": _RF["ac3"], "x": x, "kind": 0 if case["dtype"] == "int16" else 1,
            "i": torch.zeros(m, dtype=torch.float32, device="cuda"), "q": torch.zeros(m, dtype=torch.float32, device="cuda"),
            "stream": torch.cuda.current_stream().cuda_stream or 1}


def _ac3_input(case, seed):
    """The 2.88 MHz QPSK carrier at 288 kbaud in noise."""
    n, g = case["samples"], _gen(seed)
    m = min(n, 1 << 23)
    t = torch.arange(m, device="cuda", dtype=torch.float64)
    sym = torch.randint(0, 4, (m // 100 + 4,), generator=g, device="cuda")
    ph = (math.pi / 2) * sym[(t * (288e3 / FS)).long()].to(torch.float64) + t * (2 * math.pi * 2.88e6 / FS)
    x = (900 * torch.cos(ph)).to(torch.int16).repeat(-(-n // m))[:n].contiguous()
    x += torch.randint(-300, 301, (n,), generator=g, device="cuda", dtype=torch.int16)
    return x if case["dtype"] == "int16" else x.to(torch.float32)


_PREPARE = {"demodblock": _prep_demodblock, "demod": _prep_demod, "decode": _prep_decode, "mixed": _prep_mixed,
            "field": _prep_field, "tbc": _prep_tbc, "dropouts": _prep_dropouts, "rftbc": _prep_rftbc,
            "efm": _prep_efm, "ac3": _prep_ac3}


# ---- run

def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_demodblock(s):
    rv = s["rf"].demodblock(data=s["x"], mtf_level=s["case"]["mtf"], cut=True)
    out = {k: rv["video"][k] for k in rv["video"].dtype.names}
    out.update({k: rv["audio"][k] for k in rv["audio"].dtype.names})
    out["rfhpf"], out["efm"] = rv["rfhpf"], rv["efm"]
    return out


def _run_demod(s):
    rf = s["rf"]
    rf.demod_blocks_device(s["cap"].data_ptr(), s["case"]["blocks"], _stride(rf), s["ptrs"], mtf_level=1,
                           in_kind=s["kind"], stream=s["stream"])
    return s["outs"]


def _run_decode(s):
    from ldgpu.audio import downscale_audio_located
    from ldgpu.efm import field_efm_slices
    from ldgpu.field import tbc_fields
    from ldgpu.ingest import unpack_lds
    from ldgpu.lines import field_levels, tbc_batch
    rf, o = s["rf"], s["outs"]
    unpack_lds(s["packed"], 0, s["n"], out=s["cap"])
    rf.demod_blocks_device(s["cap"].data_ptr(), s["nb"], _stride(rf), _ptrs(o), mtf_level=1, stream=s["stream"])
    keys = [k for k in ("demod", "demod_05", "demod_burst", "demod_pilot") if k in o]
    fields = s["loc"].locate({k: o[k] for k in keys}, s["nb"])
    tbc_fields(rf, tbc_batch(rf, fields, o["demod"].data_ptr(), s["pics"].data_ptr(), field_levels(rf)))
    downscale_audio_located(rf, fields, o["audio_left"], o["audio_right"], out=s["audio"].view(-1),
                            stride=s["audio"].shape[1])
    _edges(s, o["efm"])
    bounds, samples = field_efm_slices(fields, o["efm"])
    a = fields.arrays()
    n, most = len(fields), s["pics"].shape[0]
    return {"pictures": s["pics"], "audio": s["audio"], "edges": s["edges"], "edge_count": s["count"],
            "efm_bounds": _upto(bounds, most), "efm_samples": _upto(samples, most), "fields": n,
            "start": np.resize(a["startloc"], most), "first": np.resize(a["isfirst"], most),
            "lines": np.resize(a["linecount"], most)}


def _upto(t, n):
    return torch.nn.functional.pad(t, (0, 0, 0, n - t.shape[0]))


def _run_mixed(s):
    mb = s["mb"]
    n = mb.run()
    mb.stream.synchronize()
    return {"fields": n, "pictures": mb.pictures.view(torch.int16),
            "start": np.concatenate([f.arrays()["startloc"] for f in mb.fields])}


def _run_field(s):
    from ldgpu.field import FieldNTSC, FieldPAL
    cls = FieldPAL if s["case"]["system"] == "PAL" else FieldNTSC
    f = cls(s["rf"], s["data"], prevfield=None, initphase=True, fields_written=0, readloc=s["readloc"])
    f.process()
    pic, audio, efm = f.downscale(linesout=f.outlinecount, final=True, audio=44100)
    drops = f.dropout_detect()
    return {"lines": np.asarray(f.linelocs), "first": bool(f.isFirstField), "phase": int(f.fieldPhaseID),
            "picture": pic, "audio": _padded(audio, 2048), "efm": _padded(efm, 900_000), "rftbc": f.rf_tbc(),
            "dropouts": _padded(np.asarray(drops, np.int64), 512)}


def _padded(a, n):
    out = np.zeros(a.shape[:-1] + (n,), a.dtype)
    out[..., :a.shape[-1]] = a
    return out


def _run_tbc(s):
    from ldgpu.field import tbc_fields
    tbc_fields(s["rf"], s["descs"])
    return {"f32": s["f32"], "u16": s["u16"]}


def _run_dropouts(s):
    from ldgpu.dropouts import run as detect
    drops, std = detect(s["rf"], s["descs"], rfstd=True)
    flat = np.zeros((3, 256 * len(drops)), np.int64)
    for k in range(3):
        v = [x for d in drops for x in d[k]]
        flat[k, :len(v)] = v
    return {"count": np.array([len(d[0]) for d in drops]), "drops": flat, "std": std}


def _run_rftbc(s):
    from ldgpu.rftbc import run as resample
    resample(s["rf"], s["descs"])
    return s["out"]


def _run_efm(s):
    _edges(s, s["efm"])
    return {"edges": s["edges"], "count": s["count"]}


def _run_ac3(s):
    n = s["case"]["samples"]
    m = (n + 15) // 16
    s["fe"].run((s["x"].data_ptr(), s["kind"], n), 0, 0, m, out_i=s["i"].data_ptr(), out_q=s["q"].data_ptr(),
                stream=s["stream"])
    return s["i"], s["q"]


_RUN = {"demodblock": _run_demodblock, "demod": _run_demod, "decode": _run_decode, "mixed": _run_mixed,
        "field": _run_field, "tbc": _run_tbc, "dropouts": _run_dropouts, "rftbc": _run_rftbc, "efm": _run_efm,
        "ac3": _run_ac3}


# ---- work

def _demod_work(system, blocks, in_bytes, digital):
    """Every output of `blocks` blocks: per block one real input transform, the
    analytic signal (two half-length inverses), one real transform of the
    demodulated signal and one real inverse per output."""
    out = 31712 * (4 * (6 if system == "PAL" else 5) + (2 if digital else 0)) + 2 * 991 * 4
    transforms = (10 if system == "PAL" else 9) - (0 if digital else 1)
    fft = 5 * 16384 * 14
    return blocks * (31712 * in_bytes + out), blocks * (transforms * fft + 32768 * 60)


def _tbc_work(system, fields, f32):
    px, line, lines = (910 * 263, 2542, 263) if system == "NTSC" else (1135 * 313, 2560, 313)
    return fields * (line * lines * 4 + px * (6 if f32 else 2)), fields * px * 80


def work(case):
    k = case["kind"]
    if k == "demodblock":
        b, f = _demod_work(case["system"], 1, 2 if case["dtype"] == "int16" else 4, True)
    elif k == "demod":
        b, f = _demod_work(case["system"], case["blocks"], 2 if case["dtype"] == "int16" else 4, case["digital"])
    elif k in ("decode", "mixed"):
        if k == "decode":
            parts = [(case["system"], case["samples"], 1.25)]
        else:
            parts = [(("NTSC", "PAL")[i % 2], case["samples"] * (3 + 2 * i) // 9 + 2_500_000, 2)
                     for i in range(case["captures"])]
        b = f = 0
        for system, n, nbytes in parts:
            db, df = _demod_work(system, max(1, n // 31712), 2, True)
            tb, tf = _tbc_work(system, max(1, n // (667_334 if system == "NTSC" else 800_000)), False)
            b, f = b + n * nbytes + db + tb, f + df + tf
    elif k == "field":
        n = 29 * 31712
        b, f = n * (4 * 5 + 2 + 2) + 910 * 263 * 2 + 2542 * 263 * 2, 910 * 263 * 80
    elif k == "tbc":
        b, f = _tbc_work(case["system"], case["fields"], True)
    elif k == "dropouts":
        b, f = case["fields"] * 29 * 31712 * 16, case["fields"] * 29 * 31712 * 12
    elif k == "rftbc":
        n = 262 * 2542 if case["system"] == "NTSC" else 312 * 2560
        b, f = case["fields"] * n * 4, case["fields"] * n * 20
    elif k == "efm":
        b, f = case["samples"] * 2 + case["samples"] // 28 * 8, case["samples"] * 2
    else:
        b = case["samples"] * (2 if case["dtype"] == "int16" else 4) + case["samples"] // 16 * 8
        f = case["samples"] * 2 * (11 / 2 + 11 / 4 + 2 * 11 / 8 + 2 * 13 / 16 + 2 * 55 / 16)
    return {"bytes": int(b), "flops": int(f)}


# ---- the same in 64 bits

def exact(case, seed):
    if case["kind"] in ("demod", "demodblock"):
        return _exact_demod(case, seed)
    if case["kind"] == "tbc" and case["wow"] != "quadratic":
        return _exact_tbc(case, seed)
    if case["kind"] == "ac3":
        return _exact_ac3(case, seed)
    if case["kind"] == "dropouts":
        hp = _dropout_input(case, _params(case["system"]), seed)[3]
        return {"count": None, "drops": None, "std": torch.stack([f.to(torch.float64).std(correction=0) for f in hp])}
    return None


def _disc(z, rate):
    d = torch.angle(z[:, 1:] * z[:, :-1].conj())
    d = torch.where(d < 0, d + 2 * math.pi, d) * (rate / (2 * math.pi))
    return torch.nn.functional.pad(d, (1, 0))


def _exact_demod(case, seed):
    """Overlap-save demodulation with complex128 transforms, from the same
    FP64 filter responses the decoder is given."""
    p = _params(case["system"])
    single = case["kind"] == "demodblock"
    digital = single or case["digital"]
    rot = _rf(case["system"], case["fft"], digital).delays["video_rot"]
    N, cut, end = p.blocklen, p.blockcut, p.blockcut_end
    U = N - cut - end
    nb = 1 if single else case["blocks"]
    x = torch.from_numpy(_block_input(case, seed)).cuda() if single else _demod_input(case, p, seed)
    F = {k: torch.from_numpy(np.asarray(p.Filters[k])).cuda() for k in
         ("Frfhpf", "RFVideo", "MTF", "FVideo", "FVideo05", "FVideoBurst") + (("FVideoPilot",) if case["system"] == "PAL" else ())}
    G = F["RFVideo"] * F["MTF"] ** p.scaled_mtf(case["mtf"] if single else 1)
    fs = float(p.freq_hz)
    video = {"demod": ("FVideo", 0), "demod_05": ("FVideo05", p.Filters["F05_offset"]),
             "demod_burst": ("FVideoBurst", p.Filters["FVideoBurst_offset"])}
    if case["system"] == "PAL":
        video["demod_pilot"] = ("FVideoPilot", 0)
    keep = {k: [] for k in list(video) + ["demod_raw", "rfhpf", "audio_left", "audio_right"]}
    fdiv = N // 1024
    for b0 in range(0, nb, 128):
        nn = min(128, nb - b0)
        blocks = x[b0 * U:b0 * U + (nn - 1) * U + N].unfold(0, N, U).to(torch.float64)
        X = torch.fft.fft(blocks)
        hp = torch.fft.ifft(X * F["Frfhpf"]).real
        keep["rfhpf"].append(hp[:, cut - rot:N - end - rot].reshape(-1))
        for ch in ("left", "right"):
            a = p.audio[ch]
            sub = torch.cat((X[:, a.lowbin:a.lowbin + 512], X[:, N - a.lowbin - 512:N - a.lowbin]), 1)
            d = _disc(torch.fft.ifft(sub * torch.from_numpy(np.asarray(a.filt1)).cuda()), a.a1_freq) + a.low_freq
            keep["audio_" + ch].append(d[:, cut // fdiv:(-end // fdiv) + 1024].reshape(-1))
        dem = _disc(torch.fft.ifft(X * G), fs)
        keep["demod_raw"].append(dem[:, cut:N - end].reshape(-1))
        D = torch.fft.fft(dem.clamp(1_500_000, fs * 0.75))
        for k, (name, roll) in video.items():
            v = torch.fft.ifft(D * F[name]).real
            keep[k].append(torch.roll(v, -int(roll), 1)[:, cut:N - end].reshape(-1))
        del X, D, dem, hp, v
    out = {k: torch.cat(v) for k, v in keep.items()}
    if digital:
        out["efm"] = None
    return out


def _natural_cubic(h, y):
    """Second derivatives of the natural cubic spline through (i h, y[i])."""
    n = len(y)
    a = np.diag(np.full(n - 2, 4.0)) + np.diag(np.ones(n - 3), 1) + np.diag(np.ones(n - 3), -1)
    return np.concatenate(([0.0], np.linalg.solve(a, 6.0 * np.diff(y, 2) / h ** 2), [0.0]))


def _exact_tbc(case, seed):
    """Spline coordinates, wow levels and the 16-tap windowed-sinc gather, FP64 over the float32 table."""
    rf = _params(case["system"])
    nf, n = case["fields"], _read_len(rf)
    outw, outl, _ = _geometry(rf)
    buf = _baseband(rf, n, seed, nf)
    lut = torch.from_numpy(rf.downscale_sinc_lut).cuda().to(torch.float64)
    out = torch.empty((nf, outw * outl), dtype=torch.float64, device="cuda")
    lines, h = _lines(rf, nf, seed), float(rf.linelen)
    for f in range(nf):
        y, off = lines[f], _offset(rf, f)
        x = np.arange((outl + off + 1) * outw) * (h / outw)
        j = np.clip((x / h).astype(np.int64), 0, len(y) - 2)
        t = x - j * h
        if case["wow"] == "cubic":
            m = _natural_cubic(h, y)
            c1 = (y[j + 1] - y[j]) / h - h * (2 * m[j] + m[j + 1]) / 6
            c3 = (m[j + 1] - m[j]) / (6 * h)
            coord = y[j] + t * (c1 + t * (m[j] / 2 + t * c3))
            wow = c1 + t * (m[j] + 3 * t * c3)
        else:
            wow = (y[j + 1] - y[j]) / h
            coord = y[j] + wow * t
        med = np.median(wow)
        mad = np.median(np.abs(wow - med))
        la = np.where(np.abs(wow - med) > (15 * mad if mad > 0 else 0.001), med, wow)
        if case["smoothing"] > 0:
            al = 1 / (case["smoothing"] * outw)
            last, w = la[0], (1 - al) ** np.arange(1, 2049)
            sm = np.empty_like(la)
            sm[0] = last
            for i in range(1, len(la), 2048):
                c = la[i:i + 2048]
                q = w[:len(c)]
                sm[i:i + len(c)] = q * (last + np.cumsum(al * c / q))
                last = sm[i + len(c) - 1]
            la = sm
        at = slice(outw * (off + 1), outw * (off + 1) + outw * outl)
        c = torch.from_numpy(coord[at]).cuda()
        ci = c.long()
        ph = (c - ci) * 65536
        ps = ph.long()
        w = torch.lerp(lut[ps], lut[ps + 1], (ph - ps)[:, None])
        taps = buf[f][(ci - 7)[:, None] + torch.arange(16, device="cuda")].to(torch.float64)
        out[f] = torch.from_numpy(la[at]).cuda() * (taps * w).sum(1)
    return {"f32": out, "u16": None}


def _exact_ac3(case, seed):
    """The front end's FIR stages over the whole input, FP64 over its float32 taps and tables."""
    from ldgpu.ac3 import Ac3Design
    d = Ac3Design(float(FS))

    def fir(u, taps, step):
        h = torch.from_numpy(np.asarray(taps, np.float64)[::-1].copy()).cuda()
        return torch.cat([torch.nn.functional.pad(u[max(0, a - len(h) + 1):a + (1 << 22)], (max(0, len(h) - 1 - a), 0))
                          .unfold(0, len(h), step) @ h for a in range(0, len(u), 1 << 22)])

    u = _ac3_input(case, seed).to(torch.float64)
    u = fir(fir(u, d.hb19, 2), d.hb19, 2)
    ph = (torch.arange(len(u), device="cuda") * d.phase_step) & 16383
    res = []
    for tab in (d.cos_lut, d.sin_lut):
        v = u * torch.from_numpy(tab).cuda().to(torch.float64)[ph]
        res.append(fir(fir(fir(v, d.hb19, 2), d.hb23, 2), d.rrc, 1))
    return tuple(res)
