"""Performance cases: the decoder's work as its users have it do, through its public entry points.

A case is a dict of plain values; its "kind" names the entry point:

  chunk     Decoder.decode_chunk_device: a whole decode of a capture window that is
            already in device memory, planes left there (the headline measurement)
  capture   cuvhs_decode_capture from page-locked host memory into page-locked
            planes, with the field records, dropouts and .tbc.json text (what the
            CLI and a capture program do)
  batch     Batch.run: many captures of mixed rates and lengths, host to host
  demod     stages.fm_demod: RF samples to video, sync and envelope
  lines     stages.hsync_refine and stages.tbc_resample: line starts and luma
  chroma    stages.chroma_decode: RF samples to the chroma plane
  grad      Adjoint.grad: one calibration step's loss and gradient (backward)
  planes    Adjoint.planes: the calibration model's planes (forward)

Captures come from the package's seeded synthesizer, which stands in for tapes;
"worn" ones carry more noise and jitter, dropouts and head switches; "whole" ones
are decoded to their end, the others are a window of a longer capture.
"""
import ctypes
import math

import numpy as np
import torch

import cuvhs_b200 as cv
from cuvhs_b200 import stages
from cuvhs_b200._lib import alloc_output, lib, max_fields_for
from cuvhs_b200.calibrate import Adjoint

DEVICE = 0


def listed():
    return [
        # a preview or a single test grab: six fields, where launches and waits count
        dict(name="chunk_28_6", kind="chunk", mhz=28.0, fields=6, system="NTSC", fmt="u8", dc=False, worn=False,
             whole=True),
        # the headline: 40 fields (20 frames) at 28 MHz
        dict(name="chunk_28_40", kind="chunk", mhz=28.0, fields=40, system="NTSC", fmt="u8", dc=False, worn=False,
             whole=True),
        # archive decode of a worn tape at 40 MHz, long chunks that do not fit L2
        dict(name="chunk_40_120_worn", kind="chunk", mhz=40.0, fields=120, system="NTSC", fmt="u8", dc=False,
             worn=True, whole=False),
        # PAL from a 16-bit capture card
        dict(name="chunk_pal_40_16_s16", kind="chunk", mhz=40.0, fields=16, system="PAL", fmt="s16", dc=False,
             worn=False, whole=True),
        # the same 40 fields from and to host memory, as the CLI moves them
        dict(name="capture_28_40", kind="capture", mhz=28.0, fields=40, system="NTSC", fmt="u8", dc=False, worn=False,
             whole=True),
        # a shelf of short captures of mixed rates decoded together
        dict(name="batch_mixed_10", kind="batch", count=10, low=2, high=24),
        # the demodulator alone: a short window, and a 16-bit window with DC correction
        dict(name="demod_28_3", kind="demod", mhz=28.0, fields=3, system="NTSC", fmt="u8", dc=False, worn=False,
             whole=False),
        dict(name="demod_358_24_u16_dc", kind="demod", mhz=35.8, fields=24, system="NTSC", fmt="u16", dc=True,
             worn=True, whole=False),
        # line refinement and luma resampling alone
        dict(name="lines_40_32", kind="lines", mhz=40.0, fields=32, system="NTSC"),
        # the chroma decode alone
        dict(name="chroma_28_24", kind="chroma", mhz=28.0, fields=24, system="NTSC", fmt="u8", dc=False, worn=True,
             whole=True),
        # one step of tape calibration on eight fields, and the model's forward planes
        dict(name="grad_28_8", kind="grad", mhz=28.0, fields=8),
        dict(name="planes_28_4", kind="planes", mhz=28.0, fields=4),
    ]


# capture rates in use: 8 fsc and 10 fsc cards, the 28 and 40 MHz samplers, a 20 MHz one
RATES = (20.0, 28.0, 28.636, 35.8, 40.0)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("chunk", "chunk", "chunk", "chunk", "capture", "batch", "demod", "demod", "lines", "chroma",
                       "chroma", "grad", "planes"))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 12), low=2, high=rng.randint(6, 24))
    if kind in ("grad", "planes"):
        return dict(kind=kind, mhz=rng.choice(RATES), fields=rng.randint(2, 12))
    top = {"chunk": 100, "capture": 60, "demod": 48, "lines": 64, "chroma": 48}[kind]
    low = {"chunk": 4, "capture": 4, "demod": 1, "lines": 2, "chroma": 4}[kind]
    case = dict(kind=kind, mhz=rng.choice(RATES), fields=_log_int(rng, low, top),
                system="PAL" if rng.random() < 0.3 else "NTSC")
    if kind == "lines":
        return case
    fmt = rng.choice(("u8", "u8", "u8", "s16", "u16"))
    whole = kind == "capture" or (kind != "demod" and rng.random() < 0.5)
    return dict(case, fmt=fmt, dc=fmt != "u8" and rng.random() < 0.5, worn=rng.random() < 0.5, whole=whole)


# ------------------------------------------------------------------ geometry

def _format(mhz, system):
    """Samples per line, per field and per field slot of a capture."""
    ntsc = system == "NTSC"
    spl = int(math.floor(mhz * 1e6 / (15734.264 if ntsc else 15625.0) + 0.5))
    spf = spl * (263 if ntsc else 313)
    return spl, spf, spf + 20 * spl


def _plane(system):
    return (263, 910) if system == "NTSC" else (313, 1135)


# ------------------------------------------------------------------- inputs

def _tape(case, seed):
    """The capture as a host array of the case's input format: of the case's
    fields, or (a window of a longer capture) reaching past all their slots."""
    worn = case["worn"]
    _, spf, slot = _format(case["mhz"], case["system"])
    fields = case["fields"] if case["whole"] else case["fields"] * slot // spf + 2
    kw = dict(sample_rate_hz=case["mhz"] * 1e6, n_fields=fields, seed=seed, snr_db=34.0 if worn else 40.0,
              jitter_bound=1.5 if worn else 0.5, system=1 if case["system"] == "PAL" else 0)
    if worn:
        kw.update(dropout_line_rate=0.003, headswitch_min=3, headswitch_max=8)
    x = cv.synth_capture(**kw)
    if case["fmt"] == "u8":
        return x
    s = (x.astype(np.int16) - 128) * 200  # a 16-bit card's gain and offset
    return (s + 40).astype(np.int16) if case["fmt"] == "s16" else (s.astype(np.int32) + 32768 + 40).astype(np.uint16)


def _fields_in(case, x):
    """Fields a chunk over the capture asks for."""
    return x.size // _format(case["mhz"], case["system"])[1] if case["whole"] else case["fields"]


def _on_device(x):
    return torch.from_numpy(x.view(np.int16) if x.dtype == np.uint16 else x).cuda(DEVICE)


def _decoder(case, batch_fields):
    return cv.Decoder(case["mhz"], device=DEVICE, batch_fields=batch_fields, input_format=case.get("fmt", "u8"),
                      dc_correct=case.get("dc", False), system=case["system"])


def _baseband(case, seed):
    """Sync and video (Hz relative to 0 IRE) of a chunk with its coarse line
    starts: line-locked sync pulses with finite edges, porches, a ramp picture
    and demodulation noise."""
    mhz, fields = case["mhz"], case["fields"]
    spl, _, slot = _format(mhz, case["system"])
    ntsc = case["system"] == "NTSC"
    lpf = 525 if ntsc else 625
    hz_ire = 1e6 / 140.0 if ntsc else 1e6 / (100.0 + 0.3 * (100.0 / 0.7))
    tip = -40.0 if ntsc else -0.3 * (100.0 / 0.7)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    n = fields * slot
    lines = n // spl + 2
    walk = torch.randn(lines, generator=gen, **f64).mul_(0.05).cumsum(0)
    start = torch.arange(lines, **f64) * (mhz * 1e6 / (15734.264 if ntsc else 15625.0)) + 0.4 * torch.sin(walk) + 3.0
    t = torch.arange(n, **f64)
    line = (torch.searchsorted(start, t, right=True) - 1).clamp_(0, lines - 2)
    us = (t - start[line]) / mhz  # microseconds into the line
    edge = 0.12
    pulse = 0.5 * (torch.tanh(us / edge) - torch.tanh((us - 4.7) / edge))
    picture = torch.where((us > 9.4) & (us < 61.0), 7.5 + 85.0 * ((us - 9.4) / 51.6 + 0.01 * line % 1.0) % 90.0, 0.0)
    noise = torch.randn(n, generator=gen, device="cuda")
    sync = (pulse * tip * hz_ire).float() + 900.0 * noise
    video = ((pulse * tip + picture) * hz_ire).float() + 6000.0 * noise
    # field f's table: lines from the first one inside its slot
    table = torch.empty(fields, lpf, **f64)
    for f in range(fields):
        first = int(math.ceil(f * slot / spl)) + 1
        at = torch.arange(first, first + lpf, device="cuda")
        table[f] = start[at.clamp(max=lines - 1)]
        table[f][at >= lines] = float(n) + 10.0 * spl  # past the signal
    coarse = torch.round(table + torch.randn(table.shape, generator=gen, **f64).mul_(1.5))
    return sync.contiguous(), video.contiguous(), coarse.contiguous()


def _batch_specs(case):
    return cv.batch_specs(case["count"], case["low"], case["high"])


def _batch_captures(case, seed):
    """Rates, lengths and impairments are the case's, the noise and picture the seed's."""
    return [(cv.synth_capture(**dict(p, seed=1000 * seed + i)), p["sample_rate_hz"] / 1e6)
            for i, p in enumerate(_batch_specs(case))]


def _calibration(case, seed):
    """A tape with perturbed pre-emphasis, carrier and line offsets, and a
    target in the neighbourhood of its model planes."""
    kw = dict(sample_rate_hz=case["mhz"] * 1e6, n_fields=case["fields"] + 1, seed=seed, snr_db=42.0, jitter_bound=0.3,
              preemph_perturb=(0.05, -0.04, 0.05), carrier_offset_hz=20e3, line_offset_bound=0.8,
              chroma_phase_bound=0.2)
    return cv.synth_capture(**kw)


# ------------------------------------------------------------------ prepare

class _Planes:
    """The decoder's device planes as tensors, looked up after each chunk."""

    def __init__(self, dec):
        self.dec, self.at = dec, {}

    def _view(self, ptr, fields):
        if ptr not in self.at:
            view = type("DevicePlane", (), {})()
            view.owner = self.dec  # the planes live as long as their decoder
            view.__cuda_array_interface__ = dict(shape=(fields,) + self.dec.field_shape, typestr="<i2",
                                                 data=(ptr, False), version=2)
            self.at[ptr] = torch.as_tensor(view, device=f"cuda:{DEVICE}")
        return self.at[ptr]

    def last(self, fields):
        y, c = ctypes.c_void_p(), ctypes.c_void_p()
        lib.cuvhs_device_outputs(self.dec._h, ctypes.byref(y), ctypes.byref(c))
        full = self.dec.batch_fields
        return self._view(y.value, full)[:fields], self._view(c.value, full)[:fields]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("chunk", "capture", "demod", "chroma"):
        x = _tape(case, seed)
        spf = _format(case["mhz"], case["system"])[1]
        nf = _fields_in(case, x)
        dec = s["dec"] = _decoder(case, nf)
        assert dec.samples_per_field == spf
        s["n"], s["nf"] = x.size, nf
    if kind == "chunk":
        s["raw"] = _on_device(x)
        s["planes"] = _Planes(dec)
    elif kind == "capture":
        s["pin"] = torch.from_numpy(x.view(np.int16) if x.dtype == np.uint16 else x).pin_memory()
        s["out"], s["bufs"] = alloc_output(max_fields_for(x.size, spf), pinned=True, shape=dec.field_shape)
        s["json"] = ctypes.create_string_buffer(1 << 20)
    elif kind == "batch":
        s["batch"] = cv.Batch(max_fields=32, round_fields=64, device=DEVICE)
        s["items"], s["bufs"] = s["batch"].prepare(_batch_captures(case, seed), pinned=True)
    elif kind == "demod":
        s["raw"] = _on_device(x)
        s["n_read"] = min(nf * dec.tile_stride, x.size)
        s["tiles"] = min(s["n_read"] // spf, nf)
    elif kind == "lines":
        dec = s["dec"] = cv.Decoder(case["mhz"], device=DEVICE, batch_fields=case["fields"], system=case["system"])
        s["sync"], s["video"], s["coarse"] = _baseband(case, seed)
        assert s["sync"].numel() == case["fields"] * dec.tile_stride
    elif kind == "chroma":
        raw = s["raw"] = _on_device(x)
        n_read = min(nf * dec.tile_stride, x.size)
        tiles = min(n_read // spf, nf)
        # the line starts, as a program that composes the stages has them
        _, sync, _ = stages.fm_demod(dec, raw, tiles, n_read)
        offs, _ = stages.discover_vsyncs(dec, sync, tiles, nf)
        ll, _ = stages.line_locations(dec, 0, offs, *stages.sync_pulses(dec, sync, tiles, offs))
        s["n_read"] = n_read
        s["ll"] = stages.hsync_refine(dec, sync, torch.from_numpy(ll).cuda(DEVICE))
    elif kind in ("grad", "planes"):
        adj = s["adj"] = Adjoint(_calibration(case, seed), case["mhz"], fields=case["fields"], device=DEVICE)
        p = s["params"] = adj.default_params()
        rng = np.random.default_rng(seed)
        p.line_offset = rng.uniform(-0.3, 0.3, p.line_offset.shape)
        p.chroma_phase = rng.uniform(-0.1, 0.1, p.chroma_phase.shape)
        if kind == "grad":
            aim = adj.default_params()
            aim.carrier_hz, aim.deviation = 12e3, 1.02
            adj.set_target(*adj.planes(aim))
    return s


# ---------------------------------------------------------------------- run

def _records(out, bufs):
    """Field records and dropouts of a filled cuvhs_output, as arrays."""
    n, m = out.fields_out, out.dropouts_out
    rec = np.frombuffer(bufs["fields"], np.uint8, n * ctypes.sizeof(bufs["fields"]) // len(bufs["fields"]))
    return dict(luma=bufs["luma"][:n], chroma=bufs["chroma"][:n], fields=rec, line=bufs["dl"][:m],
                start=bufs["ds"][:m], end=bufs["de"][:m])


def run(state):
    s = state
    kind = s["case"]["kind"]
    if kind == "chunk":
        dec = s["dec"]
        dec.reset()
        got, nxt = dec.decode_chunk_device(s["raw"].data_ptr(), s["n"], 0, s["nf"])
        luma, chroma = s["planes"].last(got)
        return dict(fields=got, next=nxt, luma=luma, chroma=chroma)
    if kind == "capture":
        dec, out = s["dec"], s["out"]
        dec.reset()
        out.fields_out = out.dropouts_out = 0
        dec._check(lib.cuvhs_decode_capture(dec._h, s["pin"].data_ptr(), s["n"], ctypes.byref(out)))
        size = lib.cuvhs_json(dec._h, ctypes.byref(out), s["json"], len(s["json"]))
        return dict(_records(out, s["bufs"]), json=np.frombuffer(s["json"], np.uint8, min(size, len(s["json"]) - 1)))
    if kind == "batch":
        for b in s["bufs"]:
            b["out"].fields_out = b["out"].dropouts_out = 0
        s["batch"].run(s["items"])
        return [{k: r[k] for k in ("luma", "chroma", "fields")} for r in (_records(b["out"], b) for b in s["bufs"])]
    if kind == "demod":
        video, sync, env = stages.fm_demod(s["dec"], s["raw"], s["tiles"], s["n_read"])
        return dict(video=video, sync=sync, envelope=env)
    if kind == "lines":
        ll = stages.hsync_refine(s["dec"], s["sync"], s["coarse"].clone())
        return dict(lines=ll, luma=stages.tbc_resample(s["dec"], s["video"], ll))
    if kind == "chroma":
        s["dec"].reset()
        chroma, ids = stages.chroma_decode(s["dec"], s["raw"], s["ll"], s["n_read"])
        return dict(chroma=chroma, ids=ids)
    if kind == "grad":
        loss, g = s["adj"].grad(s["params"])
        return dict(loss=loss, deemph=g.deemph, carrier=g.carrier_hz, deviation=g.deviation,
                    line_offset=g.line_offset, chroma_phase=g.chroma_phase)
    luma, chroma = s["adj"].planes(s["params"])
    return dict(luma=luma, chroma=chroma)


# --------------------------------------------------------------------- work

# Block filtering of one sample through one real-signal filter at the block
# lengths that suit the supports: three FFTs of N points for two blocks of
# about 0.8 N outputs, 5 N log2 N operations each.
FILTER_FLOPS = 115.0


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: the filters
    each path cannot do without (demod two, chroma one) and about 200 a
    resampled and band-passed pixel."""
    kind = case["kind"]
    if kind == "batch":
        specs = _batch_specs(case)
        parts = [dict(kind="capture", mhz=p["sample_rate_hz"] / 1e6, fields=p["n_fields"], system="NTSC", fmt="u8")
                 for p in specs]
        each = [work(p) for p in parts]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    system = case.get("system", "NTSC")
    _, spf, slot = _format(case["mhz"], system)
    rows, cols = _plane(system)
    n, px, fields = case["fields"] * spf, case["fields"] * rows * cols, case["fields"]
    size = 1 if case.get("fmt", "u8") == "u8" else 2
    if kind in ("chunk", "capture"):
        return {"bytes": n * size + 4 * px, "flops": 3 * FILTER_FLOPS * n + 220 * px}
    if kind == "demod":
        return {"bytes": n * size + 12 * n, "flops": 2 * FILTER_FLOPS * n}
    if kind == "lines":
        # every line's sync window (about 14 us) and the whole video
        return {"bytes": fields * slot * 4 * 0.22 + fields * slot * 4 + 2 * px, "flops": 20 * px}
    if kind == "chroma":
        return {"bytes": n * size + 2 * px, "flops": FILTER_FLOPS * n + 200 * px}
    if kind == "grad":
        # demod, colour-under signal and both targets in; gradients are small
        return {"bytes": 8 * n + 8 * px, "flops": 3 * FILTER_FLOPS * n + 450 * px}
    return {"bytes": 8 * n + 8 * px, "flops": FILTER_FLOPS * n + 220 * px}


# -------------------------------------------------------------------- exact

def _bandpass(w, lo, hi, order):
    tl, th, t = math.tan(lo / 2), math.tan(hi / 2), torch.tan(w / 2)
    s = (t * t - tl * th) / ((th - tl) * t)
    h = 1.0 / torch.sqrt(1.0 + s.abs().pow(2.0 * order))
    return torch.where((w <= 0) | (w >= math.pi), torch.zeros_like(h), h)


def _smooth7(n):
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _exact_demod(case, seed):
    """The demodulator in 64 bits: each tile filtered whole in the frequency domain."""
    x = _tape(case, seed)
    fs, (_, spf, slot) = case["mhz"] * 1e6, _format(case["mhz"], case["system"])
    nf = _fields_in(case, x)
    n_read = min(nf * slot, x.size)
    tiles = min(n_read // spf, nf)
    total, ny, lead = tiles * slot, fs / 2, 2048
    n_read = min(n_read, total)
    raw = torch.zeros(total, dtype=torch.float64, device="cuda")
    head = torch.from_numpy(x[:n_read].astype(np.float64)).cuda()
    head = {"u8": lambda v: (v - 128) * 256, "s16": lambda v: v, "u16": lambda v: v - 32768}[case["fmt"]](head)
    raw[:n_read] = head - head.mean() if case["dc"] else head
    tile = _smooth7(slot + lead)
    bins = tile // 2 + 1
    ntsc = case["system"] == "NTSC"
    hz_ire = 1e6 / 140 if ntsc else 1e6 / (100 + 0.3 * (100 / 0.7))
    ire0 = (4.4e6 if ntsc else 4.8e6) - 100 * hz_ire
    k = torch.arange(bins, dtype=torch.float64, device="cuda")
    w = math.pi * k / (bins - 1)
    rf = _bandpass(w, math.pi * 1.3e6 / ny, math.pi * 7.5e6 / ny, 8)
    if math.pi * 8e6 / ny < math.pi:
        rf = rf / torch.sqrt(1 + (torch.tan(w / 2) / math.tan(math.pi * 8e6 / ny / 2)).abs().pow(16))
    rf = rf / torch.sqrt(1 + (math.tan(math.pi * 1e6 / ny / 2) / torch.tan(w / 2)).abs().pow(16))
    rf[0] = 0
    hilbert = torch.full_like(rf, 2.0)
    hilbert[0] = hilbert[-1] = 1.0
    rf = torch.cat([rf * hilbert, torch.zeros(tile - bins, dtype=torch.float64, device="cuda")])
    # de-emphasis: the inverse of the pre-emphasis shelf; video and sync low-passes
    a_, w0 = 10 ** (13.9794 / 40), 2 * math.pi * 273755.82 / fs
    al, c, sa = math.sin(w0) / (2 * 0.462088186), math.cos(w0), math.sqrt(a_)
    num = (a_ + 1 - (a_ - 1) * c + 2 * sa * al, 2 * (a_ - 1 - (a_ + 1) * c), a_ + 1 - (a_ - 1) * c - 2 * sa * al)
    den = (a_ * (a_ + 1 + (a_ - 1) * c + 2 * sa * al), -2 * a_ * (a_ - 1 + (a_ + 1) * c),
           a_ * (a_ + 1 + (a_ - 1) * c - 2 * sa * al))
    z = torch.exp(-1j * w)
    shelf = (num[0] + num[1] * z + num[2] * z * z) / (den[0] + den[1] * z + den[2] * z * z)
    f = 2 * (k * ny / (bins - 1)) * (math.log(2) / 2) ** (1 / 18) / 3.0e6
    hv = shelf * torch.exp(-2 * f.pow(18))
    m = torch.arange(65, dtype=torch.float64, device="cuda") - 32
    cut = 500e3 / ny
    taps = torch.where(m == 0, torch.full_like(m, cut), torch.sin(math.pi * cut * m) / (math.pi * m)) * (
        0.54 - 0.46 * torch.cos(2 * math.pi * (m + 32) / 64))
    taps = taps / taps.sum()
    fir = torch.full_like(w, float(taps[32]))  # symmetric taps: a real response about the middle
    for j in range(1, 33):
        fir = fir + 2 * taps[32 + j] * torch.cos(j * w)
    hs = hv * fir
    at = torch.arange(tile, device="cuda")

    def window(signal, t):
        return signal[(t * slot - lead + at).clamp(0, total - 1)]

    dem = torch.empty_like(raw)
    env = torch.empty_like(raw)
    for t in range(tiles):
        v = torch.fft.ifft(torch.fft.fft(window(raw, t)) * rf) * tile
        step = torch.angle(v[lead:lead + slot] * v[lead - 1:lead - 1 + slot].conj())
        dem[t * slot:(t + 1) * slot] = step * fs / (2 * math.pi)
        env[t * slot:(t + 1) * slot] = v[lead:lead + slot].abs()
    video = torch.empty_like(raw)
    sync = torch.empty_like(raw)
    for t in range(tiles):
        spec = torch.fft.rfft(window(dem, t))
        for out, h in ((video, hv), (sync, hs)):
            out[t * slot:(t + 1) * slot] = torch.fft.irfft(spec * h, n=tile)[lead:lead + slot] - ire0
    return dict(video=video, sync=sync, envelope=env)


def exact(case, seed):
    """64-bit results of the demodulator.  The planes are whole numbers; the
    refined line starts and the calibration model start from the decoder's own
    intermediates and have no such value here."""
    if case["kind"] == "demod":
        return _exact_demod(case, seed)
    return None
