"""Dropouts of a whole decode -- the class, scan and strip kernels that detect
a chunk's dropouts, map them and conceal its planes -- against the same planes
taken unconcealed from the stage entry points, with the entries and the
concealment of test_dropout_conceal.py's restatement of the reference's steps.
Captures with many dropouts; among them some whose chroma tracks change places
part-way, so that fields are decoded and concealed a second time: their lines
may only be written again once the first concealment has passed, or old pixels
come to lie on new ones.  All values are integers and must be equal."""
import numpy as np
import pytest

import cuvhs_b200 as cv
import test_dropout_conceal as ref


def capture(system, mhz, fields, swap_at, per_line, longest, seed):
    """Samples with runs of weak signal inside the picture part of the lines
    (bursts and sync pulses stay, but where a run covers whole lines), and the
    first track swapped from field swap_at on."""
    kw = dict(sample_rate_hz=mhz * 1e6, n_fields=fields, seed=seed, snr_db=42.0, jitter_bound=0.4, start_line=0.0,
              system=1 if system == "PAL" else 0)
    per_field = 312.5 if system == "PAL" else 262.5
    starts = cv.synth_lines(**kw)[0]
    a, b = (cv.synth_capture(**dict(kw, first_track=t)) for t in (0, 1))
    x = np.concatenate([a[:int(starts[int(per_field * swap_at)])], b[int(starts[int(per_field * swap_at)]):]])
    rng = np.random.default_rng(seed)
    weak = np.zeros(x.size, bool)
    line = starts[1] - starts[0]
    for f in range(1, fields):
        rows = np.arange(int(f * per_field) + 25, int((f + 1) * per_field) - 10)
        for r in rng.choice(rows, int(per_line * rows.size), replace=per_line > 1):
            s = int(starts[r] + rng.uniform(0.2, 0.9) * line)
            n = rng.integers(20, longest)
            weak[s:s + (n if n > line else min(n, int(starts[r] + 0.97 * line) - s))] = True
    x[weak] = np.round(128.0 + 0.02 * (x[weak].astype(np.float64) - 128.0)).astype(np.uint8)
    return x


def unconcealed(mhz, system, x, fields):
    """(envelope, line locations, luma, chroma, first phase IDs) of a chunk from the stages."""
    import torch
    from cuvhs_b200 import stages
    with cv.Decoder(mhz, batch_fields=fields, system=system) as s:
        spp = s.tile_stride
        nf = min(fields, x.size // s.samples_per_field)
        n_read = min(nf * spp, x.size)
        tiles = min(n_read // s.samples_per_field, nf)
        raw = torch.from_numpy(x).cuda()
        video, sync, env = stages.fm_demod(s, raw, tiles, n_read)
        offs, _ = stages.discover_vsyncs(s, sync, tiles, nf)
        ll, _ = stages.line_locations(s, 0, offs, *stages.sync_pulses(s, sync, tiles, offs))
        ll = torch.from_numpy(ll).cuda()
        stages.hsync_refine(s, sync, ll)
        luma = stages.tbc_resample(s, video, ll).cpu().numpy().view(np.uint16)
        chroma = stages.chroma_decode(s, raw, ll, n_read)[0].cpu().numpy().view(np.uint16)
        return spp, env.cpu().numpy(), ll.cpu().numpy(), luma, chroma


@pytest.mark.gpu
@pytest.mark.parametrize("system,mhz,fields,swap_at,per_line,longest", [
    ("NTSC", 28.0, 20, 1, 0.6, 400),
    ("NTSC", 28.0, 20, 4, 0.6, 400),
    ("NTSC", 28.0, 20, 7, 0.4, 900),
    ("PAL", 40.0, 18, 3, 0.5, 500),
    # runs over many lines, which overlap and come in hundreds
    ("NTSC", 28.0, 6, 0, 0.9, 12000),
    ("NTSC", 35.8, 6, 0, 2.0, 250),
    ("PAL", 40.0, 6, 0, 0.9, 16000),
    ("PAL", 28.0, 6, 0, 2.0, 200),
])
def test_decode_conceals_as_the_reference_steps(monkeypatch, system, mhz, fields, swap_at, per_line, longest):
    x = capture(system, mhz, fields, swap_at, per_line, longest, 700 + swap_at)
    spp, env, ll, luma, chroma = unconcealed(mhz, system, x, fields)
    H, W = luma.shape[1:]
    for name, value in (("H", H), ("W", W), ("LPF", ll.shape[1]), ("ALS", 8 if system == "PAL" else 10)):
        monkeypatch.setattr(ref, name, value)
    with cv.Decoder(mhz, batch_fields=fields, system=system) as d:
        runs = []
        for _ in range(3):
            d.reset()
            runs.append(d.decode_capture(x))
    r = runs[0]
    assert r.n_fields == len(ll) >= fields - 2
    total = 0
    for f in range(r.n_fields):
        want = ref._entries(ref._runs(env, ll[f], spp, f), ll[f]) if (f + 1) * spp <= env.size else None
        got = list(zip(*(a.tolist() for a in r.dropouts[f])))
        assert want is None or got == want, f
        ref._conceal(luma[f], got)
        ref._conceal(chroma[f], got)
        total += len(got)
    # the reference looks for field f's dropouts in slot f alone, which trails
    # the field by 20 lines more each time: only the first dozen fields have any
    assert total > 300
    for q in runs:
        assert np.array_equal(q.luma, luma)
        assert np.array_equal(q.chroma, chroma)
