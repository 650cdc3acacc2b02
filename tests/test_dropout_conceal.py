"""The dropout stage's entries and concealment (cuvhs_dropouts_noalloc) on
planes and envelopes made to overlap: many runs to a field, runs over several
lines, several runs on a line, more spans and entries than the stage keeps,
line 0, and the groups of 32 entries the reference's copy loop works in.  The
oracle is a plain restatement of the reference's steps
(src/pipeline/dropout_detect.cu:17-339): one event after another, then the
copy loop one column step after another, every load of a step before its
stores.  All values are integers, so the results must be equal."""
import numpy as np
import pytest

import cuvhs_b200 as cv

H, W, LPF, ALS = 263, 910, 525, 10
BLOCK = 16


def _runs(env, ll, spp, f):
    """Start / end events of field f's envelope, in order."""
    s0, s1 = max(int(ll[ALS]), f * spp), min(int(ll[ALS + H]), (f + 1) * spp)
    down = env[f * spp:(f + 1) * spp].astype(np.float64).mean() * 0.18
    runs, start = [], -1
    for pos in range(s0, s1, BLOCK):
        m = env[pos:min(pos + BLOCK, s1)].astype(np.float64).mean()
        if m <= down and start < 0:
            start = pos
        elif m >= down * 1.25 and start >= 0:
            runs.append((start, pos))
            start = -1
    if start >= 0:
        runs.append((start, s1))
    return runs[:1024]


def _entries(runs, ll):
    spans = []
    for a, b in runs:
        if spans and a - spans[-1][1] <= 30:
            spans[-1][1] = b
        elif len(spans) < 128:
            spans.append([a, b])
    rows = ll[ALS:ALS + H + 1]

    def line_of(pos):
        return int(np.searchsorted(rows, pos, side="right")) - 1 if rows[0] <= pos < rows[H] else -1

    out = []
    for a, b in spans:
        sl, el = line_of(float(a)), line_of(b - 1.0)
        if b - a < 10 or sl < 0:
            continue
        el = H - 1 if el < 0 else el
        for k in range(sl, el + 1):
            n = rows[k + 1] - rows[k]
            sx = max(0, int((a - rows[k]) / n * W)) if k == sl else 0
            ex = min(W, int((b - rows[k]) / n * W + 0.999)) if k == el else W
            if ex > sx and len(out) < 512:
                out.append((k, sx, ex))
    return out


def _conceal(plane, entries):
    for g in range(0, len(entries), 32):
        group = [(k, k - 1 if k > 0 else k + 1, sx, ex) for k, sx, ex in entries[g:g + 32]]
        for step in range(max(ex - sx for _, _, sx, ex in group)):
            loads = [(k, sx + step, plane[src, sx + step]) for k, src, sx, ex in group if step < ex - sx]
            for k, c, v in loads:
                plane[k, c] = v


@pytest.mark.gpu
@pytest.mark.parametrize("per_line,longest", [(0.02, 300), (0.3, 900), (0.2, 12000), (2.5, 120), (0.9, 5000)])
def test_entries_and_concealment_match_the_reference_steps(per_line, longest):
    import torch
    from cuvhs_b200 import stages
    rng = np.random.default_rng(int(per_line * 100) + longest)
    fields = 3
    with cv.Decoder(28.0, batch_fields=fields) as d:
        spp = d.tile_stride
        ll = np.empty((fields, LPF))
        env = np.full(fields * spp, 1000.0, np.float32)
        for f in range(fields):
            ll[f] = f * spp + 3.25 + 1780.0 * np.arange(LPF) + rng.uniform(-1.5, 1.5, LPF)
            n = int(H * per_line)
            for s in rng.integers(int(ll[f, ALS]), int(ll[f, ALS + H]), n):
                env[s:min(s + rng.integers(20, longest), (f + 1) * spp)] = 5.0
            env[int(ll[f, ALS]) + 200:int(ll[f, ALS]) + 1500] = 5.0  # line 0, copied from line 1
        luma = rng.integers(0, 65536, (fields, H, W)).astype(np.uint16)
        chroma = rng.integers(0, 65536, (fields, H, W)).astype(np.uint16)
        dev = [torch.from_numpy(p.view(np.int16)).cuda() for p in (luma, chroma)]
        count, lines, sx, ex = (t.cpu().numpy() for t in stages.dropout_detect(
            d, torch.from_numpy(env).cuda(), torch.from_numpy(ll).cuda(), *dev))
    for f in range(fields):
        want = _entries(_runs(env, ll[f], spp, f), ll[f])
        got = [tuple(int(a[f * 512 + i]) for a in (lines, sx, ex)) for i in range(count[f])]
        assert got == want, f
        assert len(want) > 2
        _conceal(luma[f], want)
        _conceal(chroma[f], want)
    assert np.array_equal(dev[0].cpu().numpy().view(np.uint16), luma)
    assert np.array_equal(dev[1].cpu().numpy().view(np.uint16), chroma)
