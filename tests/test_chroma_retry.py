"""Captures whose chroma tracks change places part-way: two syntheses that
differ only in the first track, spliced where a field starts, so that the
decoder's flip-and-retry runs (chroma_decode.cu:782-981) with flips that
succeed, at fields on both sides of its 15-field groups and of the line pairs
(263 lines a field: a field starts inside a pair every second time).  Against
the FP64 oracle, and as a batch against one capture at a time."""
import numpy as np
import pytest

import cuvhs_b200 as cv

FIELDS = 33


def spliced(at, seed):
    """Tracks swapped from field `at` on."""
    kw = dict(sample_rate_hz=28e6, n_fields=FIELDS, seed=seed, snr_db=42.0, jitter_bound=0.4, start_line=0.0)
    starts, _, _ = cv.synth_lines(**kw)
    cut = int(starts[int(262.5 * at)])
    a, b = (cv.synth_capture(**dict(kw, first_track=t)) for t in (0, 1))
    return np.concatenate([a[:cut], b[cut:]])


@pytest.mark.gpu
@pytest.mark.parametrize("at", [1, 4, 14, 15, 16, 22, 30])
def test_swapped_tracks_match_the_oracle(at):
    from oracle.oracle import Oracle
    x = spliced(at, 90 + at)
    with cv.Decoder(28.0) as d:
        r = d.decode_capture(x)
        spp = d.tile_stride
    o = Oracle(28.0)
    n = o.decode(x)
    assert r.n_fields == n
    inside = [i for i in range(n) if int(r.file_loc[i]) + spp <= x.size]
    assert len(inside) >= FIELDS - 3
    for i in inside:
        assert np.abs(r.chroma[i].astype(np.int32) - o.chroma[i].astype(np.int32)).max() <= 1, i
    import json
    assert [f["fieldPhaseID"] for f in json.loads(r.json)["fields"]] == [
        f["fieldPhaseID"] for f in json.loads(o.json)["fields"]]


@pytest.mark.gpu
def test_swapped_tracks_in_a_batch_match_single_decodes():
    caps = [(spliced(at, 60 + at), 28.0) for at in (3, 15, 16, 29)]
    with cv.Batch(max_fields=64, round_fields=160) as b:
        batch = b.decode(caps)
    for (x, mhz), r in zip(caps, batch):
        with cv.Decoder(mhz, batch_fields=64) as d:
            s = d.decode_capture(x)
        assert r.json == s.json
        assert np.array_equal(r.luma, s.luma) and np.array_equal(r.chroma, s.chroma)
