"""Captures in which the FP64 guard flips a threshold decision, so that edges,
field windows and line locations run again from the in-pulse bits it corrected:
in a round of several captures, of which others have no flip, and alone.  The
round must give what each capture gives alone; a capture alone must give the
field windows and line locations that the stage entry points form from the
corrected float signal.  Integers and FP64 formed alike: all equal."""
import numpy as np
import pytest

import cuvhs_b200 as cv

FLIPS = [(14.0, 1), (24.0, 2), (32.0, 2)]  # the first and last flip


@pytest.mark.gpu
def test_flips_in_a_round_match_single_decodes_and_the_stages():
    import torch
    from cuvhs_b200 import stages
    caps = [(cv.synth_capture(sample_rate_hz=40e6, n_fields=60, seed=s, snr_db=snr, jitter_bound=2.0), 40.0)
            for snr, s in FLIPS]
    with cv.Batch(lanes=1, max_fields=64, round_fields=192) as b:
        b.set_timing(True)
        got = b.decode(caps)
        passes = b.stage_times()["field_windows"][1]
    alone = 0
    for (x, mhz), g in zip(caps, got):
        with cv.Decoder(mhz, batch_fields=64, debug=True) as d:
            d.set_timing(True)
            d.reset_stage_times()
            r = d.decode_capture(x)
            again = d.stage_times()["field_windows"][1] - 1
            offs, ll = d.debug_array("field_offsets"), d.debug_array("linelocs_coarse")
        alone += again
        assert g.json == r.json
        assert np.array_equal(g.luma, r.luma) and np.array_equal(g.chroma, r.chroma)
        with cv.Decoder(mhz, batch_fields=64) as s:
            nf = min(64, x.size // s.samples_per_field)
            n_read = min(nf * s.tile_stride, x.size)
            tiles = min(n_read // s.samples_per_field, nf)
            sync = stages.fm_demod(s, torch.from_numpy(x).cuda(), tiles, n_read)[1]
            so, _ = stages.discover_vsyncs(s, sync, tiles, nf)
            sl, _ = stages.line_locations(s, 0, so, *stages.sync_pulses(s, sync, tiles, so))
        assert np.array_equal(offs, so) and np.array_equal(ll, sl.ravel())
    assert alone == 2  # both kinds were there
    assert passes == 2  # one round, run again
