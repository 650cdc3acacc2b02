"""Threshold edges from K1b's in-pulse bits, the field windows and the pulses
formed inside the line-location pass, against the stage entry points on the
same signal (which take the edges from the float sync signal and run the pulse
kernel on its own).  The field counts lie on both sides of where the edge
passes change: one word a thread or four (9.7 million samples), counts summed
by the write pass or by a scan (134 million).  All values are integers."""
import numpy as np
import pytest

import cuvhs_b200 as cv


@pytest.mark.gpu
@pytest.mark.parametrize("fields", [1, 3, 19, 20, 266, 267])
def test_edges_windows_and_pulses_match_the_stages(fields):
    import torch
    from cuvhs_b200 import stages
    x = cv.synth_capture(sample_rate_hz=28e6, n_fields=fields + 1 + fields // 10, seed=77, snr_db=34.0,
                         jitter_bound=1.0, dropout_line_rate=0.01)
    with cv.Decoder(28.0, batch_fields=fields, debug=True) as d:
        spp, spf = d.tile_stride, d.samples_per_field
        n_read = min(fields * spp, x.size)
        tiles = min(n_read // spf, fields)
        d.decode_chunk(x[:n_read], 0, fields)
        got = {k: d.debug_array(k) for k in ("field_offsets", "k2_pulse_count", "k2_pulse_starts", "k2_pulse_lengths",
                                             "linelocs_coarse")}
    with cv.Decoder(28.0, batch_fields=fields) as s:
        _, sync, _ = stages.fm_demod(s, torch.from_numpy(x[:n_read]).cuda(), tiles, n_read)
        offs, _ = stages.discover_vsyncs(s, sync, tiles, fields)
        starts, lengths, counts = stages.sync_pulses(s, sync, tiles, offs)
        ll, _ = stages.line_locations(s, 0, offs, starts, lengths, counts)
    assert np.array_equal(got["field_offsets"], offs)
    assert np.array_equal(got["k2_pulse_count"], counts)
    assert np.array_equal(got["k2_pulse_starts"], starts.ravel())
    assert np.array_equal(got["k2_pulse_lengths"], lengths.ravel())
    assert np.array_equal(got["linelocs_coarse"], ll.ravel())
