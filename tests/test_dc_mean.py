"""The DC mean over captures that start off a 16-byte boundary and over every
remainder of the 16-byte loads.  A capture whose converted samples have the
exact integer mean M, decoded with DC correction, is the capture shifted by -M
decoded without it: the same floats enter the chain, so the outputs are equal
byte for byte."""
import numpy as np
import pytest

import cuvhs_b200 as cv


@pytest.mark.gpu
@pytest.mark.parametrize("fmt,dtype,zero,mean", [("u8", np.uint8, 128, 119), ("s16", np.int16, 0, -1234),
                                                 ("u16", np.uint16, 32768, 41000)])
def test_dc_mean_alignment_and_remainders(fmt, dtype, zero, mean):
    import torch
    from cuvhs_b200 import stages
    rng = np.random.default_rng(5)
    with cv.Decoder(28.0, batch_fields=1, input_format=fmt, dc_correct=True) as a, \
            cv.Decoder(28.0, batch_fields=1, input_format=fmt) as b:
        for n in (1, 7, 8, 9, 31, 33, 4099, a.tile_stride - 5, a.tile_stride):
            x = rng.integers(-60, 61, n).astype(np.int64)
            x = x if fmt == "u8" else x * 90
            step = 1 if x.sum() < 0 else -1
            x += step * (abs(int(x.sum())) // n)
            x[:abs(int(x.sum()))] += step
            assert x.sum() == 0
            want = stages.fm_demod(b, torch.from_numpy((x + zero).astype(dtype)).cuda(), 1, n)
            want = [w.cpu().numpy() for w in want]
            for off in (0, 1, 3, 15):
                buf = torch.from_numpy(np.concatenate([np.zeros(off, dtype), (x + mean).astype(dtype)])).cuda()
                got = stages.fm_demod(a, buf[off:], 1, n)
                for g, w in zip(got, want):
                    assert np.array_equal(g.cpu().numpy().view(np.uint32), w.view(np.uint32))
