"""Host data reaches the device on the stream of the kernels that read it.  The
contexts' streams do not wait for the default stream, and a copy of pageable
memory there may return before its data have reached the device, so a plain
cudaMemcpy may only read device memory (after a synchronisation)."""
import os
import re

import numpy as np
import pytest

import cuvhs_b200 as cv

CSRC = os.path.join(os.path.dirname(cv.__file__), "csrc")


@pytest.mark.parametrize("source", sorted(f for f in os.listdir(CSRC) if f.endswith((".cpp", ".cu"))))
def test_no_upload_on_the_default_stream(source):
    with open(os.path.join(CSRC, source)) as f:
        copies = re.findall(r"cudaMemcpy\s*\(.*?;", f.read(), re.S)
    assert [c for c in copies if "cudaMemcpyDeviceToHost" not in c] == []


@pytest.mark.gpu
def test_gains_of_a_new_model_are_those_of_a_pass_at_its_nominal_parameters():
    from cuvhs_b200.calibrate import Adjoint
    x = cv.synth_capture(sample_rate_hz=28e6, n_fields=3, seed=12, snr_db=40)
    for _ in range(3):
        with Adjoint(x, 28.0, fields=2) as a:
            first = a.array("gains")
            assert (first > 0.0).mean() > 0.8  # lines with a burst
            a.planes(a.default_params())
            assert np.array_equal(first.view(np.uint32), a.array("gains").view(np.uint32))
