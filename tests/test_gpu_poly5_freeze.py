"""The Poly5 freeze where the distortion itself crosses zero.

An input radius r stays where it is when |k1 r^3 + k2 r^5| < 1e-5. Where the two
terms cancel, their f32 sum is off by more than its own last places, and the f64
residual decides. The lenses below have that ring inside the image, with single
pixels on the other side of the limit in f32 and in f64.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k1, k2, focal", [(-0.0829, 0.0381, 10.0), (-0.0643, 0.0215, 9.6)])
def test_frozen_pixels_are_those_of_the_f64_residual(stages, oracle, k1, k2, focal):
    from rohditor_gb300 import OpticsExecution

    w, h = 1201, 901
    ex = OpticsExecution(w, h, distortion="poly5", distortion_k=(k1, k2, 0.0), tca="poly3",
                         tca_red=(1.0002, 0.0001, -0.0001), tca_blue=(0.9998, -0.0001, 0.0001), real_focal=focal)
    rgb = np.random.default_rng(6).uniform(0.0, 1.0, size=(h, 3 * w)).astype(np.float32)
    ref = oracle.optics_apply(oracle.optics_desc_from(ex.to_c()), rgb)
    ours = stages.optics(rgb, ex)
    assert np.array_equal(ours.view(np.uint32), ref.view(np.uint32))
