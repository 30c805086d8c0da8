"""The Newton branch of the lens remap where its forms change over.

A pixel's inverse distortion is a closed form of one Newton step (Poly3, Poly5),
a double-float iteration, or the f64 one; a thread remaps two rows and takes the
second's taps from the first's. The lenses below reach frozen centres, one step,
several steps, weak coefficients (1 / k1 beyond the closed form's range) and wide
fields; the sizes end on an odd row. Results equal the oracle's bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENSES = {
    "poly3_barrel": dict(distortion="poly3", distortion_k=(-0.01, 0, 0)),
    "poly3_pincushion": dict(distortion="poly3", distortion_k=(0.012, 0, 0)),
    "poly3_weak": dict(distortion="poly3", distortion_k=(-0.0004, 0, 0)),
    "poly3_weaker": dict(distortion="poly3", distortion_k=(2.0e-5, 0, 0)),
    "poly3_strong": dict(distortion="poly3", distortion_k=(-0.06, 0, 0), real_focal=24.0),
    "poly3_wide": dict(distortion="poly3", distortion_k=(-0.02, 0, 0), real_focal=14.0),
    "poly5_poly3_tca": dict(distortion="poly5", distortion_k=(-0.03, 0.004, 0.0), tca="poly3",
                            tca_red=(1.0004, 0.0002, -0.0003), tca_blue=(0.9996, -0.0002, 0.0002)),
    "poly3_linear_tca": dict(distortion="poly3", distortion_k=(-0.015, 0, 0), tca="linear", tca_red=(1.002, 0, 0),
                             tca_blue=(0.997, 0, 0)),
    "poly3_poly3_tca": dict(distortion="poly3", distortion_k=(-0.015, 0, 0), tca="poly3",
                            tca_red=(1.0002, 0.0001, -0.0001), tca_blue=(0.9998, -0.0001, 0.0001)),
    "tca_only": dict(tca="poly3", tca_red=(1.0002, 0.0001, -0.0001), tca_blue=(0.9998, -0.0001, 0.0001)),
}


@pytest.mark.parametrize("name", sorted(LENSES))
@pytest.mark.parametrize("size", [(65, 33), (700, 481), (1031, 1033)])
def test_newton_forms_equal_the_oracle(stages, oracle, name, size):
    from rohditor_gb300 import OpticsExecution

    w, h = size
    rng = np.random.default_rng(w + h)
    rgb = rng.uniform(-0.1, 1.3, size=(h, 3 * w)).astype(np.float32)
    kw = dict(LENSES[name])
    if h == 481:
        kw["vignetting_k"] = (-0.3, 0.05, -0.01)
    ex = OpticsExecution(w, h, **kw)
    ref = oracle.optics_apply(oracle.optics_desc_from(ex.to_c()), rgb)
    ours = stages.optics(rgb, ex)
    assert np.array_equal(ours.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("height", [8, 9, 15, 17])
def test_table_branch_at_tile_edges(stages, oracle, height):
    from rohditor_gb300 import OpticsExecution

    w = 70
    rgb = np.random.default_rng(height).uniform(0.0, 1.0, size=(height, 3 * w)).astype(np.float32)
    ex = OpticsExecution(w, height, distortion="poly5", distortion_k=(-0.02, 0.005, 0.0), tca="linear",
                         tca_red=(1.0003, 0, 0), tca_blue=(0.9997, 0, 0), vignetting_k=(-0.3, 0.05, -0.01))
    ref = oracle.optics_apply(oracle.optics_desc_from(ex.to_c()), rgb)
    ours = stages.optics(rgb, ex)
    assert np.array_equal(ours.view(np.uint32), ref.view(np.uint32))
