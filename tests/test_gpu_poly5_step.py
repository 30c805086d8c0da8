"""The Poly5 closed form where the second-order term of its second step vanishes.

One Newton step from the input radius r leaves F(r - q) = q^2 (3 a r + 10 b r^3) -
q^3 (a + 10 b r^2) + q^4 5 b r - q^5 b. With a and b of opposite signs the first
term has a zero, around which the second one decides whether the iteration stops
there. The lens below has that ring inside the image, and a TCA polynomial whose
flips keep the radial table from serving it.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_second_step_is_taken_where_the_second_order_term_vanishes(stages, oracle, sign):
    from rohditor_gb300 import OpticsExecution, _ffi

    w, h = 1201, 901
    ex = OpticsExecution(w, h, distortion="poly5", distortion_k=(0.0282599 * sign, -0.00308406 * sign, 0.0), tca="poly3",
                         tca_red=(1.0002, 0.0001, -0.0001), tca_blue=(0.9998, -0.0001, 0.0001), real_focal=10.0)
    desc = ex.to_c()
    knots, step, guard = np.zeros((1024, 4), dtype=np.float32), ctypes.c_float(), ctypes.c_int32()
    assert _ffi.load().rd_optics_radial_table(ctypes.byref(desc), knots.ctypes.data_as(_ffi.F32P), ctypes.byref(step),
                                              ctypes.byref(guard)) == 0
    assert guard.value > 0  # refused: the pixels take the Newton path
    rgb = np.random.default_rng(5).uniform(0.0, 1.0, size=(h, 3 * w)).astype(np.float32)
    ref = oracle.optics_apply(oracle.optics_desc_from(desc), rgb)
    ours = stages.optics(rgb, ex)
    assert np.array_equal(ours.view(np.uint32), ref.view(np.uint32))
