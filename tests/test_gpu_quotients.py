"""The division without special cases equals the IEEE one.

The kernels that are bit-exact against the oracle divide through a refined
hardware reciprocal; the device checks compare it with the IEEE division, for
every divisor significand with hard and hashed numerators, and for every
constant divisor with every numerator significand.
"""

import pytest

pytestmark = pytest.mark.gpu


def test_quotients_of_sampled_pairs_are_the_ieee_ones(stages):
    assert stages.check_math(5) == 0


def test_quotients_by_the_constants_are_the_ieee_ones(stages):
    assert stages.check_math(6) == 0
