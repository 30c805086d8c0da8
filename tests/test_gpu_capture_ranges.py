"""Capture sharpening where its kernels' forms change over.

An iteration walks strips of 112 columns (120 for radii of one and two pixels)
and row segments down to 8 rows, with vector copies where rows are a multiple of
16 bytes; the widths below end just before, on and just after a strip's edge and
its margins. Quotients take a form without special cases up to 2^60 and for
ceilings between 2^-60 and 2^60; the levels lie on both sides. Results equal the
oracle's bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RADII = (0.3, 0.6, 0.9, 1.2)  # kernel radii 1 to 4


def run(stages, oracle, rgb, radius, noise, ceilings, iterations):
    from rohditor_gb300 import CaptureContract

    cap = CaptureContract(amount=0.8, radius=radius, noise_protection=noise, ceilings=ceilings, iterations=iterations)
    ours = stages.capture(rgb, cap)
    ref = oracle.capture(rgb, 0.8, radius, noise, ceilings, iterations)
    assert np.array_equal(ours.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("radius", RADII)
@pytest.mark.parametrize("width", [256, 331, 336, 340, 344, 360, 363, 364, 448, 452, 481])
def test_strip_edges(stages, oracle, width, radius):
    height = 64 + width % 23
    rng = np.random.default_rng(width)
    rgb = rng.uniform(-0.05, 1.3, size=(height, 3 * width)).astype(np.float32)
    run(stages, oracle, rgb, radius, 0.4, (1.0, 0.9, 1.1), 3)


@pytest.mark.parametrize("scale", [1e-30, 1e-7, 1.0, 2.0**58, 2.0**62, 1e30])
@pytest.mark.parametrize("noise", [0.0, 1.0])
def test_level_ranges(stages, oracle, scale, noise):
    rng = np.random.default_rng(3)
    rgb = rng.uniform(-0.2, 1.5, size=(70, 3 * 300)).astype(np.float32)
    rgb[10:30, 200:420] *= np.float32(scale)  # levels of both kinds, and their boundary, in one image
    run(stages, oracle, rgb, 0.7, noise, (1.0, 0.9, 1.1), 2)


@pytest.mark.parametrize("ceilings", [(2.0**-61, 1.0, 1.0), (2.0**-60, 2.0**60, 1e-3), (2.0**61, 0.5, 3.0), (1e30, 1e-30, 1.0)])
def test_ceiling_ranges(stages, oracle, ceilings):
    rng = np.random.default_rng(4)
    rgb = rng.uniform(-0.2, 1.5, size=(66, 3 * 260)).astype(np.float32)
    run(stages, oracle, rgb, 0.7, 0.3, ceilings, 2)


@pytest.mark.parametrize("iterations", [1, 2])
@pytest.mark.parametrize("width", [256, 333, 452])
@pytest.mark.parametrize("radius", RADII)
def test_gain_of_the_last_iteration(stages, oracle, radius, width, iterations):
    # The last iteration applies the gain itself: levels whose gained channels
    # overflow stay as they are, levels above 2^60 take the plain division.
    rng = np.random.default_rng(width + iterations)
    rgb = rng.uniform(-0.2, 1.5, size=(67, 3 * width)).astype(np.float32)
    rgb[20:26, 90:300] *= np.float32(2.0**61)
    rgb[40:44, 120:180] = rng.choice(np.float32([3.4e38, -3.4e38, 0.0]), size=(4, 60))
    run(stages, oracle, rgb, radius, 0.2, (1.0, 0.9, 1.1), iterations)
