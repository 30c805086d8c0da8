"""AMaZE where its row-streamed pipeline and its two arithmetic forms change over.

A tile's stages take the branch-free division and the hardware's min / max while
every sample is 0 or of a magnitude in [2^-30, 2^20], and the IEEE forms from
the first sample outside it on; the sizes put the image's edge at the tile grid
(224-pixel cores, 16-pixel halo), and the dense patterns fill the queue of the
area interpolation. Every result equals the oracle's bit for bit, so no
tolerance is involved.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(w, h, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    m = 0.3 + 0.2 * np.sin(x / 37.0) + 0.15 * np.cos(y / 23.0) + rng.normal(0.0, 0.02, (h, w))
    return np.clip(m, 0.0, 1.2).astype(np.float32)


def stripes(w, h, seed):
    """Detail at the sampling limit: most red/blue sites are flagged by the Nyquist test."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    return (0.5 + 0.35 * np.cos(np.pi * (x + 0.4 * y)) + rng.normal(0.0, 0.01, (h, w))).astype(np.float32)


def check(stages, oracle, m, cfa="RGGB"):
    ref = oracle.demosaic(m, {"RGGB": 0, "BGGR": 1, "GRBG": 2, "GBRG": 3}[cfa], (1.0, 1.0, 1.0), 3)
    out = stages.demosaic(m, cfa, "amaze")
    assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("size", [(33, 33), (34, 225), (223, 224), (225, 33), (256, 239), (449, 450), (700, 241)])
@pytest.mark.parametrize("cfa", ["RGGB", "GRBG"])
def test_sizes_at_the_tile_grid(stages, oracle, size, cfa):
    check(stages, oracle, scene(*size, seed=size[0]), cfa)


@pytest.mark.parametrize("cfa", ["RGGB", "BGGR", "GRBG", "GBRG"])
def test_dense_nyquist_flags(stages, oracle, cfa):
    check(stages, oracle, stripes(512, 300, 3), cfa)


@pytest.mark.parametrize("factor", [2.0 ** -33, 2.0 ** -29, 2.0 ** -20, 2.0 ** 18, 2.0 ** 21, 2.0 ** 40])
def test_magnitudes_around_the_quick_forms_range(stages, oracle, factor):
    check(stages, oracle, scene(300, 280, 5) * np.float32(factor))


def test_single_samples_outside_the_range(stages, oracle):
    m = scene(600, 500, 7)
    m[::31, ::17] = 0.0  # within it
    m[250, 300] = 1.0e-15  # the first sample outside comes late in some tiles and never in others
    m[470, 20] = -3.0e-12
    m[5, 590] = 4.0e6
    check(stages, oracle, m)


def test_zero_negative_and_flat_areas(stages, oracle):
    m = scene(500, 460, 9)
    m[100:200, 50:300] = 0.0
    m[200:260, 50:300] = 0.25
    m[300:340] -= 0.5
    check(stages, oracle, m)
