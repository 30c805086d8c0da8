"""Opposed where its kernels' forms change over.

A tile of 16 x 8 cells with up to six suspected samples has them estimated by a
warp each, one with more stages its cells for a thread each; the scenes hold
single hot pixels, clusters of five to eight in a tile, blown areas, and all of
them at the image's edges and odd sizes. The cell pass takes levels by position
(one value, 1 x 2 to 2 x 2 patterns) in one form and any other pattern in the
general one. Statistics and region labels equal the oracle's, samples agree to
the bound of the existing comparison (1e-4: libm's cube root and logarithm, and
the order of the region sums, are not the device's).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEVELS = ((0.987,) * 3, (0.6, 0.98, 0.75))


def scene(w, h, seed, per_tile):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    m = (0.45 + 0.3 * np.sin(x / 19.0) * np.cos(y / 13.0) + rng.normal(0, 0.03, (h, w))).astype(np.float32)
    m = np.clip(m, 0.01, 0.9)
    for ty in range(0, h, 16):
        for tx in range(0, w, 32):
            n = per_tile if per_tile >= 0 else int(rng.integers(0, 12))
            for _ in range(n):
                m[min(ty + int(rng.integers(0, 16)), h - 1), min(tx + int(rng.integers(0, 32)), w - 1)] = rng.uniform(0.99, 1.5)
    return m


def compare(stages, oracle, m, cfa, ceiling):
    det = LEVELS[0]
    ours, stats, labels, count = stages.opposed(m, cfa, det, ceiling)
    ref, ref_stats, ref_labels, ref_count = oracle.opposed(m, {"RGGB": 0, "BGGR": 1, "GRBG": 2, "GBRG": 3}[cfa], det, ceiling)
    assert count == ref_count and np.array_equal(labels, ref_labels)
    assert stats.tolist() == ref_stats.tolist()
    assert float(np.max(np.abs(ours - ref))) <= 1e-4


@pytest.mark.parametrize("per_tile", [1, 5, 6, 7, -1])
@pytest.mark.parametrize("cfa", ["RGGB", "GBRG"])
def test_sites_per_tile(stages, oracle, per_tile, cfa):
    compare(stages, oracle, scene(333, 211, per_tile + 7, per_tile), cfa, LEVELS[1])


@pytest.mark.parametrize("size", [(2, 2), (3, 5), (31, 17), (32, 16), (33, 33)])
def test_small_and_odd_sizes(stages, oracle, size):
    m = scene(*size, seed=2, per_tile=3)
    m[-1, -1] = 1.3
    compare(stages, oracle, m, "GRBG", None)


def test_blown_area_beside_hot_pixels(stages, oracle):
    m = scene(400, 300, 5, 2)
    m[60:140, 100:220] = 1.2
    m[290:, 380:] = 1.1
    compare(stages, oracle, m, "BGGR", LEVELS[1])


@pytest.mark.parametrize("repeat", [(1, 1), (2, 1), (1, 2), (2, 2), (4, 2), (4, 4), (3, 1)])
@pytest.mark.parametrize("crop", [None, (13, 7, 203, 151)])
def test_level_patterns(device, oracle, repeat, crop):
    from rohditor_gb300 import GpuSensorProcessor, SensorDescription, opposed_levels

    w, h = 240, 170
    rng = np.random.default_rng(sum(repeat))
    black = tuple(float(v) for v in rng.uniform(200.0, 300.0, repeat[0] * repeat[1]).astype(np.float32))
    raw = np.clip(np.rint(256 + scene(w, h, 9, 2) * (4095 - 256)), 0, 4095).astype(np.uint16)
    det, ceiling = opposed_levels(1.0, (2.0, 1.0, 1.6))
    desc = SensorDescription(w, h, cfa="RGGB", crop=crop, black=black, black_repeat=repeat, white=(4095.0,),
                             highlight="opposed", detection_levels=det, neutral_ceiling=ceiling, demosaic="bilinear",
                             demosaic_balance=(2.0, 1.0, 1.6))
    src = GpuSensorProcessor(device).develop(raw, desc)
    odesc = oracle.sensor_desc(w, h, w, crop or (0, 0, w, h), 0, list(black), repeat, [4095.0])
    m, pattern = oracle.normalize(raw, odesc)
    m, stats, _, _ = oracle.opposed(m, pattern, det, ceiling)
    ref = oracle.demosaic(m, pattern, (2.0, 1.0, 1.6), 0)
    assert list(src.metrics.highlight_stats) == stats.tolist()
    assert float(np.max(np.abs(src.download() - ref))) <= 1e-4
    src.release()
