"""Raw levels in the tiled demosaics, and RCD's two arithmetic forms.

Black levels that repeat every one or two samples are applied cell by cell, other
patterns sample by sample; crops lie on and off the grid that tensor copies need.
RCD divides without special cases while every sample is of a magnitude up to
2^20. Results equal the oracle's bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALGORITHMS = {"bilinear": 0, "mhc": 1, "rcd": 2}
PATTERNS = {"RGGB": 0, "BGGR": 1, "GRBG": 2, "GBRG": 3}


def scene(w, h, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    return np.clip(0.4 + 0.3 * np.sin(x / 11.0) * np.cos(y / 7.0) + rng.normal(0, 0.05, (h, w)), -0.02, 1.2).astype(np.float32)


@pytest.mark.parametrize("algorithm", sorted(ALGORITHMS))
@pytest.mark.parametrize("repeat", [(1, 1), (2, 1), (1, 2), (2, 2), (4, 4)])
@pytest.mark.parametrize("crop", [None, (8, 3, 200, 150), (5, 4, 203, 151)])
@pytest.mark.parametrize("cfa", ["RGGB", "GBRG"])
def test_levels_by_position(device, oracle, algorithm, repeat, crop, cfa):
    from rohditor_gb300 import GpuSensorProcessor, SensorDescription, clip_levels

    w, h = 240, 170
    rng = np.random.default_rng(sum(repeat))
    black = tuple(float(v) for v in rng.uniform(0.0, 300.0, repeat[0] * repeat[1]).astype(np.float32))
    raw = np.clip(np.rint(150 + scene(w, h, 9) * (4095 - 150)), 0, 4095).astype(np.uint16)
    levels = clip_levels(1.0, (2.0, 1.0, 1.6))
    desc = SensorDescription(w, h, cfa=cfa, crop=crop, black=black, black_repeat=repeat, white=(4095.0,),
                             highlight="clip", clip_levels=levels, demosaic=algorithm,
                             demosaic_balance=(1.0, 1.0, 1.0))
    src = GpuSensorProcessor(device).develop(raw, desc)
    m, pattern = oracle.normalize(raw, oracle.sensor_desc(w, h, w, crop or (0, 0, w, h), PATTERNS[cfa], list(black),
                                                          repeat, [4095.0]))
    table = {0: [0, 1, 1, 2], 1: [2, 1, 1, 0], 2: [1, 0, 2, 1], 3: [1, 2, 0, 1]}[pattern]
    y, x = np.mgrid[0:m.shape[0], 0:m.shape[1]]
    ceiling = np.array(levels, np.float32)[np.array(table)[((y & 1) << 1) | (x & 1)]]
    ref = oracle.demosaic(np.minimum(m, ceiling), pattern, (1.0, 1.0, 1.0), ALGORITHMS[algorithm])
    assert np.array_equal(src.download().view(np.uint32), np.ascontiguousarray(ref).view(np.uint32))
    src.release()


@pytest.mark.parametrize("factor", [0.0, 2.0**-60, 2.0**-33, 1.0, 2.0**19, 2.0**20, 2.0**21, 2.0**40])
@pytest.mark.parametrize("size", [(200, 120), (97, 131)])
def test_rcd_magnitudes(stages, oracle, factor, size):
    m = scene(*size, seed=3)
    m[20:60, 30:90] *= np.float32(factor)  # both forms, and their boundary, in one image
    m[70:80, 10:40] = 0.0
    ref = oracle.demosaic(m, 2, (1.0, 1.0, 1.0), 2)
    out = stages.demosaic(m, "GRBG", "rcd")
    assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))
