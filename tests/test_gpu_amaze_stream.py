"""AMaZE's two hand-offs between the phases of a tile.

Up to 76 tiles (one SM for each of the two phases) phase B follows phase A step
by step, and learns in the middle of a tile that a sample is outside the
branch-free forms' range; above that it starts when phase A is complete. The
sizes lie on both sides, the samples at the steps where phase B starts, runs and
ends. Every result equals the oracle's bit for bit, call after call.
"""

import numpy as np
import pytest

from test_gpu_amaze_ranges import check, scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(4256, 896), (1568, 2464)])  # 76 and 77 tiles
def test_tile_counts_on_both_sides(stages, oracle, size):
    check(stages, oracle, scene(*size, seed=11))


@pytest.mark.parametrize("row", [0, 3, 27, 28, 31, 36, 120, 223, 239])
def test_samples_outside_the_range_at_any_step(stages, oracle, row):
    m = scene(460, 256, 13)
    m[min(row, 255), 100::50] = 3.0e-14
    check(stages, oracle, m)


def test_call_after_call(stages, oracle):
    for seed in range(6):
        check(stages, oracle, scene(300 + 64 * seed, 280, seed))
