"""The RL launch shape is fixed only when every candidate has been timed.

A develop times its iterations between the first and the last. With three
iterations that is one, so the candidates of a tall image (two or more segment
counts) need several develops; the shape is reported after the last of them, and
no result depends on it.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_few_iterations_time_all_candidates_before_the_shape_is_fixed(stages):
    from rohditor_gb300 import CaptureContract, rl_launch_shape

    w, h, radius = 16384, 1280, 0.7  # a round of work items is 16 segments of 80 rows; 32 of 40 is the second candidate
    rgb = np.random.default_rng(9).uniform(0.05, 0.9, size=(h, 3 * w)).astype(np.float32)
    cap = CaptureContract(amount=0.6, radius=radius, noise_protection=0.3, ceilings=(1.0, 1.0, 1.0), iterations=3)
    assert rl_launch_shape(w, h, radius) is None
    first = stages.capture(rgb, cap)
    assert rl_launch_shape(w, h, radius) is None  # one of at least two candidates is timed
    shape = None
    for _ in range(3):
        assert np.array_equal(stages.capture(rgb, cap).view(np.uint32), first.view(np.uint32))
        shape = shape or rl_launch_shape(w, h, radius)
    assert shape is not None and 0.0 < shape.best_ms <= shape.default_ms
    assert shape.segments % shape.default_segments == 0
    assert rl_launch_shape(w, h, radius) == shape
