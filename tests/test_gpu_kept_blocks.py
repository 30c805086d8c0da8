"""A context's kept device blocks and its pinned upload area.

Blocks that a call frees serve the next allocations of the same size, uploads
pass through a bounded pinned area: sizes that alternate, several contexts and
threads at once, more uploads than the area holds and a budget below what is
kept must give what a fresh context gives.
"""

import threading

import numpy as np
import pytest

from rohditor_gb300 import CaptureContract, Device, GpuPreviewError, Stages

from test_gpu_output import adjustments
from rohditor_gb300 import OutputSpec

pytestmark = pytest.mark.gpu

SIZES = ((640, 300), (333, 257), (640, 300), (800, 129))


def image(w, h, seed):
    return np.random.default_rng(seed).uniform(0.0, 1.2, size=(h, 3 * w)).astype(np.float32)


def sharpened(stages, w, h, seed):
    cap = CaptureContract(amount=0.6, radius=0.7, noise_protection=0.4, ceilings=(1.0, 1.0, 1.0), iterations=3)
    return stages.capture(image(w, h, seed), cap)


def fresh():
    out = []
    for k, (w, h) in enumerate(SIZES):
        dev = Device(0)
        out.append(sharpened(Stages(dev), w, h, k))
        dev.close()
    return out


def test_alternating_sizes_in_one_context():
    want = fresh()
    dev = Device(0)
    stages = Stages(dev)
    for _ in range(4):
        for k, (w, h) in enumerate(SIZES):
            assert np.array_equal(sharpened(stages, w, h, k), want[k])
    dev.close()


def test_contexts_on_several_threads():
    want, wrong = fresh(), []

    def work(k):
        dev = Device(0)
        stages = Stages(dev)
        for _ in range(6):
            if not np.array_equal(sharpened(stages, *SIZES[k], k), want[k]):
                wrong.append(k)
        dev.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(SIZES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_more_uploads_than_the_area_holds(stages):
    rgb = image(301, 97, 5)
    spec = OutputSpec(format="srgb8")
    want = [stages.output(rgb, adjustments(exposure_ev=0.1 * k), spec, histogram=False)[0] for k in range(3)]
    for k in range(40):  # two tables of 16 KB each
        got = stages.output(rgb, adjustments(exposure_ev=0.1 * (k % 3)), spec, histogram=False)[0]
        assert np.array_equal(got, want[k % 3])


def test_budget_counts_what_is_in_use_not_what_is_kept():
    dev = Device(0)
    stages = Stages(dev)
    want = sharpened(stages, 640, 300, 1)
    dev.set_budget(1 << 20)  # the kept blocks would do, the working set is refused
    with pytest.raises(GpuPreviewError):
        sharpened(stages, 640, 300, 1)
    dev.set_budget(64 << 20)
    assert np.array_equal(sharpened(stages, 640, 300, 1), want)
    dev.close()
