"""Kept device blocks given back when an allocation fails.

A request beyond the device's memory fails in the pool, which makes the context
take back what every context keeps. Beside it, on other threads, contexts work
with kept blocks, captured batches are built and run, and served loops replace
their contexts' streams: all of it gives what it gives alone.
"""

import ctypes
import threading

import numpy as np
import pytest

from rohditor_gb300 import (CaptureContract, ColorContract, Device, OpticsExecution, SensorDescription, Stages,
                            clip_levels)
from rohditor_gb300.batch import BatchImage, develop_batch
from rohditor_gb300.served import PreviewServer
from rohditor_gb300.workloads import CAMERA_TO_REC2020, preview_dimensions

pytestmark = pytest.mark.gpu

RD_OVER_BUDGET = 3
BEYOND = 1 << 42  # bytes; no GPU has them


def sharpen(stages, seed=1, w=640, h=300):
    rgb = np.random.default_rng(seed).uniform(0.0, 1.2, size=(h, 3 * w)).astype(np.float32)
    return stages.capture(rgb, CaptureContract(amount=0.6, radius=0.7, noise_protection=0.4, ceilings=(1.0, 1.0, 1.0),
                                               iterations=3))


def refused(dev) -> bool:
    p = ctypes.c_void_p()
    return dev.lib.rd_device_alloc(dev.handle, BEYOND, ctypes.byref(p)) == RD_OVER_BUDGET


def images():
    wb = (2.0, 1.0, 1.6)
    out = []
    for k, (w, h) in enumerate(((512, 384), (700, 467))):
        raw = np.random.default_rng(k).integers(260, 4095, size=(h, w), dtype=np.uint16)
        sensor = SensorDescription(w, h, black=(256.0,), white=(4095.0,), highlight="clip",
                                   clip_levels=clip_levels(1.0, wb), demosaic="mhc", demosaic_balance=wb)
        cap = CaptureContract(amount=0.5, radius=0.7, noise_protection=0.5, ceilings=clip_levels(1.0, wb), iterations=3)
        optics = OpticsExecution(w, h, distortion="poly5", distortion_k=(-0.02, 0.005, 0.0))
        out.append(BatchImage(raw, sensor, cap, optics, preview_dimensions(w, h, 256), wb, CAMERA_TO_REC2020,
                              ColorContract(wb_gains=wb, camera_to_rec2020=CAMERA_TO_REC2020)))
    return out


def test_a_failed_allocation_leaves_other_contexts_usable():
    a, b = Device(0), Device(0)
    stages = Stages(b)
    want = sharpen(stages)
    for _ in range(3):
        assert refused(a)
        assert np.array_equal(sharpen(stages), want)
    a.close()
    b.close()


def test_failed_allocations_beside_captures_and_stream_changes():
    batch = images()
    want_batch = develop_batch(batch, lanes=1)[0]
    dev = Device(0)
    want = sharpen(Stages(dev))
    dev.close()
    wrong, stop = [], threading.Event()

    def run(name, work):
        try:
            work()
        except Exception as e:  # noqa: BLE001
            wrong.append(f"{name}: {e!r}")

    def failing():
        d = Device(0)
        while not stop.is_set():
            if not refused(d):
                wrong.append("an allocation beyond the device succeeded")
                break
        d.close()

    def sharpening():
        d = Device(0)
        stages = Stages(d)
        for _ in range(40):
            if not np.array_equal(sharpen(stages), want):
                wrong.append("sharpening")
        d.close()

    def capturing():
        for k in range(12):
            got = develop_batch(batch, lanes=2, graph=True, flat=k % 2 == 1)[0]
            for (x, hx), (y, hy) in zip(got, want_batch):
                if not (np.array_equal(x, y) and np.array_equal(hx, hy)):
                    wrong.append("captured batch")

    def serving():
        for _ in range(12):
            PreviewServer(0).close()

    workers = [threading.Thread(target=run, args=(f.__name__, f)) for f in (sharpening, capturing, serving)]
    other = threading.Thread(target=run, args=("failing", failing))
    for t in workers + [other]:
        t.start()
    for t in workers:
        t.join()
    stop.set()
    other.join()
    assert not wrong, wrong
