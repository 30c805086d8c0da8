"""Kept device blocks stay within the budget.

What a context has in use and what it keeps for its next calls stay within its
budget together, as the pool counts them, and a served loop within its own.
"""

import ctypes

import numpy as np
import pytest

from rohditor_gb300 import CaptureContract, Device, Stages

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def pool_use() -> int:
    """Bytes of the device's stream-ordered pool that are in use (kept blocks included)."""
    cu = ctypes.CDLL("libcuda.so.1")
    pool, value = ctypes.c_void_p(), ctypes.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, ctypes.byref(value)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return value.value


def sharpen(stages, w, h, seed=1):
    rgb = np.random.default_rng(seed).uniform(0.0, 1.2, size=(h, 3 * w)).astype(np.float32)
    return stages.capture(rgb, CaptureContract(amount=0.6, radius=0.7, noise_protection=0.4, ceilings=(1.0, 1.0, 1.0),
                                               iterations=3))


def test_in_use_and_kept_stay_within_the_budget():
    budget = 24 * MIB
    dev = Device(0, budget)
    stages = Stages(dev)
    before = pool_use()
    for k in range(24):  # about 6 MB each, no two alike
        sharpen(stages, 640 + 8 * k, 300)
        dev.synchronize()
        assert pool_use() - before <= budget
    dev.set_budget(8 * MIB)
    dev.synchronize()
    assert pool_use() - before <= 8 * MIB
    dev.close()


def test_trim_gives_kept_blocks_back():
    dev = Device(0)
    stages = Stages(dev)
    before = pool_use()
    want = sharpen(stages, 640, 300)
    dev.synchronize()
    kept = dev.kept_bytes
    assert kept >= 5 * MIB and pool_use() - before >= kept
    dev.trim(kept // 2)
    assert dev.kept_bytes <= kept // 2
    dev.trim()
    assert dev.kept_bytes == 0 and pool_use() <= before
    assert np.array_equal(sharpen(stages, 640, 300), want)
    dev.close()


def test_a_served_loop_keeps_within_its_budget():
    from rohditor_gb300 import OpticsExecution, SensorDescription, clip_levels
    from rohditor_gb300.served import PreviewServer
    from rohditor_gb300.workloads import CAMERA_TO_REC2020, preview_dimensions

    wb, budget = (2.0, 1.0, 1.6), 160 * MIB
    before = pool_use()
    server = PreviewServer(0, budget)
    for k in range(10):  # admitted at about 100 MB each, of which 11 MB stay resident
        w, h = 1024 + 16 * k, 768
        raw = np.random.default_rng(k).integers(260, 4095, size=(h, w), dtype=np.uint16)
        sensor = SensorDescription(w, h, black=(256.0,), white=(4095.0,), highlight="clip",
                                   clip_levels=clip_levels(1.0, wb), demosaic="mhc", demosaic_balance=wb)
        cap = CaptureContract(amount=0.5, radius=0.7, noise_protection=0.5, ceilings=clip_levels(1.0, wb), iterations=3)
        optics = OpticsExecution(w, h, distortion="poly5", distortion_k=(-0.02, 0.005, 0.0))
        server.open(k, raw, sensor, cap, optics, preview_dimensions(w, h, 256), wb, CAMERA_TO_REC2020)
        server.drain()
        assert pool_use() - before <= budget
    stats = server.stats()
    server.close()
    assert stats["evictions"] > 0
