"""The RL iteration's bounded copy wait, made to run out.

Images below 256 x 64 iterate in rl_stream_kernel, whose inner strips' rows arrive
by tensor copy; their guide and mask pass has none. With the first copy of every
block withheld the iteration's own wait must give up, and the context stay usable.
"""

import numpy as np
import pytest

from rohditor_gb300 import CaptureContract, GpuPreviewError

pytestmark = pytest.mark.gpu

RD_INVALID_INPUT, RD_WAIT_NONE, RD_WAIT_RL_COPY = 8, 0, 2


@pytest.mark.parametrize("radius", [0.33, 0.7, 1.2])
def test_iteration_copy_wait_runs_out_and_the_context_stays_usable(device, stages, oracle, radius):
    w, h = 640, 48  # rows of 2560 bytes, strips of 120 to 126 columns: the second to fifth lie inside the image
    rgb = np.random.default_rng(12).uniform(0.02, 0.9, size=(h, 3 * w)).astype(np.float32)
    cap = CaptureContract(amount=0.6, radius=radius, noise_protection=0.4, ceilings=(1.0, 1.0, 1.0), iterations=3)
    ref = oracle.capture(rgb, cap.amount, cap.radius, cap.noise_protection, cap.ceilings, cap.iterations)
    device.check(device.lib.rd_ctx_set_wait_test(device.handle, 2000, RD_WAIT_RL_COPY))
    try:
        with pytest.raises(GpuPreviewError) as err:
            stages.capture(rgb, cap)
    finally:
        device.check(device.lib.rd_ctx_set_wait_test(device.handle, 0, RD_WAIT_NONE))
    assert err.value.code == RD_INVALID_INPUT
    assert "tensor copy timed out" in str(err.value)
    out = stages.capture(rgb, cap)
    assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))
