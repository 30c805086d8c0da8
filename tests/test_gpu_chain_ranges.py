"""The adjustment chain and the transfer where their forms change over.

Pixels that stay finite and below 2^20 take a form of the chain without special
cases, all others the general one; the thresholds lie at the magnitudes, tiny
channels, zero and negative luminances, hues at the band centres, equal channels
and targets near the blend's transition drawn below. 8- and 16-bit codes come
from an estimate of the transfer that is decided exactly near a boundary between
two codes. Results equal the oracle's exact arithmetic bit for bit.
"""

import numpy as np
import pytest

from rohditor_gb300 import OutputSpec

from test_gpu_output import adjustments, oracle_output, same_bits

pytestmark = pytest.mark.gpu


def edge_image():
    rng = np.random.default_rng(5)
    mags = [0.0, -0.0, 1e-38, 1e-30, 2.0**-41, 2.0**-40, 2.0**-39, 1e-7, 1e-6, 4e-6, 1e-4, 0.02, 0.0031308, 0.5, 1.0,
            1.0 + 2.0**-23, 4.0, 2.0**19, 2.0**20, 2.0**21, 1e30, 3e38, np.inf, np.nan]
    a = rng.choice(mags, size=(40, 61, 3)) * rng.choice((1.0, 1.0, -1.0), size=(40, 61, 3))
    grey = rng.uniform(-0.05, 1.2, size=(8, 61, 1)) * np.ones(3)              # equal channels
    near = rng.uniform(-2e-6, 2e-6, size=(8, 61, 3))                          # luminances about the 1e-6 bound
    low = rng.uniform(-0.03, 0.05, size=(8, 61, 3))                           # targets about the transition
    k = np.arange(61)
    hue = np.stack([np.stack([np.ones(61), k / 60.0, np.zeros(61)], 1), np.stack([np.zeros(61), np.ones(61), k / 60.0], 1),
                    np.stack([k / 60.0, np.zeros(61), np.ones(61)], 1), np.stack([np.ones(61), np.zeros(61), k / 60.0], 1)])
    tiny = np.stack([np.ones(61), np.zeros(61), 2.0 ** -(k + 20.0)], 1)[None]  # a hue next to a whole turn
    img = np.concatenate([a, grey, near, low, hue, tiny]).astype(np.float32)
    return np.ascontiguousarray(img).reshape(img.shape[0], -1)


EDITS = {
    "none": dict(exposure_ev=0.0, base_lut=None, tone_lut=None, saturation=1.0, vibrance=0.0, hsl=None),
    "tables": dict(saturation=1.0, vibrance=0.0, hsl=None),
    "hsl": dict(exposure_ev=0.0, base_lut=None, tone_lut=None, saturation=1.0, vibrance=0.0),
    "all": dict(light=True, grading=True),
    "strong": dict(exposure_ev=4.0, saturation=-3.0, vibrance=1.0, hsl_scale=8.0, grading=True),
}


@pytest.mark.parametrize("fmt", ["srgb8", "srgb16", "extended_f32"])
@pytest.mark.parametrize("policy", ["clip", "chroma_compress"])
@pytest.mark.parametrize("edit", sorted(EDITS))
def test_chain_forms_equal_the_oracle(stages, oracle, edit, policy, fmt):
    from rohditor_gb300 import light_tone_lut
    from rohditor_gb300.workloads import hsl_bands

    kw = dict(EDITS[edit])
    if kw.pop("light", False):
        kw["light_tone_lut"] = light_tone_lut(0.5, -0.6, 0.4, -1.0, 0.3)
    if kw.pop("grading", False):
        kw["grading"] = np.random.default_rng(9).uniform(-1, 1, (3, 3)).astype(np.float32)
    scale = kw.pop("hsl_scale", None)
    if scale:
        kw["hsl"] = (np.asarray(hsl_bands(3), np.float32) * scale).astype(np.float32)
    color = adjustments(**kw)
    rgb = edge_image()
    spec = OutputSpec(format=fmt, primaries="srgb", policy=policy, headroom=2.5,
                      dither="ordered8x8" if fmt == "srgb16" else "none")
    ours, _, gamut = stages.output(rgb, color, spec, histogram=False)
    ref, ref_gamut = oracle_output(oracle, rgb, color, spec, exact=True)
    assert same_bits(ours, ref)
    assert np.array_equal(gamut, ref_gamut)
