"""JPEG packing where its symbol loop changes over.

The packing visits a block's non-zero coefficients by masks of the even and the
odd ones: blocks with a single coefficient at every place, runs of zeros up to
three codes long, a full block, and intervals whose bits end anywhere in a word
(one block to a few intervals). Decoding gives the oracle's coefficients.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def encoder(device):
    from rohditor_gb300 import JpegEncoder

    return JpegEncoder(device)


def cosine_block(v, u, amplitude):
    y, x = np.mgrid[0:8, 0:8]
    return amplitude * np.cos((2 * x + 1) * u * np.pi / 16) * np.cos((2 * y + 1) * v * np.pi / 16)


def check(encoder, oracle, image, quality):
    got = oracle.jpeg_decode(encoder.encode(image, quality))
    assert np.array_equal(got["coef"], oracle.jpeg_coefficients(image, quality))


@pytest.mark.parametrize("quality", [20, 75, 100])
def test_single_frequencies(encoder, oracle, quality):
    blocks = [np.clip(128 + cosine_block(v, u, 90), 0, 255) for v in range(8) for u in range(8)]
    grey = np.concatenate([np.concatenate(blocks[8 * r : 8 * r + 8], axis=1) for r in range(8)], axis=0)
    check(encoder, oracle, np.repeat(np.rint(grey)[:, :, None], 3, axis=2).astype(np.uint8), quality)


@pytest.mark.parametrize("width", [8, 16, 8 * 31, 8 * 32, 8 * 33, 8 * 65])
@pytest.mark.parametrize("quality", [3, 60, 100])
def test_intervals_of_any_length(encoder, oracle, width, quality):
    rng = np.random.default_rng(width)
    image = rng.integers(0, 256, (8, width, 3), dtype=np.uint8)
    image[:, : width // 2] //= 16  # blocks of few and of many symbols side by side
    check(encoder, oracle, image, quality)
