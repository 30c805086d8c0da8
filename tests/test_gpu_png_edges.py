"""PNG encoding where its kernels' forms change over.

Scanlines are filtered in tiles of 8192 bytes staged by 16-byte copies, so the
widths below end just before, on and after a tile, and an image starts off a
16-byte boundary. The encoder's chunks of 32 bytes are all literals unless a run
of three repeated bytes touches them: runs of every length up to a few chunks
start at every place of one. The inflated stream equals the oracle's filtered
scanlines, checksums included, and decodes to the input.
"""

import ctypes

import numpy as np
import pytest

from pngfile import decode

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def encoder(device):
    from rohditor_gb300 import PngEncoder

    return PngEncoder(device)


def check(png, oracle, image):
    got = decode(png, oracle)
    assert got["stream"] == oracle.png_filter(image)
    assert np.array_equal(got["pixels"], image)


def noise(h, w, dtype, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    base = (x[..., None] * (3, 1, 2) + y[..., None] * (1, 5, 3)) * 7
    return ((base + rng.integers(0, 40, (h, w, 3))) % (np.iinfo(dtype).max + 1)).astype(dtype)


@pytest.mark.parametrize("dtype,widths", [(np.uint8, (2, 3, 2730, 2731, 5461, 5462)),
                                          (np.uint16, (2, 3, 1365, 1366, 2730, 2731))])
def test_tile_edges(encoder, oracle, dtype, widths):
    for w in widths:
        for h in (1, 2, 5):
            image = noise(h, w, dtype, w + h)
            check(encoder.encode(image, b"", None), oracle, image)


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_runs_of_every_length_and_place(encoder, oracle, dtype):
    rng = np.random.default_rng(7)
    line = []
    for length in list(range(1, 12)) + [30, 31, 32, 33, 34, 63, 64, 65, 257, 258, 259, 260, 261, 516, 520]:
        for gap in range(1, 34, 3):
            line += list(rng.integers(1, 250, gap)) + [int(rng.integers(0, 256))] * length
    flat = np.array(line + [7] * (-len(line) % 6), dtype=np.uint8)
    rows = flat.reshape(1, -1, 3) if dtype == np.uint8 else flat.view(">u2").astype(np.uint16).reshape(1, -1, 3)
    for image in (rows, np.concatenate([rows, rows[:, ::-1]])):
        image = np.ascontiguousarray(image)
        check(encoder.encode(image, b"", None), oracle, image)


def test_rows_off_a_copy_boundary(device, encoder, oracle):
    import torch

    image = noise(9, 1501, np.uint8, 3)
    room = encoder.bound(1501, 9, 8, 0, 0)
    for offset in (1, 7, 13):
        store = torch.zeros(image.size + 32, dtype=torch.uint8, device="cuda")
        store[offset : offset + image.size] = torch.from_numpy(image.reshape(-1)).cuda()
        out = torch.zeros(room, dtype=torch.uint8, device="cuda")
        size = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        device.check(device.lib.rd_encode_png_device(
            device.handle, ctypes.c_void_p(store.data_ptr() + offset), 1501, 9, 3 * 1501, 8, None, 0, None, 0,
            ctypes.c_void_p(out.data_ptr()), room, ctypes.c_void_p(size.data_ptr())))
        device.synchronize()
        check(out[: int(size[0])].cpu().numpy().tobytes(), oracle, image)
