"""The PNG chunk checksum without a GPU: the shares and the tree that combines them
(deflate.cuh, driven as png_chunk_kernel drives them) against zlib, at lengths
around the edges of a share, of a warp's shares and of the largest chunk."""

import os
import shutil
import subprocess
import zlib

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHARE, LARGEST = 132, 32768 + 64 + 16


def test_shares_combine_to_the_crc(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "crc_host"
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", "-o", str(exe),
                    os.path.join(ROOT, "tests", "native", "crc_host.cpp")], check=True)
    data = np.random.default_rng(4).integers(0, 256, LARGEST, dtype=np.uint8).tobytes()
    (tmp_path / "data").write_bytes(data)
    lengths = [*range(1, 24), LARGEST - 1, LARGEST]
    for shares in (1, 2, 3, 31, 32, 33, 64, 128, 247, 248):
        lengths += [SHARE * shares + d for d in range(-5, 6)]
    out = subprocess.run([str(exe), str(tmp_path / "data"), *map(str, lengths)], capture_output=True, text=True,
                         check=True)
    assert [int(v) for v in out.stdout.split()] == [zlib.crc32(data[:n]) for n in lengths]
