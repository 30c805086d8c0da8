"""The kept device blocks without a GPU: block_cache.cuh over a pool that counts
bytes and knows which streams live and which are being captured (see
tests/native/block_cache_host.cpp), the threads with the race detector."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = os.path.join(ROOT, "tests", "native", "block_cache_host.cpp")


def build(path, *flags):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    return subprocess.run([cxx, "-O1", "-g", "-std=c++17", "-Wall", "-pthread", *flags, "-o", str(path), SOURCE],
                          capture_output=True, text=True)


@pytest.mark.parametrize("scenario", ["reclaim", "captured", "refused", "room", "passed_by", "threads"])
def test_kept_blocks(tmp_path, scenario):
    exe = tmp_path / "block_cache_host"
    done = build(exe)
    assert done.returncode == 0, done.stderr
    run = subprocess.run([str(exe), scenario], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr


def test_kept_blocks_have_no_data_races(tmp_path):
    exe = tmp_path / "block_cache_host"
    if build(exe, "-fsanitize=thread").returncode != 0:
        pytest.skip("no thread sanitizer")
    run = subprocess.run([str(exe), "threads"], capture_output=True, text=True, timeout=300)
    if "unexpected memory mapping" in run.stderr:
        pytest.skip("the sanitizer does not start here")
    assert run.returncode == 0, run.stderr[-3000:]
