"""The plan build's device memory pieces (device_slab.hpp) against a fake
allocator, on the CPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_pieces_never_overlap_and_are_given_back(tmp_path, seed):
    exe = tmp_path / "slab"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", str(exe),
                    os.path.join(HERE, "cpp", "slab_driver.cpp")], check=True)
    r = subprocess.run([str(exe), str(seed)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr
