"""device_slab.hpp: pieces from what a slab has free, on the CPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_a_slab_asked_not_to_grow_does_not(tmp_path):
    exe = tmp_path / "slab_room"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", str(exe),
                    os.path.join(HERE, "cpp", "slab_room_driver.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr
