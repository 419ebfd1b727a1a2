"""The FP64 near field's kernel evaluation (green64.cuh) on the CPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_special_values_and_errors(tmp_path):
    exe = tmp_path / "green64"
    subprocess.run(["g++", "-std=gnu++17", "-O2", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "cpp", "green64_driver.cpp"), "-lquadmath"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr
