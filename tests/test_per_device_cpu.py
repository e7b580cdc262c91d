"""Kernel function attributes are set for every device of a process: the once-per-device helper, compiled and run on the CPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, os.pardir, "cl-eden-kernel_b200", "csrc")


def test_set_up_once_per_device(tmp_path):
    exe = str(tmp_path / "per_device_test")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-I", CSRC, os.path.join(HERE, "per_device_test.cpp"), "-o", exe, "-pthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
