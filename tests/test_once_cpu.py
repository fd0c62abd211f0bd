"""Kernel attributes are set once per device, before any thread's first launch, and again after a failure.  Needs no GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_set_once_per_device_over_a_fake_runtime(tmp_path):
    exe = str(tmp_path / "once_fake")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-x", "c++", "-I/usr/local/cuda/include", "-I" + os.path.join(HERE, "..", "include"),
                           "-o", exe, os.path.join(HERE, "once_fake.cpp")])
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout == "ok\n"
