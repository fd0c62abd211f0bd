"""The staging area (hx_stage.cu) over a CUDA runtime written for the test: what it copies, what a call that fails leaves behind, and
when it gives its workspace back.  Needs no GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_staging_over_a_fake_runtime(tmp_path):
    exe = str(tmp_path / "stage_fake")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-x", "c++", "-I/usr/local/cuda/include", "-I" + os.path.join(HERE, "..", "include"),
                           "-o", exe, os.path.join(HERE, "stage_fake.cpp")])
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout == "ok\n"
