"""A camera sample's pixel and sub-sample without 64-bit divisions, against plain division: every small divisor, those
around powers of two, the largest, and samples on both sides of 2^32 (host code, no GPU)."""
import os
import subprocess

from azimuth_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_sample_of_is_plain_division(tmp_path):
    exe = str(tmp_path / "sample_of_check")
    subprocess.check_call([build.NVCC, "-std=c++17", "-O1"] + build.ARCH + build.INCLUDES +
                          [os.path.join(HERE, "sample_of_check.cu"), "-o", exe])
    run = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout
