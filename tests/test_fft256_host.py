"""The 256-sample forward transform of csrc/fft256.cuh on the host, lanes emulated."""
import os
import subprocess

from util import ROOT


def test_error_of_the_one_exchange_transform(tmp_path):
    exe = str(tmp_path / "fft256_host_check")
    # fused multiply-adds as the device compiler makes them
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=fast", "-I/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "host", "fft256_host_check.cpp"), "-o", exe])
    vals = {k: float(v) for k, v in (line.split() for line in subprocess.check_output([exe], text=True).strip().splitlines())}
    # |X| is O(sqrt(256)) for unit-variance input; 2e-5 absolute is ~1e-6 relative
    assert vals["max"] < 2e-5
    # no further from the exact transform than the 32-point form of the same rows; two rms values of 25600 errors each
    # agree to 1 / sqrt(25600) = 0.6 % where the errors are equally large
    assert vals["rms256"] <= 1.02 * vals["rms32"], vals
