"""The transforms of two real rows of csrc/fft_real.cuh on the host, lanes emulated."""
import os
import subprocess

from util import ROOT


def test_transforms_of_two_real_rows(tmp_path):
    exe = str(tmp_path / "fft_real_host_check")
    # fused multiply-adds as the device compiler makes them
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-march=native", "-ffp-contract=fast", "-I/usr/local/cuda/include",
                           os.path.join(ROOT, "tests", "host", "fft_real_host_check.cpp"), "-o", exe])
    vals = {k: float(v) for k, v in (line.split() for line in subprocess.check_output([exe], text=True).strip().splitlines())}
    # rms of a rounding 2.5e-8: eight levels of additions 7e-8, two factors (their own rounding and a product's) 6e-8, one
    # more addition to separate or join the rows: 9.4e-8 in independent directions; a quarter more for the estimate
    assert set(vals) == {"forward128", "inverse128", "forward256", "inverse256"}
    assert all(v <= 1.2e-7 for v in vals.values()), vals
