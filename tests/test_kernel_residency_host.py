"""Registers of the FP32 contraction: two CTAs of 256 threads share an SM's 65536 and nothing is spilled."""
import os
import re
import subprocess

from turbofno_b200.build import CSRC, NVCC_FLAGS


def test_fp32_contraction_fits_an_sm_twice(tmp_path):
    src = tmp_path / "contraction.cu"
    src.write_text('#include "%s"\ntemplate __global__ void tfno::spectral_tile_kernel<2, false, false, 1>(tfno::TileParams);\n' % os.path.join(CSRC, "spectral_kernels.cuh"))
    log = subprocess.run(["nvcc"] + NVCC_FLAGS + ["-Xptxas", "-v", "-c", str(src), "-o", str(tmp_path / "contraction.o")],
                         check=True, capture_output=True, text=True).stderr
    entry = log[log.index("spectral_tile_kernel"):]
    registers, spilled = int(re.search(r"Used (\d+) registers", entry).group(1)), int(re.search(r"(\d+) bytes spill stores", entry).group(1))
    assert (registers + 7) // 8 * 8 * 256 * 2 <= 65536 and spilled == 0, log
