"""Kernels that are launched as so many thread blocks per SM have the registers
for it, as the compiler reports them (65 536 a multiprocessor, in units of
eight a thread)."""
import os
import re
import shutil
import subprocess

import pytest

from nihu_gb300 import build

BLOCKS, THREADS = 3, 128  # k_pairs_singular: assemble_pairs.cu's launch


@pytest.mark.skipif(not shutil.which(build.nvcc()), reason="no nvcc")
def test_pair_lists_singular_kernel(tmp_path):
    out = subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-Xptxas", "-v", "-cubin",
                          os.path.join(build.CSRC, "assemble_pairs.cu"), "-o", str(tmp_path / "pairs.cubin")],
                         capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    used = re.findall(r"entry function '\S*k_pairs_singular\S*'.*?Used (\d+) registers", out.stderr, re.S)
    assert len(used) == 4  # two output types, real and complex wave numbers
    for n in used:
        assert -(-int(n) // 8) * 8 * THREADS * BLOCKS <= 65536
