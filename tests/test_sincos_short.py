"""The FP32 sine and cosine series of the Galerkin near pairs, compiled for the
host from the kernel's source: within |x| <= 1.57, where the kernel takes them,
no further from the exact values than the CUDA library's FP32 functions may be.

Tolerance: those are given as 2 ulp, 1.2e-7 beside values up to 1; and on
average at the end of the range, where roundings cancel, a quarter of one.
"""
import ctypes
import os
import re
import subprocess

import numpy as np

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nihu_gb300", "csrc", "assemble_galerkin.cu")


def test_series(tmp_path):
    text = open(SRC).read()
    body = re.search(r"__device__ __forceinline__ void sincos_short\(.*?\n}\n", text, re.S).group(0)
    c = tmp_path / "series.cpp"
    c.write_text("#include <cmath>\n#define __device__\n#define __forceinline__ inline\n" + body +
                 'extern "C" void eval(int n, const float *x, float *s, float *c)\n'
                 "{\n    for (int i = 0; i < n; ++i) sincos_short(x[i], true, s[i], c[i]);\n}\n")
    lib = tmp_path / "series.so"
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", str(c), "-o", str(lib)], check=True)
    x = np.concatenate([np.linspace(-1.57, 1.57, 200001), np.linspace(1.5, 1.57, 20001)]).astype(np.float32)
    s, k = np.empty_like(x), np.empty_like(x)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    ctypes.CDLL(str(lib)).eval(len(x), ptr(x), ptr(s), ptr(k))
    d = x.astype(float)
    for got, exact in ((s, np.sin(d)), (k, np.cos(d))):
        assert np.abs(got - exact).max() <= 1.2e-7
        # a quarter of a rounding where the next term of the series is largest
        assert abs((got - exact)[d > 1.5].mean()) <= 1.5e-8
