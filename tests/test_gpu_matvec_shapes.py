"""Matvecs on both sides of the rule that splits their columns (256 or 32 at
least to a block): square, wide and tall, with columns left over.

Tolerance: complex64 sums at most 256 FP32 products a block, 6e-8 sqrt(256) of
the absolute sum, complex128 n eps of it.
"""
import numpy as np
import pytest

import nihu_gb300 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (33, 31), (320, 33), (511, 2049), (100, 5003), (1000, 20001), (20001, 1000), (5003, 100),
                                 (4001, 4000), (5120, 5121)])
@pytest.mark.parametrize("dtype,tol", [(np.complex64, 1e-6), (np.complex128, 1e-12)])
def test_shapes(gpu_ctx, m, n, dtype, tol):
    rng = np.random.default_rng([m, n])
    A = np.empty((m, n), dtype, order="F")
    A.real, A.imag = rng.random((m, n)), rng.random((m, n))
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    y = g.matvec(A, x, ctx=gpu_ctx)
    scale = np.abs(A).astype(float) @ np.abs(x)
    assert (np.abs(y - A.astype(complex) @ x) <= tol * scale).all()
