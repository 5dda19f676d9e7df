"""The mixed-precision LU at the edges of its kernels: panels of 16 columns (the
last one ragged), 512 rows a thread block and up to eight blocks a cluster,
panels of 8 and 4 columns beyond 8192 and 16384 rows, solve blocks of 64 rows
round eight thread blocks.

Tolerance: backward error |A x - b| / (|A| |x|) <= 1e-13.  The refinement stops
when the correction is within 64 roundings of FP64; the residual itself is
formed in FP64, sqrt(n) eps <= 3e-14 of |A| |x| for n <= 16400.
"""
import re

import numpy as np
import pytest

import nihu_gb300 as g

pytestmark = pytest.mark.gpu


def rand_c(rng, *shape):
    x = np.empty(shape, complex)
    x.real = rng.random(shape)
    x.imag = rng.random(shape)
    x -= 0.5 + 0.5j
    return x


def backward_error(A, x, b):
    return np.linalg.norm(A @ x - b) / (np.linalg.norm(A) * np.linalg.norm(x))


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 63, 64, 65, 128, 129, 511, 512, 513, 527, 529, 577, 1024, 1025,
                               1041, 2049, 4100])
def test_orders(gpu_ctx, n):
    # random entries: nearly every column exchanges rows
    rng = np.random.default_rng(n)
    A, b = rand_c(rng, n, n), rand_c(rng, n)
    assert backward_error(A, g.lu_solve(A, b, ctx=gpu_ctx), b) <= 1e-13


@pytest.mark.parametrize("n", [8209, 16400])
def test_narrow_panels(gpu_ctx, n):
    rng = np.random.default_rng(n)
    A, b = rand_c(rng, n, n), rand_c(rng, n)
    x = g.lu_solve(A, b, ctx=gpu_ctx)
    assert backward_error(A, x, b) <= 1e-13


@pytest.mark.parametrize("n", [40, 700, 1300])
def test_exchanges_within_and_across_panels(gpu_ctx, n):
    # a scaled permutation plus noise: the pivot of column j is row perm[j], and
    # rows come back to earlier places; cycles inside and between the panels
    rng = np.random.default_rng(n)
    for perm in (np.arange(n)[::-1], np.roll(np.arange(n), 1), np.roll(np.arange(n), -17), rng.permutation(n)):
        A = 1e-3 * rand_c(rng, n, n)
        A[perm, np.arange(n)] += 2 + np.arange(n) / n
        b = rand_c(rng, n)
        x = g.lu_solve(A, b, ctx=gpu_ctx)
        ref = np.linalg.solve(A, b)
        assert np.abs(x - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n,col", [(5, 0), (100, 37), (600, 599), (1100, 16)])
def test_zero_column_is_named(gpu_ctx, n, col):
    rng = np.random.default_rng(n)
    A = rand_c(rng, n, n)
    A[:, col] = 0
    with pytest.raises(g.NihuError, match=re.escape(f"zero pivot in column {col})")):
        g.lu_solve(A, rand_c(rng, n), ctx=gpu_ctx)


def test_budget_without_room_for_the_inverses(gpu_ctx):
    # FP64 matrix, FP32 factors and the vectors fit, 1 KB a row more does not
    n = 600
    rng = np.random.default_rng(n)
    A, b = rand_c(rng, n, n), rand_c(rng, n)
    ctx = g.api.Context(hbm_budget_bytes=24 * n * n + 200 * n)
    assert backward_error(A, g.lu_solve(A, b, ctx=ctx), b) <= 1e-13
