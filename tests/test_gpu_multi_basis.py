"""The Gram-Schmidt passes of the lockstep GMRES (four basis vectors a block,
coefficients staged 64 at a time, an FP32 copy of the basis) at the edges of
their tiles: rows around the block's 256 and its split, single and several
right-hand sides, a basis longer than a tile, and a context with a memory
budget, which keeps no copy.

Tolerance: the solver's own, 1e-6 on the relative residual; formed here in FP64
against a complex64 matrix, whose products it accumulates in FP32 (1e-7 sqrt(n)
of the residual's terms): 1e-5.
"""
import numpy as np
import pytest

import nihu_gb300 as g

pytestmark = pytest.mark.gpu


def rand_c(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def solve(ctx, n, nrhs, spread, restart=50):
    rng = np.random.default_rng(n + nrhs)
    A = (np.eye(n) + spread * rand_c(rng, n, n) / np.sqrt(2 * n)).astype(np.complex64)
    B = rand_c(rng, n, nrhs)
    X, outer, inner, res = g.solve_multi(A, B, inner_mode=g.GEMM_BF16X9, tol=1e-6, inner_tol=1e-5, restart=restart, ctx=ctx)
    err = np.linalg.norm(A.astype(np.complex128) @ X - B, axis=0) / np.linalg.norm(B, axis=0)
    assert res.max() <= 1e-6 and err.max() <= 1e-5
    return X, inner


@pytest.mark.parametrize("n", [1, 2, 5, 255, 256, 257, 1030, 2049, 2300])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_sizes(gpu_ctx, n, nrhs):
    solve(gpu_ctx, n, nrhs, 0.5)


def test_basis_longer_than_a_tile(gpu_ctx):
    _, inner = solve(gpu_ctx, 600, 2, 0.95, restart=200)
    assert inner > 64


def test_with_a_memory_budget(gpu_ctx):
    ctx = g.api.Context(hbm_budget_bytes=1 << 30)
    X, _ = solve(ctx, 700, 3, 0.5)
    Y, _ = solve(gpu_ctx, 700, 3, 0.5)
    assert np.abs(X - Y).max() <= 1e-6 * np.abs(Y).max()


@pytest.mark.parametrize("n", [257, 600, 2049])
def test_with_the_copy(gpu_ctx, n):
    # n nrhs >= 32768 values keep the FP32 copy
    solve(gpu_ctx, n, -(-32768 // n), 0.5)
