"""GMRES of one system (the step kernel): sizes at the edges of its row slices
(32 rows a CTA, one CTA per SM at most), short restarts, a guess, a zero
residual, the iteration limit, against numpy's dense solve.

Tolerance: the stopping rule bounds the residual by 1e-10 of its start, so the
solution of these well-conditioned systems (condition below 10) is within 1e-8;
a complex64 matrix is the exact one here, its products round at 6e-8 per term
of 32-column sums, which leaves the solution within 1e-5.
"""
import numpy as np
import pytest

import nihu_gb300 as g

pytestmark = pytest.mark.gpu


def system(n, dtype, seed=0):
    rng = np.random.default_rng([n, seed])
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * (0.3 / np.sqrt(2 * n)) + np.eye(n)
    A = np.asfortranarray(A.astype(dtype))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return A, b, np.linalg.solve(A.astype(np.complex128), b)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 321, 1024, 4865, 5000])
@pytest.mark.parametrize("dtype,tol", [(np.complex64, 1e-5), (np.complex128, 1e-8)])
@pytest.mark.parametrize("restart", [1, 3, 50])
def test_solution(gpu_ctx, n, dtype, tol, restart):
    A, b, ref = system(n, dtype)
    x, it, res = g.gmres(A, b, restart=restart, max_iters=400, tol=1e-6 if dtype == np.complex64 else 1e-10, ctx=gpu_ctx)
    assert np.linalg.norm(x - ref) <= tol * np.linalg.norm(ref)
    assert 1 <= it <= 400 and res < 1e-6


def test_guess_and_zero_residual(gpu_ctx):
    A, b, ref = system(200, np.complex128)
    x, it, res = g.gmres(A, b, x0=ref + 1e-3, tol=1e-10, ctx=gpu_ctx)
    assert np.linalg.norm(x - ref) <= 1e-8 * np.linalg.norm(ref)
    x, it, res = g.gmres(A, np.zeros(200), ctx=gpu_ctx)
    assert it == 0 and res == 0.0 and not x.any()


@pytest.mark.parametrize("restart", [4, 50])
def test_iteration_limit(gpu_ctx, restart):
    A, b, _ = system(300, np.complex128)
    with pytest.raises(g.NotConvergedError):
        g.gmres(A, b, restart=restart, max_iters=6, tol=1e-12, ctx=gpu_ctx)
