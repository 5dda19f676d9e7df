"""A GMRES cycle of more steps than the step kernel has threads (256), through
the composite solve, whose restart has no bound of its own below 2048.

The mesh is 600 large triangles thrown into the unit cube: every one is near
most others, the matrix DLP - I/2 has no clustered spectrum (condition number
1.1e4) and needs about 410 steps at 1e-8.

Tolerance: the stopping rule bounds the residual by 1e-8 of the right-hand
side, up to the loss of orthogonality of the FP64 basis (CGS2: a few eps), and
the matrices the solve assembles are the ones compared with: 2e-8.  The solution
is then within the condition number times that, 2.2e-4.
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu


def soup(n, seed=0):
    rng = np.random.default_rng(seed)
    centre = rng.random((n, 1, 3))
    nodes = (centre + rng.random((n, 3, 3)) - 0.5).reshape(-1, 3)
    return meshes._pack(nodes, np.arange(3 * n).reshape(n, 3), meshes.TRIA_1)


@pytest.mark.parametrize("restart", [500, 600])
def test_more_than_256_steps(gpu_ctx, restart):
    mesh, k = soup(600), 2.0
    n = len(mesh[1])
    S, D = (np.zeros((n, n), complex, order="F") for _ in range(2))
    dm = g.api.DeviceMesh(gpu_ctx, *mesh)
    gpu_ctx.check(g.lib().nihu_gb_assemble(gpu_ctx.handle, dm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, k, 1.0, 0.0,
                                           g.REGULAR_FP64, g.C128, S.ctypes.data, D.ctypes.data, n, 0, g.HOST))
    rng = np.random.default_rng(1)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    A, b = D - 0.5 * np.eye(n), S @ q
    p, it, res = g.solve_cbie(g.create_mesh(*mesh), k, q, dtype=g.C128, precision="fp64", restart=restart,
                              max_iters=restart, tol=1e-8, ctx=gpu_ctx)
    assert 256 < it <= 500 and res < 1e-8
    assert np.linalg.norm(A @ p - b) <= 2e-8 * np.linalg.norm(b)
    ref = np.linalg.solve(A, b)
    assert np.linalg.norm(p - ref) <= 2.2e-4 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [63, 64, 65, 97, 255, 256])
def test_every_step_of_a_cycle(gpu_ctx, n):
    # a cyclic shift in a random unitary basis, from its first basis vector: the
    # residual stays what it is for n - 1 steps
    rng = np.random.default_rng(n)
    U = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    A, b = np.asfortranarray(np.roll(U, 1, axis=1) @ U.conj().T), U[:, 0].copy()
    x, it, res = g.gmres(A, b, restart=n, max_iters=n, tol=1e-10, ctx=gpu_ctx)
    assert it == n and np.linalg.norm(A @ x - b) <= 1e-10


@pytest.mark.parametrize("n", [321, 4900])
def test_cycles_beyond_a_vector_per_thread(gpu_ctx, n):
    # eigenvalues in a disc of radius 0.9 about 1: about a factor of 0.9 a step
    rng = np.random.default_rng(n)
    A = np.empty((n, n), complex, order="F")
    A.real, A.imag = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    A *= 0.9 / np.sqrt(2 * n)
    A[np.arange(n), np.arange(n)] += 1
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x, it, res = g.gmres(A, b, restart=200, max_iters=200, tol=1e-6, ctx=gpu_ctx)
    assert 65 <= it <= 200 and res < 1e-6
    assert np.linalg.norm(A @ x - b) <= 2e-6 * np.linalg.norm(b)
