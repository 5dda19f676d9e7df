"""Memory budgets that hold a call's vectors and no more: what each call takes is
stated here to the byte, and a context with that budget still makes it.

    matvec  16 m per split, one split for 256 columns
    gmres   the basis 16 n (r + 1), the matvec's partial sums, two vectors 32 n,
            and 16 (r + 1) for each 1024 rows and once more
    LU      the FP32 factors 8 n^2, the row order 4 n, two vectors 32 n, 16,
            and the matvec's partial sums

The caller's arrays belong to another context.  Results as without a budget:
FP64 throughout, conditions below 1e3, so 1e-10.
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import _capi as C
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu

CTX = 16  # a context's own device memory


class Arrays:
    """Device copies of host arrays, in ctx."""

    def __init__(self, ctx, *host):
        self.ctx, self.host, self.ptr = ctx, host, []
        for h in host:
            p = ctypes.c_void_p()
            ctx.check(g.lib().nihu_gb_device_alloc(ctx.handle, h.nbytes, ctypes.byref(p)))
            self.ptr.append(p)
            ctx.check(g.lib().nihu_gb_memcpy(ctx.handle, p, C.DEVICE, h.ctypes.data, C.HOST, h.nbytes))

    def __enter__(self):
        return self.ptr

    def __exit__(self, *_):
        for p in self.ptr:
            g.lib().nihu_gb_device_free(self.ctx.handle, p)

    def read(self, i):
        out = np.empty_like(self.host[i])
        self.ctx.check(g.lib().nihu_gb_memcpy(self.ctx.handle, out.ctypes.data, C.HOST, self.ptr[i], C.DEVICE, out.nbytes))
        return out


def partials(n):
    return 16 * n * max(1, n // 256)


def gmres_bytes(n, restart):
    return 16 * n * (restart + 1) + partials(n) + 32 * n + 16 * (restart + 1) * (min(-(-n // 1024), 64) + 1)


def system(n):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * (0.3 / np.sqrt(2 * n)) + np.eye(n)
    return np.asfortranarray(A), rng.standard_normal(n) + 1j * rng.standard_normal(n)


def rel(x, ref):
    return np.linalg.norm(x - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("n", [1, 300, 1280, 2000])
def test_matvec(gpu_ctx, n):
    A, x = system(n)
    ctx = g.Context(hbm_budget_bytes=CTX + partials(n))
    dev = Arrays(gpu_ctx, A, x, np.zeros(n, complex))
    with dev as (a, b, y):
        ctx.check(g.lib().nihu_gb_matvec(ctx.handle, g.C128, a, n, n, n, b, y, 1.0, 0.0, 0.0, 0.0, g.DEVICE))
        assert rel(dev.read(2), A @ x) <= 1e-13


@pytest.mark.parametrize("n,restart", [(2, 1), (2, 2), (33, 33), (320, 50), (1280, 50), (1280, 256), (2000, 7), (300, 256)])
def test_gmres(gpu_ctx, n, restart):
    A, b = system(n)
    ctx = g.Context(hbm_budget_bytes=CTX + gmres_bytes(n, restart))
    dev = Arrays(gpu_ctx, A, b, np.zeros(n, complex))
    it, res = ctypes.c_int(0), ctypes.c_double(0.0)
    with dev as (a, rhs, x):
        ctx.check(g.lib().nihu_gb_gmres(ctx.handle, g.C128, a, n, n, rhs, x, restart, 400, 1e-12, ctypes.byref(it),
                                        ctypes.byref(res), g.DEVICE))
        assert rel(dev.read(2), np.linalg.solve(A, b)) <= 1e-10


@pytest.mark.parametrize("n", [12, 64, 600, 1280, 2000])
def test_lu(gpu_ctx, n):
    A, b = system(n)
    ctx = g.Context(hbm_budget_bytes=CTX + 8 * n * n + 4 * n + 32 * n + 16 + partials(n))
    ctx.check(g.lib().nihu_gb_ctx_set_profiling(ctx.handle, 1))
    dev = Arrays(gpu_ctx, A, b, np.zeros(n, complex))
    with dev as (a, rhs, x):
        ctx.check(g.lib().nihu_gb_lu_solve(ctx.handle, a, n, n, rhs, x, g.DEVICE))
        assert rel(dev.read(2), np.linalg.solve(A, b)) <= 1e-10
    assert "lu_factor" in phases(ctx) and "lu_factor_fp64" not in phases(ctx)  # the budget has room for the fast path


def phases(ctx):
    name, ms, launches = ctypes.c_char_p(), ctypes.c_double(), ctypes.c_int64()
    out, i = set(), 0
    while g.lib().nihu_gb_ctx_profile(ctx.handle, i, ctypes.byref(name), ctypes.byref(ms), ctypes.byref(launches)) == C.OK:
        out.add(name.value.decode())
        i += 1
    return out


@pytest.mark.parametrize("n", [64, 1280])
def test_lu_without_room_for_the_factors(gpu_ctx, n):
    # the FP64 factorisation is in place and needs the row order alone
    A, b = system(n)
    ctx = g.Context(hbm_budget_bytes=CTX + 4 * n)
    dev = Arrays(gpu_ctx, A, b, np.zeros(n, complex))
    with dev as (a, rhs, x):
        ctx.check(g.lib().nihu_gb_lu_solve(ctx.handle, a, n, n, rhs, x, g.DEVICE))
        assert rel(dev.read(2), np.linalg.solve(A, b)) <= 1e-10


@pytest.mark.parametrize("solver", ["gmres", "lu"])
def test_composite_solve(solver):
    # both matrices, three vectors, and what the solver takes; the near pairs' list first
    mesh, k = meshes.icosphere(3), 2.0
    n = len(mesh[1])
    q = np.ones(n, complex)
    probe = g.Context()
    dm = g.api.DeviceMesh(probe, *mesh)
    nnz = ctypes.c_int64()
    L = g.lib()
    probe.check(L.nihu_gb_near_pairs(probe.handle, dm.handle, dm.handle, ctypes.byref(nnz), None, None))
    held = L.nihu_gb_ctx_device_bytes(probe.handle)
    p = np.zeros(n, complex)
    it, res = ctypes.c_int(0), ctypes.c_double(0.0)

    def solve(ctx, m):
        ctx.check(L.nihu_gb_solve_cbie(ctx.handle, m.handle, g.HELMHOLTZ_3D, k, g.REGULAR_FP64, g.C128,
                                       q.ctypes.data, p.ctypes.data, int(solver == "lu"), 50, 200, 1e-12,
                                       ctypes.byref(it), ctypes.byref(res)))
        return p.copy()

    ref = solve(probe, dm)
    own = gmres_bytes(n, 50) if solver == "gmres" else 8 * n * n + 4 * n + 32 * n + 16 + 2 * partials(n)
    ctx = g.Context(hbm_budget_bytes=held + 32 * n * n + 48 * n + own)
    m = g.api.DeviceMesh(ctx, *mesh)
    ctx.check(L.nihu_gb_near_pairs(ctx.handle, m.handle, m.handle, ctypes.byref(nnz), None, None))
    assert rel(solve(ctx, m), ref) <= 1e-10
