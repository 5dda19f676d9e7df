"""The two-row kernels round no more than the one-row kernels that scaled and
accumulating calls (Galerkin) and frequency batches (collocation) take: both
against the FP64 mode, beyond the near pairs.

Tolerance: the same operations in another order of rows: root mean square errors
within 2% of one another (a rounding that the points of a rule share instead of
averaging it makes 6 to 17%).
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu

MESHES = {"triangles": meshes.icosphere(2), "quads": meshes.cylinder(32, 18, 2)}


class Case:
    def __init__(self, ctx, name):
        nodes, el = MESHES[name]
        q, _ = np.linalg.qr(np.random.default_rng(3).standard_normal((3, 3)))
        self.ctx, self.dm = ctx, g.api.DeviceMesh(ctx, nodes @ q.T, el)
        n, L = self.dm.n, g.lib()
        nnz = ctypes.c_int64()

        def near(c, r):
            ctx.check(L.nihu_gb_near_pairs(ctx.handle, self.dm.handle, self.dm.handle, ctypes.byref(nnz), c, r))

        near(None, None)
        col, rows = np.zeros(n + 1, np.int64), np.zeros(nnz.value, np.int32)
        near(col.ctypes.data, rows.ctypes.data)
        self.far = ~np.eye(n, dtype=bool)
        self.far[rows, np.repeat(np.arange(n), np.diff(col))] = False

    def matrices(self, dtype, call):
        n = self.dm.n
        out = [np.zeros((n, n), np.complex64 if dtype == g.C64 else complex, order="F") for _ in range(2)]
        self.ctx.check(call(out[0].ctypes.data, out[1].ctypes.data, n))
        return [x.astype(complex)[self.far] for x in out]


def check(two, one, exact):
    for x, y, ref in zip(two, one, exact):
        assert np.linalg.norm(x - ref) <= 1.02 * np.linalg.norm(y - ref)


@pytest.mark.parametrize("k", [0.0, 2.0, 5.0, 20.0])
def test_galerkin_quads(gpu_ctx, k):
    c = Case(gpu_ctx, "quads")
    family = g.HELMHOLTZ_3D if k else g.LAPLACE_3D

    def run(precision, dtype, accumulate):
        return c.matrices(dtype, lambda a, b, n: g.lib().nihu_gb_assemble_galerkin(
            gpu_ctx.handle, c.dm.handle, c.dm.handle, family, g.SLP | g.DLP, k, 1.0, 0.0, precision, dtype, a, b, n, accumulate,
            g.HOST))

    check(run(g.REGULAR_FP32, g.C64, 0), run(g.REGULAR_FP32, g.C64, 1), run(g.REGULAR_FP64, g.C128, 0))


@pytest.mark.parametrize("mesh", MESHES)
@pytest.mark.parametrize("k", [0.0, 2.0, 5.0, 20.0])
def test_collocation(gpu_ctx, mesh, k):
    c = Case(gpu_ctx, mesh)
    family = g.HELMHOLTZ_3D if k else g.LAPLACE_3D
    h, m, L, n = gpu_ctx.handle, c.dm.handle, g.lib(), c.dm.n

    def run(precision, dtype):
        return c.matrices(dtype, lambda a, b, ld: L.nihu_gb_assemble(h, m, m, family, g.SLP | g.DLP, k, 1.0, 0.0, precision, dtype,
                                                                     a, b, ld, 0, g.HOST))

    # a batch of one wave number, into device memory
    out, ptr, ks = [], [ctypes.c_void_p(), ctypes.c_void_p()], np.array([k])
    for p in ptr:
        gpu_ctx.check(L.nihu_gb_device_alloc(h, 8 * n * n, ctypes.byref(p)))
    gpu_ctx.check(L.nihu_gb_assemble_sweep(h, m, m, family, g.SLP | g.DLP, ks.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                                           len(ks), g.REGULAR_FP32, g.C64, ptr[0], ptr[1], n, n * n))
    for p in ptr:
        x = np.zeros((n, n), np.complex64, order="F")
        gpu_ctx.check(L.nihu_gb_memcpy(h, x.ctypes.data, g.HOST, p, g.DEVICE, x.nbytes))
        L.nihu_gb_device_free(h, p)
        out.append(x.astype(complex)[c.far])
    check(run(g.REGULAR_FP32, g.C64), out, run(g.REGULAR_FP64, g.C128))
