"""The two-row Galerkin kernel rounds no more than the one-row kernel that takes
scaled and accumulating calls: both against the FP64 mode, beyond the near pairs
(their kernels are shared).

Tolerance: the same operations in another order of rows: root mean square errors
within 2% of one another (over 80 000 entries those of two roundings more would
differ by 4%).
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2.0, 5.0, 20.0])
def test_far_pairs(gpu_ctx, k):
    nodes, el = meshes.icosphere(2)
    q, _ = np.linalg.qr(np.random.default_rng(3).standard_normal((3, 3)))
    dm = g.api.DeviceMesh(gpu_ctx, nodes @ q.T, el)
    n, L = dm.n, g.lib()
    nnz = ctypes.c_int64()
    gpu_ctx.check(L.nihu_gb_near_pairs(gpu_ctx.handle, dm.handle, dm.handle, ctypes.byref(nnz), None, None))
    col, rows = np.zeros(n + 1, np.int64), np.zeros(nnz.value, np.int32)
    gpu_ctx.check(L.nihu_gb_near_pairs(gpu_ctx.handle, dm.handle, dm.handle, ctypes.byref(nnz), col.ctypes.data, rows.ctypes.data))
    far = ~np.eye(n, dtype=bool)
    far[rows, np.repeat(np.arange(n), np.diff(col))] = False

    def matrices(precision, dtype, accumulate):
        out = [np.zeros((n, n), np.complex64 if dtype == g.C64 else complex, order="F") for _ in range(2)]
        gpu_ctx.check(L.nihu_gb_assemble_galerkin(gpu_ctx.handle, dm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, k, 1.0,
                                                  0.0, precision, dtype, out[0].ctypes.data, out[1].ctypes.data, n, accumulate,
                                                  g.HOST))
        return [x.astype(complex)[far] for x in out]

    exact = matrices(g.REGULAR_FP64, g.C128, 0)
    two, one = (matrices(g.REGULAR_FP32, g.C64, accumulate) for accumulate in (0, 1))
    for x, y, ref in zip(two, one, exact):
        assert np.linalg.norm(x - ref) <= 1.02 * np.linalg.norm(y - ref)
