"""Field points of a trial mesh whose columns, 16 to a thread block, are more
than the 65 535 blocks a grid's second dimension takes: the two-row kernels of
the collocation and Galerkin matrices, against the oracle on the columns about
the line where the launch is split, the first and the last ones.

Tolerance: the FP32 mode's bar, 1e-5 of the largest entry per matrix.
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes
from test_gpu_two_row import on_device, rel

pytestmark = pytest.mark.gpu

SPLIT = 65535 * 16
N = SPLIT + 37
W = 725  # nodes along a side


def plate():
    """N triangles of 1/724 in the plane z = 0."""
    y, x = np.divmod(np.arange(W * (W + 1)), W)
    nodes = np.column_stack([x, y, np.zeros(len(x))]) / (W - 1.0)
    cell = np.arange((N + 1) // 2)
    a = cell // (W - 1) * W + cell % (W - 1)
    faces = np.stack([np.column_stack([a, a + 1, a + W]), np.column_stack([a + 1, a + W + 1, a + W])], 1)
    return meshes._pack(nodes, faces.reshape(-1, 3)[:N], meshes.TRIA_1)


def rows_above(trial):
    """Three of its triangles, lifted off it: above the first, the split's and the last column."""
    nodes, el = trial
    corners = nodes[el[[0, SPLIT, N - 1], 1:4]] + np.array([0.0, 0.0, 0.003])
    return meshes._pack(corners.reshape(-1, 3), np.arange(9).reshape(3, 3), meshes.TRIA_1)


@pytest.mark.parametrize("galerkin", [False, True])
def test_columns_beyond_one_grid(gpu_ctx, oracle, galerkin):
    trial = plate()
    test = rows_above(trial)
    dm, tm = g.api.DeviceMesh(gpu_ctx, *trial), g.api.DeviceMesh(gpu_ctx, *test)
    L = g.lib()
    call = L.nihu_gb_assemble_galerkin if galerkin else L.nihu_gb_assemble
    k = 6.0
    got = on_device(gpu_ctx, 3, N, 1, lambda a, b, ld: call(
        gpu_ctx.handle, tm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, k, 1.0, 0.0, g.REGULAR_FP32, g.C64, a, b, ld, 0,
        g.DEVICE))
    cols = np.r_[0:60, SPLIT - 60:N]
    part = trial[0], np.ascontiguousarray(trial[1][cols])
    for out, op in zip(got, (oracle.SLP, oracle.DLP)):
        assert np.isfinite(out).all() and (out != np.complex64(7 + 3j)).all()
        ref = (oracle.assemble_galerkin(test, part, oracle.HELMHOLTZ, op, k, threads=8) if galerkin else
               oracle.assemble(test, part, oracle.HELMHOLTZ, op, k, same_mesh=False, threads=8))
        assert rel(out[:, cols], ref) <= 1e-5
