"""Nearly singular quadrilaterals of FP32 quadrature into complex64 where the
polar scheme's angles and the static part meet their limits, against the
oracle: a flat plate (every collocation point in its neighbours' planes and on
the lines of their sides), stretched plates, a folded pair of plates, distorted
quads, and points close above an element.

Tolerance: the FP32 mode's bar, 1e-5 of the largest entry per matrix.
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu

QUAD = int(meshes.cube_sphere(2)[1][0, 0])


def plate(nx, ny, fold=0.0, stretch=1.0):
    """nx x ny squares in the plane z = 0, the half x > 0 turned up by the angle fold."""
    x, y = np.meshgrid(np.arange(nx + 1.0) - nx // 2, stretch * np.arange(ny + 1.0), indexing="ij")
    up = np.maximum(x, 0)
    nodes = np.stack([np.where(x > 0, x * np.cos(fold), x), y, up * np.sin(fold)], axis=-1).reshape(-1, 3) * 0.1
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    a = (i * (ny + 1) + j).ravel()
    el = np.stack([np.full(a.size, QUAD), a, a + ny + 1, a + ny + 2, a + 1], axis=1)
    return nodes, np.ascontiguousarray(el.astype(np.int32))


def distorted():
    nodes, el = meshes.cube_sphere(5)
    rng = np.random.default_rng(7)
    return nodes + 0.05 * (rng.random(nodes.shape) - 0.5), el


MESHES = {"plate": lambda: plate(6, 5), "stretched": lambda: plate(4, 4, stretch=1.7), "folded": lambda: plate(6, 4, fold=1.2),
          "nearly flat": lambda: plate(6, 4, fold=1e-6), "distorted": distorted, "one": lambda: plate(1, 1)}


def assemble(ctx, test, mesh, family, k):
    trial = g.api.DeviceMesh(ctx, *mesh)
    tm = trial if test is mesh else g.api.DeviceMesh(ctx, *test)
    out = [np.zeros((tm.n, trial.n), np.complex64, order="F") for _ in range(2)]
    ctx.check(g.lib().nihu_gb_assemble(ctx.handle, tm.handle, trial.handle, family, g.SLP | g.DLP, k, 1.0, 0.0, g.REGULAR_FP32,
                                       g.C64, *(ctypes.c_void_p(o.ctypes.data) for o in out), tm.n, 0, g.HOST))
    return out


def check(ctx, oracle, test, mesh, k):
    family, fam = (g.HELMHOLTZ_3D, oracle.HELMHOLTZ) if k else (g.LAPLACE_3D, oracle.LAPLACE)
    S, D = assemble(ctx, test, mesh, family, k)
    s = oracle.assemble(test, mesh, fam, oracle.SLP, k, threads=8)
    d = oracle.assemble(test, mesh, fam, oracle.DLP, k, threads=8)
    assert np.abs(S - s).max() <= 1e-5 * np.abs(s).max()
    # a flat plate's DLP vanishes: against the size of a DLP next to an element, 1/2
    assert np.abs(D - d).max() <= 1e-5 * max(np.abs(d).max(), 0.5)


@pytest.mark.parametrize("k", [0.0, 3.0])
@pytest.mark.parametrize("name", MESHES)
def test_one_mesh(gpu_ctx, oracle, name, k):
    mesh = MESHES[name]()
    check(gpu_ctx, oracle, mesh, mesh, k)


@pytest.mark.parametrize("k", [0.0, 3.0])
@pytest.mark.parametrize("shift", [(0, 0, 0.02), (0.05, 0, 0.03), (0.05, 0.05, 0.04), (0.031, -0.047, 0.05), (0.05, 0.012, -0.02)])
def test_points_above(gpu_ctx, oracle, shift, k):
    # above the middle, a side, a corner and elsewhere
    mesh = plate(5, 5)
    check(gpu_ctx, oracle, (mesh[0] + np.array(shift), mesh[1]), mesh, k)


@pytest.mark.parametrize("k", [0.0, 3.0])
@pytest.mark.parametrize("n", [3, 14, 18, 30])
def test_lanes_by_number_of_pairs(gpu_ctx, oracle, n, k):
    # 54 to 5400 quads: four lanes a pair, two, and (from about 7 000 quads) one;
    # rows of two ends of the mesh
    mesh = meshes.cube_sphere(n)
    if n < 30:
        return check(gpu_ctx, oracle, mesh, mesh, k)
    family, fam = (g.HELMHOLTZ_3D, oracle.HELMHOLTZ) if k else (g.LAPLACE_3D, oracle.LAPLACE)
    S, D = assemble(gpu_ctx, mesh, mesh, family, k)
    for rows in ((0, 40), (len(mesh[1]) - 40, len(mesh[1]))):
        s = oracle.assemble(mesh, mesh, fam, oracle.SLP, k, rows=rows, threads=8)
        d = oracle.assemble(mesh, mesh, fam, oracle.DLP, k, rows=rows, threads=8)
        assert np.abs(S[rows[0]:rows[1]] - s).max() <= 1e-5 * np.abs(s).max()
        assert np.abs(D[rows[0]:rows[1]] - d).max() <= 1e-5 * np.abs(d).max()
