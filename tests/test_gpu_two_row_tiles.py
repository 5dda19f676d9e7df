"""The two-row kernels where a block has more columns than one flush of its lists
(8): 12 columns (1283 elements), 16 (2003, the last block three), and rows at the
edges of a block (256), against the oracle on bands of rows: the first, the ones
about every block edge, the last.

A block takes (row blocks) x (columns) / (4 x SMs) columns, up to 16; the sizes
here ask for 152 SMs or fewer to reach what they name.

Tolerance: the FP32 mode's bar, 1e-5 of the largest entry per matrix (here of
the bands).
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes
from test_gpu_galerkin_two_row import galerkin
from test_gpu_two_row import collocation, on_device, rel

pytestmark = pytest.mark.gpu

SIZES = [255, 256, 257, 1283, 2003]


def part(n):
    nodes, el = meshes.icosphere(4)
    return nodes, np.ascontiguousarray(el[:n])


def bands(n):
    edges = [(0, 12)] + [(e - 4, e + 4) for e in range(256, n - 4, 256)] + [(n - 12, n)]
    return [(max(a, 0), min(b, n)) for a, b in edges]


def check(got, n, ref):
    rows = bands(n)
    want = np.concatenate([ref(r) for r in rows])
    assert rel(np.concatenate([got[a:b] for a, b in rows]), want) <= 1e-5


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("k", [0.0, 3.0, 2.0 - 0.4j])
def test_collocation(gpu_ctx, oracle, n, k):
    mesh = part(n)
    family, fam = (g.HELMHOLTZ_3D, oracle.HELMHOLTZ) if k else (g.LAPLACE_3D, oracle.LAPLACE)
    for out, op in zip(collocation(gpu_ctx, mesh, mesh, family, g.SLP | g.DLP, k), (oracle.SLP, oracle.DLP)):
        check(out, n, lambda r: oracle.assemble(mesh, mesh, fam, op, k, rows=r, threads=8))


@pytest.mark.parametrize("n", SIZES)
def test_burton_miller_system(gpu_ctx, oracle, n):
    mesh, k, c = part(n), 3.0, 0.2 - 0.4j
    dm = g.api.DeviceMesh(gpu_ctx, *mesh)
    A, B = on_device(gpu_ctx, n, n, 1, lambda a, b, ld: g.lib().nihu_gb_assemble_burton_miller(
        gpu_ctx.handle, dm.handle, g.HELMHOLTZ_3D, k, c.real, c.imag, g.REGULAR_FP32, g.C64, a, b, ld, g.DEVICE))
    one = np.eye(n)

    def ref(r, first, second, diagonal):
        op = [oracle.assemble(mesh, mesh, oracle.HELMHOLTZ, o, k, rows=r, threads=8) for o in (first, second)]
        return op[0] + c * op[1] + diagonal * one[r[0]:r[1]]

    check(A, n, lambda r: ref(r, oracle.DLP, oracle.HSP, -0.5))
    check(B, n, lambda r: ref(r, oracle.SLP, oracle.DLPT, c / 2))


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("k", [0.0, 3.0])
def test_galerkin(gpu_ctx, oracle, n, k):
    mesh = part(n)
    family, fam = (g.HELMHOLTZ_3D, oracle.HELMHOLTZ) if k else (g.LAPLACE_3D, oracle.LAPLACE)
    for out, op in zip(galerkin(gpu_ctx, mesh, mesh, family, g.SLP | g.DLP, k), (oracle.SLP, oracle.DLP)):
        check(out, n, lambda r: oracle.assemble_galerkin(mesh, mesh, fam, op, k, rows=r, threads=8))
