"""FP64 quadrature on small meshes, whose columns are split into blocks of 1 to
32 by the number of rows: one column a block, uneven last blocks, a column
panel of a larger matrix, and the full 32, against the oracle.

Tolerance: the FP64 mode's 1e-11 of the largest entry.
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu


def part(n):
    nodes, el = meshes.icosphere(3)
    return nodes, np.ascontiguousarray(el[:n])


def rel(got, ref):
    return np.abs(got - ref).max() / max(np.abs(ref).max(), 1e-12)


def run(ctx, rows, cols, call):
    out = [np.full((rows, cols), 7 + 3j, np.complex128, order="F") for _ in range(2)]
    ctx.check(call(out[0].ctypes.data, out[1].ctypes.data))
    return out


# rows x columns: 16 blocks per SM put 1, 2, 3 and up to 32 columns in a block
SHAPES = [(1, 1), (1, 1280), (31, 33), (257, 300), (1280, 257), (1280, 1280)]


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("k", [2.0, 2.0 - 0.3j])
def test_collocation(gpu_ctx, oracle, rows, cols, k):
    nodes, el = part(rows)
    test, mesh = (nodes * 1.3, el), part(cols)
    dm, tm = g.api.DeviceMesh(gpu_ctx, *mesh), g.api.DeviceMesh(gpu_ctx, *test)
    k = complex(k)
    S, D = run(gpu_ctx, rows, cols, lambda a, b: g.lib().nihu_gb_assemble_c(
        gpu_ctx.handle, tm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, k.real, k.imag, 1.0, 0.0, g.REGULAR_FP64, g.C128,
        ctypes.c_void_p(a), ctypes.c_void_p(b), rows, 0, g.HOST))
    kk = k if k.imag else k.real
    assert rel(S, oracle.assemble(test, mesh, oracle.HELMHOLTZ, oracle.SLP, kk, threads=8)) <= 1e-11
    assert rel(D, oracle.assemble(test, mesh, oracle.HELMHOLTZ, oracle.DLP, kk, threads=8)) <= 1e-11


@pytest.mark.parametrize("n", [1, 33, 257, 1280])
def test_burton_miller(gpu_ctx, oracle, n):
    mesh = part(n)
    dm = g.api.DeviceMesh(gpu_ctx, *mesh)
    c = 0.2 - 0.4j
    A, B = run(gpu_ctx, n, n, lambda a, b: g.lib().nihu_gb_assemble_burton_miller(
        gpu_ctx.handle, dm.handle, g.HELMHOLTZ_3D, 3.0, c.real, c.imag, g.REGULAR_FP64, g.C128, ctypes.c_void_p(a),
        ctypes.c_void_p(b), n, g.HOST))
    S, D, T, H = (oracle.assemble(mesh, mesh, oracle.HELMHOLTZ, op, 3.0, threads=8)
                  for op in (oracle.SLP, oracle.DLP, oracle.DLPT, oracle.HSP))
    assert rel(A, D + c * H - 0.5 * np.eye(n)) <= 1e-11
    assert rel(B, S + c * T + c / 2 * np.eye(n)) <= 1e-11


@pytest.mark.parametrize("rows,cols", SHAPES[:-1])
def test_galerkin(gpu_ctx, oracle, rows, cols):
    nodes, el = part(rows)
    test, mesh = (nodes * 1.3, el), part(cols)
    dm, tm = g.api.DeviceMesh(gpu_ctx, *mesh), g.api.DeviceMesh(gpu_ctx, *test)
    S, D = run(gpu_ctx, rows, cols, lambda a, b: g.lib().nihu_gb_assemble_galerkin(
        gpu_ctx.handle, tm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, 3.0, 1.0, 0.0, g.REGULAR_FP64, g.C128,
        ctypes.c_void_p(a), ctypes.c_void_p(b), rows, 0, g.HOST))
    assert rel(S, oracle.assemble_galerkin(test, mesh, oracle.HELMHOLTZ, oracle.SLP, 3.0, threads=8)) <= 1e-11
    assert rel(D, oracle.assemble_galerkin(test, mesh, oracle.HELMHOLTZ, oracle.DLP, 3.0, threads=8)) <= 1e-11
