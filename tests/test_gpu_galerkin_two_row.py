"""The Galerkin kernels of FP32 quadrature into complex64 at the edges of their
tiles (64 rows a warp, 256 rows and up to 16 columns a block, flushes of 8
columns), with a leading dimension that allows no wide store, against the
oracle: each operator by itself and both, one mesh and two, triangles (their
near pairs have a kernel of their own) and quadrilaterals, and a wave number
beyond the short series of the near kernel.

Tolerance: the FP32 mode's bar, 1e-5 of the largest entry per matrix.  The
sums have FP32 terms only; a phase k r <= 80 rounds by 5e-6 of an entry, and
the entries at that distance are below 1e-2 of the largest.
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import _capi as C
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 64, 65, 129, 255, 257, 513]


def part(n):
    nodes, el = meshes.icosphere(3)
    return nodes, np.ascontiguousarray(el[:n])


def rel(got, ref):
    return np.abs(got - ref).max() / np.abs(ref).max()


def galerkin(ctx, test, mesh, family, ops, k):
    """SLP and DLP through nihu_gb_assemble_galerkin on the device, the unwanted one left alone."""
    L = g.lib()
    trial = g.api.DeviceMesh(ctx, *mesh)
    tm = trial if test is mesh else g.api.DeviceMesh(ctx, *test)
    m, n, ld = tm.n, trial.n, tm.n + 1
    host = [np.full((n, ld), 7 + 3j, np.complex64) for _ in range(2)]
    ptr = [ctypes.c_void_p(), ctypes.c_void_p()]
    try:
        for p, h in zip(ptr, host):
            ctx.check(L.nihu_gb_device_alloc(ctx.handle, h.nbytes, ctypes.byref(p)))
            ctx.check(L.nihu_gb_memcpy(ctx.handle, p, C.DEVICE, h.ctypes.data, C.HOST, h.nbytes))
        ctx.check(L.nihu_gb_assemble_galerkin(ctx.handle, tm.handle, trial.handle, family, ops, k, 1.0, 0.0,
                                              g.REGULAR_FP32, g.C64, ptr[0], ptr[1], ld, 0, g.DEVICE))
        for p, h in zip(ptr, host):
            ctx.check(L.nihu_gb_memcpy(ctx.handle, h.ctypes.data, C.HOST, p, C.DEVICE, h.nbytes))
    finally:
        for p in ptr:
            if p:
                L.nihu_gb_device_free(ctx.handle, p)
    for op, h in zip((g.SLP, g.DLP), host):
        assert (h[:, m if ops & op else 0:] == np.complex64(7 + 3j)).all()
    return [h[:, :m].T for h in host]


def check(ctx, oracle, test, mesh, family, ops, k):
    got = galerkin(ctx, test, mesh, family, ops, k)
    fam = oracle.HELMHOLTZ if family == g.HELMHOLTZ_3D else oracle.LAPLACE
    for bit, op, x in ((g.SLP, oracle.SLP, got[0]), (g.DLP, oracle.DLP, got[1])):
        if ops & bit:
            ref = oracle.assemble_galerkin(test, mesh, fam, op, k, threads=8)
            if np.abs(ref).max() > 1e-12:
                assert rel(x, ref) <= 1e-5
            else:  # the DLP of one flat element: rounding of terms of the size of its SLP, 3e-4
                assert np.abs(x).max() <= 1e-9


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("family,k", [(g.HELMHOLTZ_3D, 3.0), (g.LAPLACE_3D, 0.0)])
@pytest.mark.parametrize("ops", [g.SLP, g.DLP, g.SLP | g.DLP])
def test_one_mesh(gpu_ctx, oracle, n, family, k, ops):
    mesh = part(n)
    check(gpu_ctx, oracle, mesh, mesh, family, ops, k)


@pytest.mark.parametrize("k", [3.0, 40.0])
@pytest.mark.parametrize("rows,cols", [(1, 17), (65, 1), (257, 33)])
def test_two_meshes(gpu_ctx, oracle, rows, cols, k):
    # the rows' mesh moved off the columns': nothing matches
    nodes, el = part(rows)
    check(gpu_ctx, oracle, (nodes * 1.13 + 0.02, el), part(cols), g.HELMHOLTZ_3D, g.SLP | g.DLP, k)


@pytest.mark.parametrize("ops", [g.SLP, g.DLP, g.SLP | g.DLP])
def test_large_wave_number(gpu_ctx, oracle, ops):
    mesh = part(400)
    check(gpu_ctx, oracle, mesh, mesh, g.HELMHOLTZ_3D, ops, 40.0)


@pytest.mark.parametrize("ops", [g.SLP, g.DLP, g.SLP | g.DLP])
@pytest.mark.parametrize("n", [5, 65, 150])
def test_quads(gpu_ctx, oracle, n, ops):
    nodes, el = meshes.cube_sphere(5)
    mesh = nodes, np.ascontiguousarray(el[:n])
    check(gpu_ctx, oracle, mesh, mesh, g.HELMHOLTZ_3D, ops, 3.0)
