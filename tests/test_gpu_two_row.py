"""The kernels whose threads own two rows, at the edges of their tiles (64 rows
a warp, 512 rows and up to 32 columns a block, flushes of 8 columns), with
leading dimensions that allow no wide store, against the oracle.

Tolerance: the FP32 mode's bar, 1e-5 of the largest entry per matrix; FP32
rounding of the entries and sums of at most 42 FP32 terms stay below 1e-6.
"""
import ctypes

import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import _capi as C
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 64, 65, 127, 319, 511, 513, 1027]


def part(n):
    """The first n elements of a sphere of 1280 triangles (an open surface)."""
    nodes, el = meshes.icosphere(3)
    return nodes, np.ascontiguousarray(el[:n])


def rel(got, ref):
    return np.abs(got - ref).max() / np.abs(ref).max()


def on_device(ctx, n_rows, n_cols, pad, call):
    """Two complex64 matrices of leading dimension n_rows + pad filled by call(pa, pb, ld); the padding stays untouched."""
    L = g.lib()
    ld = n_rows + pad
    host = [np.full((n_cols, ld), 7 + 3j, np.complex64) for _ in range(2)]
    ptr = [ctypes.c_void_p(), ctypes.c_void_p()]
    try:
        for p, h in zip(ptr, host):
            ctx.check(L.nihu_gb_device_alloc(ctx.handle, h.nbytes, ctypes.byref(p)))
            ctx.check(L.nihu_gb_memcpy(ctx.handle, p, C.DEVICE, h.ctypes.data, C.HOST, h.nbytes))
        ctx.check(call(ptr[0], ptr[1], ld))
        for p, h in zip(ptr, host):
            ctx.check(L.nihu_gb_memcpy(ctx.handle, h.ctypes.data, C.HOST, p, C.DEVICE, h.nbytes))
    finally:
        for p in ptr:
            if p:
                L.nihu_gb_device_free(ctx.handle, p)
    for h in host:
        assert (h[:, n_rows:] == np.complex64(7 + 3j)).all()
    return [h[:, :n_rows].T for h in host]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("family", [g.HELMHOLTZ_3D, g.LAPLACE_3D])
def test_burton_miller_system(gpu_ctx, oracle, n, family):
    mesh = part(n)
    k = 3.0 if family == g.HELMHOLTZ_3D else 0.0
    c = 0.2 - 0.4j
    dm = g.api.DeviceMesh(gpu_ctx, *mesh)
    A, B = on_device(gpu_ctx, n, n, 1, lambda a, b, ld: g.lib().nihu_gb_assemble_burton_miller(
        gpu_ctx.handle, dm.handle, family, k, c.real, c.imag, g.REGULAR_FP32, g.C64, a, b, ld, g.DEVICE))
    fam = oracle.HELMHOLTZ if family == g.HELMHOLTZ_3D else oracle.LAPLACE
    S, D, T, H = (oracle.assemble(mesh, mesh, fam, op, k, threads=8) for op in (oracle.SLP, oracle.DLP, oracle.DLPT, oracle.HSP))
    assert rel(A, D + c * H - 0.5 * np.eye(n)) <= 1e-5
    assert rel(B, S + c * T + c / 2 * np.eye(n)) <= 1e-5


def collocation(ctx, mesh, test, family, ops, k, alpha=1.0, accumulate=0):
    """SLP and DLP matrices through nihu_gb_assemble_c on the device; the outputs start at 7 + 3j."""
    dm = g.api.DeviceMesh(ctx, *mesh)
    tm = dm if test is mesh else g.api.DeviceMesh(ctx, *test)
    return on_device(ctx, len(test[1]), len(mesh[1]), 1, lambda a, b, ld: g.lib().nihu_gb_assemble_c(
        ctx.handle, tm.handle, dm.handle, family, ops, complex(k).real, complex(k).imag, complex(alpha).real,
        complex(alpha).imag, g.REGULAR_FP32, g.C64, a, b, ld, accumulate, g.DEVICE))


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("k", [0.0, 3.0, 2.0 - 0.4j])
@pytest.mark.parametrize("ops", [g.SLP, g.DLP, g.SLP | g.DLP])
def test_collocation(gpu_ctx, oracle, n, k, ops):
    mesh = part(n)
    family, fam = (g.HELMHOLTZ_3D, oracle.HELMHOLTZ) if k else (g.LAPLACE_3D, oracle.LAPLACE)
    got = collocation(gpu_ctx, mesh, mesh, family, ops, k)
    for out, op in zip(got, (oracle.SLP, oracle.DLP)):
        if ops & op:
            ref = oracle.assemble(mesh, mesh, fam, op, k, threads=8)
            assert np.abs(out - ref).max() <= 1e-5 * max(np.abs(ref).max(), 1e-3)  # one element's DLP is zero
        else:
            assert (out == np.complex64(7 + 3j)).all()


@pytest.mark.parametrize("k", [3.0, 2.0 - 0.4j])
def test_collocation_scaled_and_added(gpu_ctx, oracle, k):
    mesh = part(319)
    alpha = 0.5 - 2.0j
    for out, op in zip(collocation(gpu_ctx, mesh, mesh, g.HELMHOLTZ_3D, g.SLP | g.DLP, k, alpha, 1), (oracle.SLP, oracle.DLP)):
        ref = alpha * oracle.assemble(mesh, mesh, oracle.HELMHOLTZ, op, k, threads=8)
        assert np.abs(out - (7 + 3j) - ref).max() <= 1e-5 * np.abs(ref).max() + 1e-6  # 7 + 3j + entry in FP32


@pytest.mark.parametrize("quads", [False, True])
def test_field_points(gpu_ctx, oracle, quads):
    """Rows and columns of other meshes, one of them with both element types."""
    trial = meshes.cube_sphere(5) if quads else part(333)
    nodes, el = meshes.icosphere(2, radius=1.6)
    test = (nodes, el[:75])
    for a, b in ((test, trial), (trial, test)):
        for out, op in zip(collocation(gpu_ctx, b, a, g.HELMHOLTZ_3D, g.SLP | g.DLP, 2.5), (oracle.SLP, oracle.DLP)):
            assert rel(out, oracle.assemble(a, b, oracle.HELMHOLTZ, op, 2.5, same_mesh=False, threads=8)) <= 1e-5
