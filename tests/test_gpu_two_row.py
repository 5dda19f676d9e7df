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
