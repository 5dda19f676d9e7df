"""Plates folded by small angles: DLP and DLPt entries are of the order of the
angle, although they are differences of terms of order one.

Tolerance: the FP32 mode's bar, 1e-5 of the matrix's largest entry, against the
FP64 mode, whose own rounding at the smallest angle is 1e-16 / 3e-10 of it.
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import _capi as C
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu


def folded(angle, n=8):
    y, x = np.divmod(np.arange((n + 1) ** 2), n + 1)
    nodes = np.column_stack([x, y, np.zeros(len(x))]) / n
    over = nodes[:, 0] > 0.5
    nodes[over, 2] = (nodes[over, 0] - 0.5) * np.sin(angle)
    nodes[over, 0] = 0.5 + (nodes[over, 0] - 0.5) * np.cos(angle)
    a = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel()
    faces = np.stack([np.column_stack([a, a + 1, a + n + 2]), np.column_stack([a, a + n + 2, a + n + 1])], 1).reshape(-1, 3)
    return meshes._pack(nodes, faces, meshes.TRIA_1)


def on_host(ctx, n, dtype, call):
    out = [np.zeros((n, n), dtype, order="F") for _ in range(2)]
    ctx.check(call(out[0].ctypes.data, out[1].ctypes.data, n))
    return [x.astype(complex) for x in out]


def modes(ctx, n, call):
    return (on_host(ctx, n, np.complex64, lambda a, b, ld: call(a, b, ld, g.REGULAR_FP32, g.C64)),
            on_host(ctx, n, np.complex128, lambda a, b, ld: call(a, b, ld, g.REGULAR_FP64, g.C128)))


@pytest.mark.parametrize("angle", [1e-3, 1e-5, 1e-7, 1e-8])
@pytest.mark.parametrize("k", [2.0 + 0j, 2.0 - 0.4j])
def test_fold(gpu_ctx, angle, k):
    L = g.lib()
    dm = g.api.DeviceMesh(gpu_ctx, *folded(angle))
    h, args = gpu_ctx.handle, (g.HELMHOLTZ_3D,)
    calls = {
        "DLP": lambda a, b, ld, prec, dt: L.nihu_gb_assemble_c(h, dm.handle, dm.handle, *args, g.DLP, k.real, k.imag, 1.0, 0.0,
                                                               prec, dt, a, b, ld, 0, C.HOST),
        "DLPt": lambda a, b, ld, prec, dt: L.nihu_gb_assemble_bm_c(h, dm.handle, dm.handle, *args, g.DLPT, k.real, k.imag, 1.0,
                                                                   0.0, prec, dt, b, a, ld, 0, C.HOST),
    }
    for name, call in calls.items():
        got, ref = modes(gpu_ctx, dm.n, call)
        scale = np.abs(ref[1]).max()
        assert 0.01 * angle < scale < 10 * angle, name
        assert np.abs(got[1] - ref[1]).max() <= 1e-5 * scale, name


@pytest.mark.parametrize("angle", [1e-5, 1e-7, 1e-8])
def test_pair_list(gpu_ctx, angle):
    nodes, el = folded(angle)
    mesh = g.create_mesh(nodes, el)
    n = len(el)
    r, c = (x.ravel() for x in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    for ops, out in ((g.DLP, 0), (g.DLPT, 1)):
        got = g.assemble_pairs(mesh, mesh, r, c, ops, 2.0, dtype=g.C64, ctx=gpu_ctx)[out].astype(complex)
        ref = g.assemble_pairs(mesh, mesh, r, c, ops, 2.0, dtype=g.C128, precision="fp64", ctx=gpu_ctx)[out]
        assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("ops", [g.SLP, g.DLP, g.DLPT, g.HSP, g.SLP | g.DLP, g.DLPT | g.HSP, g.DLP | g.DLPT, g.SLP | g.HSP])
def test_operators_of_a_sharp_fold(gpu_ctx, ops):
    # collocation points close above the insides of elements, and only some of the
    # operators asked for: the others contribute nothing
    nodes, el = folded(np.deg2rad(175))
    mesh = g.create_mesh(nodes, el)
    n = len(el)
    r, c = (x.ravel() for x in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    got = g.assemble_pairs(mesh, mesh, r, c, ops, 2.0, dtype=g.C64, ctx=gpu_ctx)
    ref = g.assemble_pairs(mesh, mesh, r, c, ops, 2.0, dtype=g.C128, precision="fp64", ctx=gpu_ctx)
    for x, y in zip(got, ref):
        if y is not None:
            assert np.abs(x.astype(complex) - y).max() <= 1e-5 * np.abs(y).max()
