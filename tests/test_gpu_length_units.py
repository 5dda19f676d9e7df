"""The same body in other length units (a power of two of them, so that every
coordinate is exact): SLP entries are in proportion, DLP entries the same.

Tolerance: the FP32 mode's bar, 1e-5 of the largest entry.  Nothing but the
exponents differs, so they agree far better where every step stays in range.
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes
from test_gpu_two_row import on_device, rel

pytestmark = pytest.mark.gpu


def matrices(ctx, mesh, k):
    dm = g.api.DeviceMesh(ctx, *mesh)
    return on_device(ctx, dm.n, dm.n, 0, lambda a, b, ld: g.lib().nihu_gb_assemble_c(
        ctx.handle, dm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, k.real, k.imag, 1.0, 0.0, g.REGULAR_FP32, g.C64, a, b,
        ld, 0, g.DEVICE))


@pytest.mark.parametrize("power", [-45, -20, 20, 45])
@pytest.mark.parametrize("k", [3.0 + 0j, 2.0 - 0.4j])
def test_triangles(gpu_ctx, power, k):
    nodes, el = meshes.icosphere(2)
    unit = 2.0 ** power
    S, D = matrices(gpu_ctx, (nodes, el), k)
    T, E = matrices(gpu_ctx, (nodes * unit, el), k / unit)
    assert rel(T.astype(complex) / unit, S) <= 1e-5
    assert rel(E, D) <= 1e-5


@pytest.mark.parametrize("power", [-20, 20, 40])
@pytest.mark.parametrize("k", [3.0 + 0j, 2.0 - 0.4j])
def test_burton_miller_operators(gpu_ctx, power, k):
    # DLPt entries stay the same, HSP entries go with the inverse length (its rule in
    # the element's plane asks for |z| <= 1e-12, which leaves out the smallest units)
    nodes, el = meshes.icosphere(2)
    unit = 2.0 ** power

    def operators(nodes, k):
        dm = g.api.DeviceMesh(gpu_ctx, nodes, el)
        return on_device(gpu_ctx, dm.n, dm.n, 0, lambda a, b, ld: g.lib().nihu_gb_assemble_bm_c(
            gpu_ctx.handle, dm.handle, dm.handle, g.HELMHOLTZ_3D, g.DLPT | g.HSP, k.real, k.imag, 1.0, 0.0, g.REGULAR_FP32,
            g.C64, a, b, ld, 0, g.DEVICE))

    T, H = operators(nodes, k)
    U, G = operators(nodes * unit, k / unit)
    assert rel(U, T) <= 1e-5
    assert rel(G.astype(complex) * unit, H) <= 1e-5


@pytest.mark.parametrize("power", [-30, 30])
def test_quads(gpu_ctx, power):
    nodes, el = meshes.cube_sphere(4)
    unit = 2.0 ** power
    S, D = matrices(gpu_ctx, (nodes, el), 3.0 + 0j)
    T, E = matrices(gpu_ctx, (nodes * unit, el), (3.0 + 0j) / unit)
    assert rel(T.astype(complex) / unit, S) <= 1e-5
    assert rel(E, D) <= 1e-5
