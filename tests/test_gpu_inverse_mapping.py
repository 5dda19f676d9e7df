"""Strongly twisted quads on which Newton's iteration of the inverse mapping wanders
before it finds the foot point: which pairs it gives up on (after 100 steps)
depends on its roundings, so the arithmetic of its steps is part of what a call
accepts.  These meshes are accepted, by the oracle and by the divisions and
square root of the iteration as it is written.
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu


def twisted(seed, n=9):
    rng = np.random.default_rng(seed)
    y, x = np.meshgrid(np.arange(n + 1.0), np.arange(n + 1.0), indexing="ij")
    nodes = np.stack([x, y, np.zeros_like(x)], -1).reshape(-1, 3)
    nodes[:, :2] += (0.05 + 0.12 * rng.random()) * np.random.default_rng(seed).standard_normal((len(nodes), 2))
    nodes /= n
    nodes[:, 2] = 0.2 * rng.random() * np.sin(5 * nodes[:, 0] + rng.random()) * np.cos(4 * nodes[:, 1])
    a = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel()
    return meshes._pack(nodes, np.column_stack([a, a + 1, a + n + 2, a + n + 1]), meshes.QUAD_1)


@pytest.mark.parametrize("seed", [35, 87, 108, 205, 277])
@pytest.mark.parametrize("precision", [g.REGULAR_FP32, g.REGULAR_FP64])
def test_accepted(gpu_ctx, seed, precision):
    dm = g.api.DeviceMesh(gpu_ctx, *twisted(seed))
    S, D = (np.zeros((dm.n, dm.n), complex, order="F") for _ in range(2))
    gpu_ctx.check(g.lib().nihu_gb_assemble(gpu_ctx.handle, dm.handle, dm.handle, g.HELMHOLTZ_3D, g.SLP | g.DLP, 2.0, 1.0, 0.0,
                                           precision, g.C128, S.ctypes.data, D.ctypes.data, dm.n, 0, g.HOST))
    assert np.isfinite(S).all() and np.isfinite(D).all()
