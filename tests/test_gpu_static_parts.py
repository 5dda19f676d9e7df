"""The nearly singular static (Laplace) parts of the four operators, float-float
(complex64 results under FP32 regular quadrature) and FP64, against the oracle.

The Laplace family has no dynamic part, so a nearly singular entry is its
static part alone.  Tolerance of the complex64 entries: the store rounds to
2^-24 = 6e-8 relative and the float-float sums hold 1e-11 of the terms, of
which up to three digits cancel between the sides: 2e-7 of the entry plus
1e-8 of the largest.  FP64: 1e-11 of the largest.
"""
import numpy as np
import pytest

import nihu_gb300 as g
from nihu_gb300 import meshes

pytestmark = pytest.mark.gpu


def plate(n):
    """Flat unit square of 4 n^2 triangles (crossed cells): coplanar pairs, centres on other elements' side lines."""
    nodes, faces, at = [], [], {}
    for i in range(n + 1):
        for j in range(n + 1):
            at[i, j] = len(nodes)
            nodes.append((i / n, j / n, 0.0))
    for i in range(n):
        for j in range(n):
            c = len(nodes)
            nodes.append(((i + 0.5) / n, (j + 0.5) / n, 0.0))
            q = [at[i, j], at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]]
            faces += [(q[a], q[(a + 1) % 4], c) for a in range(4)]
    el = np.full((len(faces), 5), -1, np.int32)
    el[:, 0] = g.TRIA_1
    el[:, 1:4] = faces
    return np.array(nodes), el


def fold(angle):
    """Two plates sharing an edge under an angle: planes seen edge-on from the other side."""
    a, ea = plate(3)
    b = np.stack([-np.cos(angle) * a[:, 0], a[:, 1], np.sin(angle) * a[:, 0]], axis=1)
    eb = ea.copy()
    eb[:, 1:4] = ea[:, 1:4] + len(a)
    return np.concatenate([a, b]), np.concatenate([ea, eb])


def sphere(scale, shift):
    nodes, el = meshes.icosphere(2)
    return nodes * scale + shift, el


CASES = {"unit": lambda: sphere(1.0, 0.0), "small": lambda: sphere(1e-4, 0.0), "large": lambda: sphere(1e5, 0.0),
         "shifted": lambda: sphere(1.0, 40.0), "plate": lambda: plate(4), "fold_right": lambda: fold(np.pi / 2),
         "fold_flat": lambda: fold(1e-3)}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("ops", [g.SLP, g.DLP, g.DLPT, g.HSP])
def test_static_parts_of_near_pairs(gpu_ctx, oracle, name, ops):
    mesh = CASES[name]()
    m = g.create_mesh(*mesh)
    col_ptr, rows = g.near_pairs(m, m, ctx=gpu_ctx)
    cols = np.repeat(np.arange(len(mesh[1])), np.diff(col_ptr)).astype(np.int32)
    ref = oracle.assemble_pairs(mesh, mesh, oracle.LAPLACE, ops, 0.0, rows, cols, same_mesh=True, threads=8)
    ok = np.isfinite(ref)  # the reference's formula divides by zero where a centre lies exactly on a side's line
    assert ok.mean() > 0.5
    big = np.abs(ref[ok]).max()
    for dtype, precision, rel, floor in ((g.C64, "fp32", 2e-7, 1e-8), (g.C128, "fp64", 0.0, 1e-11)):
        out = g.assemble_pairs(m, m, rows, cols, ops, family=g.LAPLACE_3D, dtype=dtype, precision=precision, ctx=gpu_ctx)
        got = out[0] if ops in (g.DLP, g.HSP) else out[1]
        assert np.isfinite(got).all()
        err = np.abs(got[ok] - ref[ok])
        # entries of coplanar elements vanish: the floor is then the element's own scale
        scale = max(big, {g.DLP: 1e-1, g.DLPT: 1e-1}.get(ops, 0.0))
        assert (err <= rel * np.abs(ref[ok]) + floor * scale).all(), (precision, err.max() / scale)


@pytest.mark.parametrize("k", [2.0 - 0.4j, 7.0 + 1.0j, 20.0 - 4.0j, 150.0 - 1.0j])
@pytest.mark.parametrize("n", [1, 20, 80, 319, 640, 1280])
def test_near_entries_of_a_complex_wave_number(gpu_ctx, oracle, n, k):
    """The nearly singular and self entries with their dynamic part: float-float
    up to |k| r = 64, FP64 beyond; one, two or four lanes per pair by the number
    of pairs.  Tolerance as above; E - 1 is formed from E, so the floor is
    1e-8 of the largest entry here too."""
    nodes, el = meshes.icosphere(3 if n > 320 else 2)
    mesh = (nodes, np.ascontiguousarray(el[:n]))
    m = g.create_mesh(*mesh)
    sp = g.constant_view(m)
    kind = oracle.classify(mesh, mesh, same_mesh=True)
    rows, cols = (x.astype(np.int32) for x in np.nonzero(kind < 0))
    for op, make in ((oracle.SLP, g.helmholtz_3d_SLP_kernel), (oracle.DLP, g.helmholtz_3d_DLP_kernel)):
        got = np.zeros((n, n), np.complex64, order="F")
        (g.dirac(sp) * g.create_integral_operator(make(k))[sp]).eval_into(got, ctx=gpu_ctx)
        ref = oracle.assemble_pairs(mesh, mesh, oracle.HELMHOLTZ, op, k, rows, cols, same_mesh=True, threads=8)
        err = np.abs(got[rows, cols] - ref)
        assert (err <= 2e-7 * np.abs(ref) + 1e-8 * max(np.abs(ref).max(), 1e-3)).all(), err.max()
