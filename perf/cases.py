"""The calls whose speed counts: what programs do with this library, over the sizes they do it at.

Every case is one pass through a public entry point (the C ABI on device
buffers, as a C or ctypes program holds them, or the Python front end), on a
mesh, wave number and data made from a seed.  ``listed()`` gives the fixed
cases, ``draw()`` more of the same ranges, ``prepare()`` the state a program
keeps between calls (mesh handle, output buffers, plan), ``run()`` one pass,
``work()`` the bytes and operations it cannot do without, and ``exact()`` the
same outputs in 64 bits from a restatement in torch.

Meshes are rotated, slightly deformed spheres of flat triangles (20 f^2 of
them for subdivision frequency f, so an icosphere of s levels is f = 2^s) and
closed cylinders of flat quads; ``drop`` leaves the last elements out (an
opening in the surface), which makes odd and ragged element counts.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import nihu_gb300 as g
from nihu_gb300 import _capi as C

DEV = "cuda"
ALL4 = C.SLP | C.DLP | C.DLPT | C.HSP


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest solve of a sweep or a test: latency and launches count
        {"name": "dense_320", "kind": "dense", "f": 4, "drop": 0, "ops": 3, "fp64": 0, "laplace": 0, "k": 2.0, "k_im": 0.0},
        # the benchmark's workload: both matrices of one large sphere
        {"name": "dense_20480", "kind": "dense", "f": 32, "drop": 0, "ops": 3, "fp64": 0, "laplace": 0, "k": 5.0, "k_im": 0.0},
        # an ordinary mesh of odd element count in a lossy medium
        {"name": "dense_lossy_odd", "kind": "dense", "f": 15, "drop": 7, "ops": 3, "fp64": 0, "laplace": 0, "k": 4.0, "k_im": -0.3},
        # quads: the closed cylinder of the many-plane-wave workload, smaller
        {"name": "dense_quads", "kind": "quads", "n_theta": 96, "n_z": 72, "n_ring": 9, "drop": 0, "ops": 3, "k": 4.0},
        # `result << space * operator[space]` on numpy matrices, the way the reference's programs are written
        {"name": "shift_host_1280", "kind": "host", "f": 8, "drop": 0, "fp64": 0, "k": 1.0},
        # Burton-Miller system matrices of the large sphere
        {"name": "bm_20480", "kind": "bm", "f": 32, "drop": 0, "fp64": 0, "k": 5.0},
        # Galerkin matrices of an ordinary sphere
        {"name": "galerkin_5120", "kind": "galerkin", "f": 16, "drop": 0, "ops": 3, "fp64": 0, "k": 5.0},
        # near field of a fast multipole solver: the Burton-Miller entries of a pair list
        {"name": "pairs_20480", "kind": "pairs", "f": 32, "drop": 0, "fp64": 0, "box": 0.125, "k": 5.0},
        # one whole solve: assembly, right-hand side, GMRES
        {"name": "cbie_5120", "kind": "cbie", "f": 16, "lu": 0, "k": 2.0},
        # one whole double precision solve by LU, the pulsating-sphere program
        {"name": "cbie_lu_1280", "kind": "cbie", "f": 8, "lu": 1, "k": 1.0},
        # many plane waves on one matrix
        {"name": "multi_rhs_64", "kind": "multi", "f": 28, "nrhs": 64, "k": 3.8},
        # a frequency sweep over meshes of uneven size, replayed by a plan
        {"name": "sweep_48", "kind": "sweep", "f0": 4, "f1": 8, "f2": 16, "count": 48, "k": 5.4},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    k = round(rng.uniform(0.3, 5.5), 3)
    kind = rng.choice(["dense", "dense", "dense", "field", "quads", "host", "bm", "bm", "galerkin", "pairs", "cbie",
                       "cbie", "multi", "sweep"])
    if kind == "dense":
        fp64 = int(rng.random() < 0.25)
        lossy = rng.random() < 0.2
        return {"kind": kind, "f": logint(4, 14 if fp64 else 30), "drop": rng.choice([0, 0, rng.randint(1, 40)]),
                "ops": rng.choice([1, 2, 3, 3, 3]), "fp64": fp64, "laplace": int(not lossy and rng.random() < 0.2),
                "k": k, "k_im": round(rng.uniform(-0.5, -0.05), 3) if lossy else 0.0}
    if kind == "field":
        return {"kind": kind, "f": logint(6, 26), "ft": logint(2, 20), "drop": rng.randint(0, 19), "ops": rng.choice([1, 3, 3]),
                "fp64": 0, "laplace": int(rng.random() < 0.2), "k": k}
    if kind == "quads":
        t = 4 * logint(4, 20)
        return {"kind": kind, "n_theta": t, "n_z": logint(12, 64), "n_ring": rng.randint(2, 8), "drop": rng.randint(0, 5),
                "ops": rng.choice([1, 2, 3, 3]), "k": k}
    if kind == "host":
        return {"kind": kind, "f": logint(4, 10), "drop": rng.choice([0, rng.randint(1, 15)]), "fp64": int(rng.random() < 0.3), "k": k}
    if kind in ("bm", "galerkin"):
        c = {"kind": kind, "f": logint(4, 24 if kind == "bm" else 15), "drop": rng.choice([0, 0, rng.randint(1, 40)]), "fp64": 0, "k": k}
        if kind == "galerkin":
            c["ops"] = rng.choice([1, 2, 3, 3])
        return c
    if kind == "pairs":
        f = logint(8, 30)
        return {"kind": kind, "f": f, "drop": rng.randint(0, 9), "fp64": 0, "box": round(4.0 / f, 4), "k": k}
    if kind == "cbie":
        lu = int(rng.random() < 0.3)
        return {"kind": kind, "f": logint(4, 8) if lu else logint(4, 24), "lu": lu, "k": k}
    if kind == "multi":
        return {"kind": kind, "f": logint(12, 27), "nrhs": rng.choice([7, 16, 33, 48, 64]), "k": k}
    return {"kind": kind, "f0": logint(3, 5), "f1": logint(6, 10), "f2": logint(11, 15), "count": logint(12, 44), "k": k}


# ------------------------------------------------------------------ meshes and data

@functools.lru_cache(maxsize=None)
def _sphere(f):
    """Icosahedron faces split into f^2 triangles, nodes on the unit sphere, shared nodes merged."""
    t = (1 + 5 ** 0.5) / 2
    v = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                  (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)]) / math.sqrt(1 + t * t)
    # each face's closing edge (last corner to first) closes no other face
    faces = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (5, 9, 1), (11, 4, 5), (10, 2, 11), (7, 6, 10),
             (1, 8, 7), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10),
             (8, 6, 7), (9, 8, 1)]
    at = {}
    tri = []
    for i in range(f + 1):
        for j in range(f + 1 - i):
            at[i, j] = len(at)
    ij = np.array(list(at))
    for i in range(f):
        for j in range(f - i):
            tri.append((at[i, j], at[i + 1, j], at[i, j + 1]))
            if i + j < f - 1:
                tri.append((at[i + 1, j], at[i + 1, j + 1], at[i, j + 1]))
    tri = np.array(tri)
    pts, els = [], []
    for n, (a, b, c) in enumerate(faces):
        p = v[a] + np.outer(ij[:, 0] / f, v[b] - v[a]) + np.outer(ij[:, 1] / f, v[c] - v[a])
        pts.append(p / np.linalg.norm(p, axis=1, keepdims=True))
        els.append(tri + n * len(ij))
    pts, els = np.concatenate(pts), np.concatenate(els)
    _, first, inverse = np.unique(np.round(pts, 9), axis=0, return_index=True, return_inverse=True)
    els = inverse.reshape(-1)[els]
    out = np.full((len(els), 5), -1, np.int32)
    out[:, 0] = g.TRIA_1
    out[:, 1:4] = els
    return pts[first], out


@functools.lru_cache(maxsize=None)
def _cylinder(n_theta, n_z, n_ring):
    return g.meshes.cylinder(n_theta, n_z, n_ring)


def _rotation(rng):
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    q = q * np.sign(np.diag(r))
    return q * np.linalg.det(q)


def _deformed(f, drop, seed, radius=1.0):
    """A rotated sphere with a smooth 2 % bump field, without its last `drop` elements."""
    rng = np.random.default_rng([seed, f])
    nodes, elems = _sphere(f)
    d, ph = rng.standard_normal((4, 3)), rng.uniform(0, 2 * np.pi, 4)
    bump = 0.005 * np.cos(2 * nodes @ d.T + ph).sum(axis=1)
    nodes = radius * (nodes * (1 + bump)[:, None]) @ _rotation(rng).T
    return np.ascontiguousarray(nodes), np.ascontiguousarray(elems[: len(elems) - drop])


def _wave(case, seed):
    """The case's wave number within 2 % of it."""
    return float(case["k"] * (1 + 0.02 * np.random.default_rng([seed, 77]).uniform(-1, 1)))


# interior resonances of the sphere, where the plain integral equation is singular and no program solves it
RESONANCES = (math.pi, 4.4934, 5.7635, 2 * math.pi)


def _solvable(k):
    for r in RESONANCES:
        if abs(k - r) < 0.3:
            return r - 0.32
    return k


def _neumann(nodes, elems, k, rng):
    """Neumann data of a rigid body in a plane wave."""
    cen, nrm = g.meshes.centroids_and_normals(nodes, elems)
    d = rng.standard_normal(3)
    d /= np.linalg.norm(d)
    return 1j * k * (nrm @ d) * np.exp(-1j * k * (cen @ d))


def _f64(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=DEV)


class Tri:
    """Corners, centres, sizes, normals and Jacobians of flat triangles on the device."""

    def __init__(self, nodes, elems):
        self.el = torch.as_tensor(elems[:, 1:4].astype(np.int64), device=DEV)
        c = _f64(nodes)[self.el]
        self.c, self.n = c, len(elems)
        self.cen = c.mean(1)
        self.size = sum((c[:, (a + 1) % 3] - c[:, a]).norm(dim=1) for a in range(3)) / 3
        self.e1, self.e2 = c[:, 1] - c[:, 0], c[:, 2] - c[:, 0]
        nrm = torch.linalg.cross(self.e1, self.e2)
        self.J = nrm.norm(dim=1)
        self.nrm = nrm / self.J[:, None]


def _nystrom(nodes, elems, k, dtype):
    """DLP - I/2 by the one-point rule, column-major: a dense second-kind matrix as a solver meets it."""
    t = Tri(nodes, elems)
    out = torch.empty((t.n, t.n), dtype=dtype, device=DEV)
    for j0 in range(0, t.n, 1024):
        r = t.cen[None, :, :] - t.cen[j0:j0 + 1024, None, :]
        d = r.norm(dim=2)
        d[torch.arange(d.shape[0], device=DEV), torch.arange(j0, j0 + d.shape[0], device=DEV)] = 1.0
        # r points from trial to test: -(r . n_y) is (y - x) . n_y
        v = (1 + 1j * k * d) * torch.exp(-1j * k * d) / d ** 3 / (4 * math.pi) * ((r * t.nrm[j0:j0 + 1024, None, :]).sum(2)
                                                                              * (t.J / 2)[j0:j0 + 1024, None])
        v[torch.arange(d.shape[0], device=DEV), torch.arange(j0, j0 + d.shape[0], device=DEV)] = -0.5
        out[j0:j0 + 1024] = v.to(dtype)
    return out


def _near_field(cen, box, count):
    """The pairs of elements in the same or a neighbouring leaf box, elements in box order: `count` of them."""
    key = torch.floor((cen + 1.2) / box).to(torch.int64)
    order = torch.argsort((key[:, 0] * 4096 + key[:, 1]) * 4096 + key[:, 2], stable=True)
    key = key[order]
    rows, cols = [], []
    for i0 in range(0, len(key), 1024):
        hit = ((key[i0:i0 + 1024, None, :] - key[None, :, :]).abs() <= 1).all(2).nonzero()
        rows.append(order[hit[:, 0] + i0])
        cols.append(order[hit[:, 1]])
    rows, cols = torch.cat(rows).to(torch.int32), torch.cat(cols).to(torch.int32)
    at = torch.arange(count, device=DEV) % len(rows)
    return rows[at], cols[at]


def _pair_count(case):
    """What boxes of 4/f hold on a sphere of 20 f^2 triangles, less the few per cent by which that turns with it."""
    return 250 * _count(case)


# ------------------------------------------------------------------ state and one pass

def _out(cols, rows, fp64):
    return torch.empty((cols, rows), dtype=torch.complex128 if fp64 else torch.complex64, device=DEV)


def _sweep_parts(case, seed):
    rng = np.random.default_rng([seed, 5])
    meshes = [_deformed(case[m], 0, seed) for m in ("f0", "f1", "f2")]
    mesh_of = np.arange(case["count"]) % 3
    ks = np.array([_solvable(x) for x in rng.uniform(0.1, case["k"], case["count"])])
    qs = [_neumann(*meshes[m], k, rng) for m, k in zip(mesh_of, ks)]
    return meshes, mesh_of, ks, qs


def prepare(case, seed):
    ctx = g.default_context()
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx, "case": case}
    if kind == "sweep":
        meshes, mesh_of, s["ks"], s["q"] = _sweep_parts(case, seed)
        s["plan"] = g.SweepPlan([g.create_mesh(*m) for m in meshes], mesh_of, k_max=6.0, ctx=ctx)
        return s
    k = s["k"] = _wave(case, seed)
    fp64 = s["fp64"] = bool(case.get("fp64", 0))
    if kind == "quads":
        nodes, elems = _cylinder(case["n_theta"], case["n_z"], case["n_ring"])
        nodes, elems = nodes @ _rotation(np.random.default_rng([seed, 9])).T, elems[: len(elems) - case["drop"]]
    else:
        nodes, elems = _deformed(case["f"], case.get("drop", 0), seed)
    n = len(elems)
    if kind == "host":
        s["mesh"] = g.create_mesh(nodes, elems)
        s["mesh"].device(ctx)
        return s
    if kind == "cbie":
        s["k"] = _solvable(k)
        s["mesh"] = g.create_mesh(nodes, elems)
        s["mesh"].device(ctx)
        s["q"] = _neumann(nodes, elems, s["k"], np.random.default_rng([seed, 3]))
        return s
    if kind == "multi":
        s["k"] = _solvable(k)
        s["A"] = _nystrom(nodes, elems, s["k"], torch.complex64)
        rng = np.random.default_rng([seed, 4])
        s["B"] = torch.as_tensor(np.stack([_neumann(nodes, elems, s["k"], rng) for _ in range(case["nrhs"])]), device=DEV)
        s["X"] = torch.empty_like(s["B"])
        s["n"] = n
        return s
    trial = s["trial"] = g.api.DeviceMesh(ctx, nodes, elems)
    s["n"] = s["m"] = n
    s["test"] = trial
    if kind == "field":
        fn, fe = _deformed(case["ft"], case["drop"], seed + 1, radius=1.5)
        s["test"] = g.api.DeviceMesh(ctx, fn, fe)
        s["m"] = len(fe)
    if kind == "pairs":
        s["rows"], s["cols"] = _near_field(Tri(nodes, elems).cen, case["box"], _pair_count(case))
        s["coef"] = np.array([1, 0, 1, 0, 0, -1 / k, 0, -1 / k], np.float64)
        s["ident"] = np.array([-0.5, 0, 0, -0.5 / k], np.float64)
        s["out"] = [torch.empty(len(s["rows"]), dtype=torch.complex64, device=DEV) for _ in range(2)]
    else:
        s["out"] = [_out(s["n"], s["m"], fp64) for _ in range(2)]
    torch.cuda.synchronize()
    return s


def run(s):
    kind, case, ctx = s["kind"], s["case"], s["ctx"]
    L = g.lib()
    if kind == "sweep":
        p = s["plan"].run(s["ks"], s["q"])[0]
        # pressures in the precision of the assembled matrices
        return np.concatenate(p).astype(np.complex64)
    if kind == "host":
        n = s["mesh"].num_elements
        sp = g.constant_view(s["mesh"])
        prec = "fp64" if s["fp64"] else "fp32"
        dt = np.complex128 if s["fp64"] else np.complex64
        Ls, Ms = np.zeros((n, n), dt, order="F"), np.zeros((n, n), dt, order="F")
        (g.dirac(sp) * g.create_integral_operator(g.helmholtz_3d_SLP_kernel(s["k"]))[sp]).eval_into(Ls, precision=prec)
        (g.dirac(sp) * g.create_integral_operator(g.helmholtz_3d_DLP_kernel(s["k"]))[sp]).eval_into(Ms, precision=prec)
        Ms << g.dirac(sp) * (-0.5 * g.identity_integral_operator())[sp]
        return Ls.T, Ms.T
    if kind == "cbie":
        if case["lu"]:
            return g.solve_cbie(s["mesh"], s["k"], s["q"], dtype=g.C128, solver="lu", precision="fp64", ctx=ctx)[0]
        return g.solve_cbie(s["mesh"], s["k"], s["q"], ctx=ctx)[0].astype(np.complex64)
    if kind == "multi":
        n, nrhs = s["n"], case["nrhs"]
        ctx.check(L.nihu_gb_solve_multi(ctx.handle, s["A"].data_ptr(), n, n, s["B"].data_ptr(), s["X"].data_ptr(), nrhs,
                                        C.GEMM_BF16X3, C.GEMM_BF16X6, 30, 20, 1e-6, 1e-3, None, None, None, C.DEVICE))
        return s["X"].to(torch.complex64)
    prec, dtype = (C.REGULAR_FP64, C.C128) if s["fp64"] else (C.REGULAR_FP32, C.C64)
    a, b = (o.data_ptr() for o in s["out"])
    t, r, k = s["test"].handle, s["trial"].handle, s["k"]
    if kind == "bm":
        ctx.check(L.nihu_gb_assemble_burton_miller(ctx.handle, r, C.HELMHOLTZ_3D, k, 0.0, -1 / k, prec, dtype, a, b, s["m"], C.DEVICE))
        return tuple(s["out"])
    if kind == "pairs":
        ctx.check(L.nihu_gb_assemble_pairs(ctx.handle, t, r, C.HELMHOLTZ_3D, ALL4, k, s["coef"].ctypes.data, s["ident"].ctypes.data,
                                           prec, dtype, len(s["rows"]), s["rows"].data_ptr(), s["cols"].data_ptr(), a, b, C.DEVICE))
        return tuple(s["out"])
    family = C.LAPLACE_3D if case.get("laplace") else C.HELMHOLTZ_3D
    ops = case["ops"]
    if kind == "galerkin":
        ctx.check(L.nihu_gb_assemble_galerkin(ctx.handle, t, r, family, ops, k, 1.0, 0.0, prec, dtype, a, b, s["m"], 0, C.DEVICE))
    else:
        ctx.check(L.nihu_gb_assemble_c(ctx.handle, t, r, family, ops, k, case.get("k_im", 0.0), 1.0, 0.0, prec, dtype, a, b, s["m"],
                                       0, C.DEVICE))
    return tuple(o for i, o in enumerate(s["out"]) if ops >> i & 1)


# ------------------------------------------------------------------ work

def _count(case):
    if case["kind"] == "quads":
        m = case["n_theta"] // 4
        return case["n_theta"] * case["n_z"] + 2 * (m * m + case["n_theta"] * case["n_ring"]) - case["drop"]
    return 20 * case["f"] ** 2 - case.get("drop", 0)


def work(case):
    """Bytes: geometry and data read once, results written once; matrices that a solve keeps to itself count once
    written and once per product read.  Flops: one kernel point per pair (about 40 for SLP and DLP together, 80 for
    the four operators) and the products of a solve."""
    kind = case["kind"]
    if kind == "sweep":
        n2 = sum(20 * case[m] ** 2 * 20 * case[m] ** 2 for m in ("f0", "f1", "f2")) * case["count"] / 3
        return {"bytes": n2 * 8 * 9, "flops": n2 * (40 + 8 * 9)}
    n = _count(case)
    es = 16 if case.get("fp64") or case.get("lu") else 8
    if kind == "cbie":
        if case["lu"]:
            return {"bytes": 3.0 * es * n * n, "flops": 40.0 * n * n + 8 / 3 * n ** 3}
        return {"bytes": 8.0 * n * n * 10, "flops": n * n * (40.0 + 8 * 8)}
    if kind == "multi":
        return {"bytes": 20 * 8.0 * n * n + 2 * 16.0 * n * case["nrhs"], "flops": 20 * 8.0 * n * n * case["nrhs"]}
    if kind == "pairs":
        pairs = float(_pair_count(case))
        return {"bytes": pairs * 24, "flops": pairs * 80 * 4}
    m = 20 * case["ft"] ** 2 - case["drop"] if kind == "field" else n
    ops = 3 if kind in ("bm", "host") else case["ops"]
    return {"bytes": float(m) * n * es * bin(ops).count("1") + 200.0 * (m + n), "flops": float(m) * n * (80 if kind == "bm" else 40)}


# ------------------------------------------------------------------ the same in 64 bits

# symmetric triangle rules (Dunavant 1985): orbits (a, w) of 3 and (a, b, w) of 6 points, (w,) the centroid;
# the digits seed a Newton iteration on the moment equations
ORBITS = {
    0: [(1.0,)],
    2: [(1 / 6, 1 / 3)],
    4: [(0.445948, 0.223382), (0.091576, 0.109952)],
    6: [(0.249287, 0.116786), (0.063089, 0.050845), (0.053145, 0.310352, 0.082851)],
    7: [(-0.149570,), (0.260346, 0.175615), (0.065130, 0.053347), (0.048690, 0.312865, 0.077114)],
    8: [(0.144316,), (0.459293, 0.0950916), (0.170569, 0.103217), (0.0505472, 0.0324585), (0.00839478, 0.263113, 0.0272303)],
    14: [(0.488964, 0.0218836), (0.417645, 0.0327884), (0.273478, 0.0517741), (0.177206, 0.0421626), (0.0617999, 0.0144337),
         (0.0193910, 0.00492340), (0.0571248, 0.172267, 0.0246658), (0.0929162, 0.336861, 0.0385715),
         (0.0146470, 0.298373, 0.0144363), (0.00126833, 0.118974, 0.00501023)],
}


@functools.lru_cache(maxsize=None)
def _rule(degree):
    """(xi, eta, w) of the rule on the triangle (0,0), (1,0), (0,1), weights adding up to 1/2."""
    shapes = [len(o) for o in ORBITS[degree]]
    x = np.array([v for o in ORBITS[degree] for v in o])

    def points(x):
        out, k = [], 0
        for s in shapes:
            if s == 1:
                out.append((1 / 3, 1 / 3, x[k]))
            elif s == 2:
                a, w = x[k:k + 2]
                out += [(p, q, w / 3) for p, q in ((a, 1 - 2 * a), (1 - 2 * a, a), (a, a))]
            else:
                a, b, w = x[k:k + 3]
                c = 1 - a - b
                out += [(p, q, w / 6) for p, q in ((a, b), (b, a), (a, c), (c, a), (b, c), (c, b))]
            k += s
        return out

    def residual(x):
        pts = points(x)
        return np.array([sum(w * p ** a * q ** (t - a) for p, q, w in pts)
                         - 2 * math.factorial(a) * math.factorial(t - a) / math.factorial(t + 2)
                         for t in range(degree + 1) for a in range(t + 1)])

    for _ in range(12):
        jac = np.stack([residual(x + 1e-30j * np.eye(len(x))[i]).imag / 1e-30 for i in range(len(x))], axis=1)
        x = x - np.linalg.lstsq(jac, residual(x), rcond=None)[0]
    return np.array([(p, q, w / 2) for p, q, w in points(x)])


def _points(t, j, degree):
    """Points (len(j), q, 3) and weights times Jacobian (len(j), q) of a rule on triangles j."""
    r = _f64(_rule(degree))
    y = t.c[j, 0][:, None] + r[:, 0][None, :, None] * t.e1[j][:, None] + r[:, 1][None, :, None] * t.e2[j][:, None]
    return y, r[:, 2][None] * t.J[j][:, None]


def _kernels(r, nx, ny, k, ops, static):
    """{op: K_k (or K_k - K_0 with static)} at r = y - x; k complex or None for Laplace."""
    d = (r * r).sum(-1).sqrt()
    g0 = 1 / (4 * math.pi * d)
    z = 1j * (k if k is not None else 0.0) * d
    e = torch.exp(-z)
    s = 1.0 if static else 0.0
    out = {}
    rny = (r * ny).sum(-1) / d
    if ops & (C.DLPT | C.HSP):
        rnx = -(r * nx).sum(-1) / d
    p = (1 + z) * e - s
    if ops & C.SLP:
        out[C.SLP] = g0 * (e - s)
    if ops & C.DLP:
        out[C.DLP] = -g0 / d * rny * p
    if ops & C.DLPT:
        out[C.DLPT] = -g0 / d * rnx * p
    if ops & C.HSP:
        a, b = rnx * rny, (nx * ny).sum(-1)
        m = 3 * a + b
        out[C.HSP] = g0 / d ** 2 * ((m * (1 + z) + a * z * z) * e - s * m)
    return out


# the degree of each operator's rule by d/D: below the first limit the first degree, ..., else 0
DEGREES = {C.SLP: ((1.8, 4), (9.1, 2)), C.DLP: ((2.8, 4), (15.8, 2)), C.DLPT: ((2.8, 4), (15.8, 2)),
           C.HSP: ((1.9, 6), (3.6, 4), (22.3, 2))}


def _degree(ratio, op):
    deg = torch.zeros(ratio.shape, dtype=torch.int64, device=DEV)
    for lim, d in reversed(DEGREES[op]):
        deg[ratio < lim] = d
    return deg


def _near(x, nx, t, j, k, ops):
    """Nearly singular pairs: points x (normals nx) against triangles j."""
    out = {}
    if k is not None:
        y, w = _points(t, j, 14)
        v = _kernels(y - x[:, None], nx[:, None], t.nrm[j][:, None], k, ops, True)
        out = {op: (q * w).sum(1) for op, q in v.items()}
    t0 = t.e1[j] / t.e1[j].norm(dim=1, keepdim=True)
    t2 = t.nrm[j]
    t1 = torch.linalg.cross(t2, t0)
    loc = torch.stack([((t.c[j] - x[:, None]) * a[:, None]).sum(2) for a in (t0, t1)], 2)
    z = ((x - t.c[j, 0]) * t2).sum(1)
    n0, n1, n2 = ((a * nx).sum(1) for a in (t0, t1, t2))
    st = {op: torch.zeros(len(j), dtype=torch.float64, device=DEV) for op in (C.SLP, C.DLP, C.DLPT, C.HSP) if ops & op}
    sg, az = torch.sign(z), z.abs()
    for s in range(3):
        c1, c2 = loc[:, s], loc[:, (s + 1) % 3]
        u = (c2 - c1) / (c2 - c1).norm(dim=1, keepdim=True)
        f = c1 - u * (c1 * u).sum(1, keepdim=True)
        dref = f.norm(dim=1)
        th0 = torch.atan2(f[:, 1], f[:, 0])
        a1, a2 = torch.atan2(c1[:, 1], c1[:, 0]), torch.atan2(c2[:, 1], c2[:, 0])
        wrap = (a2 - a1).abs() > math.pi
        a1, a2 = torch.where(wrap & (a2 > a1), a1 + 2 * math.pi, a1), torch.where(wrap & (a2 <= a1), a2 + 2 * math.pi, a2)
        for ng, part in ((6, ops & (C.SLP | C.DLP | C.DLPT)), (21, ops & C.HSP)):
            if not part:
                continue
            xg, wg = (_f64(v) for v in np.polynomial.legendre.leggauss(ng))
            th = (a1[:, None] * (1 - xg) + a2[:, None] * (1 + xg)) / 2
            w = (a2 - a1)[:, None] / 2 * wg
            R = dref[:, None] / torch.cos(th - th0[:, None])
            zz = z[:, None]
            r = (R * R + zz * zz).sqrt()
            ca, sa = torch.cos(th), torch.sin(th)
            rnx = R * (n0[:, None] * ca + n1[:, None] * sa) - n2[:, None] * zz
            if part & C.SLP:
                st[C.SLP] += ((r - az[:, None]) * w).sum(1)
            if part & C.DLP:
                st[C.DLP] += sg * ((1 - az[:, None] / r) * w).sum(1)
            if part & C.DLPT:
                st[C.DLPT] += ((-rnx / r + (n0[:, None] * ca + n1[:, None] * sa) * torch.log(R + r) - (n2 * sg)[:, None]) * w).sum(1)
            if part & C.HSP:
                flat = az[:, None] <= 1e-12
                v = torch.where(flat, -n2[:, None] / R, R * R / (r ** 3 * torch.where(flat, 1.0, zz)) * rnx)
                st[C.HSP] += (v * w).sum(1)
    return {op: out.get(op, 0) + v / (4 * math.pi) for op, v in st.items()}


def _self(t, j, k, ops):
    """A triangle seen from its own centre: DLP and DLPt are zero."""
    R = t.c[j] - t.cen[j][:, None]
    r = R.norm(dim=2)
    u = R / r[:, :, None]
    i0 = torch.zeros(len(j), dtype=torch.float64, device=DEV)
    i2 = i0.clone()
    for a in range(3):
        b = (a + 1) % 3
        c = t.c[j, a] - t.c[j, b]
        c = c / c.norm(dim=1, keepdim=True)
        th, al = torch.acos((u[:, a] * u[:, b]).sum(1)), torch.acos((u[:, a] * c).sum(1))
        i0 += r[:, a] * torch.sin(al) * torch.log(torch.tan((al + th) / 2) / torch.tan(al / 2))
        i2 += (torch.cos(al + th) - torch.cos(al)) / (r[:, a] * torch.sin(al))
    zero = torch.zeros(len(j), dtype=torch.complex128, device=DEV)
    s, h = i0 + zero, i2 + zero
    if k is not None:
        y, w = _points(t, j, 7)
        d = (y - t.cen[j][:, None]).norm(dim=2)
        z = 1j * k * d
        # (e^-z - 1)/d and ((1 + z) e^-z - 1 + z^2/2)/d^3 by their series: z stays below 1 on these elements
        ps, ph, f = torch.zeros_like(z), torch.zeros_like(z), 1.0
        for n in range(1, 30):
            f *= n
            ps = ps + (-1j * k) ** n * d ** (n - 1) / f
            if n >= 3:
                ph = ph + (1 - n) * (-1j * k) ** n * d ** (n - 3) / f
        s = s + (ps * w).sum(1)
        h = h + k * k / 2 * i0 + (ph * w).sum(1)
    out = {C.SLP: s / (4 * math.pi), C.DLP: zero, C.DLPT: zero, C.HSP: h / (4 * math.pi)}
    return {op: v for op, v in out.items() if ops & op}


def _entries(x, nx, t, i, j, k, ops, same):
    """{op: entries} of collocation pairs (test point i of x, triangle j)."""
    out = {op: torch.zeros(len(i), dtype=torch.complex128, device=DEV) for op in (C.SLP, C.DLP, C.DLPT, C.HSP) if ops & op}
    ratio = (t.cen[j] - x[i]).norm(dim=1) / t.size[j]
    self_ = (i == j) if same else torch.zeros_like(i, dtype=torch.bool)
    near = (ratio < 1.5) & ~self_
    for op in out:
        deg = torch.where(near | self_, -1, _degree(ratio, op))
        for d in (0, 2, 4, 6):
            at = (deg == d).nonzero()[:, 0]
            for a in at.split(1 << 21):
                y, w = _points(t, j[a], d)
                ny = t.nrm[j[a]][:, None]
                out[op][a] = (_kernels(y - x[i[a]][:, None], nx[i[a]][:, None], ny, k, op, False)[op] * w).sum(1)
    for a in near.nonzero()[:, 0].split(1 << 17):
        for op, v in _near(x[i[a]], nx[i[a]], t, j[a], k, ops).items():
            out[op][a] = v.to(torch.complex128)
    a = self_.nonzero()[:, 0]
    if len(a):
        for op, v in _self(t, j[a], k, ops).items():
            out[op][a] = v
    return out


def _matrices(test, t, k, ops, same, fill):
    """Calls fill(j0, {op: (columns, rows) block}) over column blocks."""
    step = max(1, (8 << 20) // test.n)
    rows = torch.arange(test.n, device=DEV)
    for j0 in range(0, t.n, step):
        cols = torch.arange(j0, min(t.n, j0 + step), device=DEV)
        v = _entries(test.cen, test.nrm, t, rows.repeat(len(cols)), cols.repeat_interleave(test.n), k, ops, same)
        fill(j0, {op: q.view(len(cols), test.n) for op, q in v.items()})


def _dense(test, t, k, ops, same):
    out = {op: torch.empty((t.n, test.n), dtype=torch.complex128, device=DEV) for op in (C.SLP, C.DLP) if ops & op}

    def fill(j0, v):
        for op, q in v.items():
            out[op][j0:j0 + len(q)] = q

    _matrices(test, t, k, ops, same, fill)
    return tuple(out.values())


def _gmres(apply, B, tol=1e-13, steps=160):
    """X with A X = B (rows are right-hand sides), one Krylov space for each."""
    beta = B.norm(dim=1)
    V = [B / beta[:, None]]
    H = torch.zeros((len(B), steps + 1, steps), dtype=torch.complex128, device=DEV)
    e1 = torch.zeros((len(B), steps + 1, 1), dtype=torch.complex128, device=DEV)
    e1[:, 0, 0] = beta
    for m in range(steps):
        w = apply(V[m])
        for _ in range(2):
            for q, v in enumerate(V):
                h = (v.conj() * w).sum(1)
                H[:, q, m] += h
                w = w - h[:, None] * v
        nw = w.norm(dim=1)
        H[:, m + 1, m] = nw
        V.append(w / nw[:, None])
        if m % 4 == 3 or m == steps - 1:
            y = torch.linalg.lstsq(H[:, :m + 2, :m + 1], e1[:, :m + 2]).solution
            res = (H[:, :m + 2, :m + 1] @ y - e1[:, :m + 2]).norm(dim=1)[:, 0] / beta
            if float(res.max()) < tol:
                break
    return sum(y[:, q] * V[q] for q in range(m + 1))


def _solve_cbie(nodes, elems, k, q):
    t = Tri(nodes, elems)
    S, D = _dense(t, t, complex(k), 3, True)
    D.diagonal().sub_(0.5)
    b = (torch.as_tensor(q, device=DEV)[None] @ S)
    return _gmres(lambda v: v @ D, b)[0]


def _galerkin_matched(match):
    """(xi, eta of the first, of the second element, w) of the singular rules in coordinate differences: corner (0),
    edge (1), face (2); Sauter and Schwab, Boundary Element Methods, 5.2."""
    x, w = np.polynomial.legendre.leggauss(4)
    x, w = (x + 1) / 2, w / 2
    u = np.stack(np.meshgrid(x, x, x, x, indexing="ij"), -1).reshape(-1, 4).T
    wt = np.prod(np.stack(np.meshgrid(w, w, w, w, indexing="ij"), -1).reshape(-1, 4), axis=1)
    p, q, r, s = u
    subs = []
    if match == 2:
        b1, b2 = p, p * q
        a1 = (1 - b1) * r
        subs.append((a1, a1 * s, b1, b2, p * (1 - b1) * a1))
        b1, b2 = p * q, p * (q - 1)
        a1 = (1 - b1 + b2) * r - b2
        subs.append((a1, (a1 + b2) * s - b2, b1, b2, p * (1 - b1 + b2) * (a1 + b2)))
        b1, b2 = p * q, p
        a1 = (1 - b2) * r + b2 - b1
        subs.append((a1, (a1 - b2 + b1) * s, b1, b2, p * (1 - b2) * (a1 - b2 + b1)))
    elif match == 1:
        jac = q * p * p * (1 - p)
        for b1, b2, a1, a2 in ((-p * q, -p * q * r, (1 - p) * s + p, p * (1 - q + q * r)),
                               (p * q, p * q * r, (1 - p) * s + p * (1 - q), p * (1 - q)),
                               (-p * q * r, p * q * (1 - r), (1 - p) * s + p, p * (1 - q)),
                               (p * q * r, p * q * (r - 1), (1 - p) * s + p * (1 - q * r), p * (1 - q * r)),
                               (-p * q * r, -p * q, (1 - p) * s + p, p),
                               (p * q * r, p * q, (1 - p) * s + p * (1 - q * r), p * (1 - q))):
            subs.append((a1, a2, b1, b2, jac))
    else:
        subs.append((p, p * q, p * r - p, p * r * s - p * q, r * p ** 3))
    out = []
    for a1, a2, b1, b2, jac in subs:
        one = np.stack([a1 - a2, a2, (a1 + b1) - (a2 + b2), a2 + b2, wt * jac], 1)
        out.append(one)
        if match != 1:
            out.append(one[:, [2, 3, 0, 1, 4]])
    return np.concatenate(out)


def _galerkin(t, k, ops):
    """Galerkin SLP and DLP of triangles on one mesh."""
    out = {op: torch.zeros((t.n, t.n), dtype=torch.complex128, device=DEV) for op in (C.SLP, C.DLP) if ops & op}
    eq = t.el
    step = max(1, (4 << 20) // t.n)
    rows = torch.arange(t.n, device=DEV)
    for j0 in range(0, t.n, step):
        cols = torch.arange(j0, min(t.n, j0 + step), device=DEV)
        i, j = rows.repeat(len(cols)), cols.repeat_interleave(t.n)
        ratio = (t.cen[j] - t.cen[i]).norm(dim=1) / t.size[j]
        shared = torch.zeros(len(i), dtype=torch.int64, device=DEV)
        close = (ratio < 8).nonzero()[:, 0]
        same = eq[i[close]][:, :, None] == eq[j[close]][:, None, :]
        shared[close] = same.sum((1, 2))
        val = {op: torch.zeros(len(i), dtype=torch.complex128, device=DEV) for op in out}
        for op in out:
            deg = _degree(ratio, op)
            deg[ratio < 1.5] = 4 if op == C.SLP else 6
            deg[ratio < 1.1] = 6 if op == C.SLP else 8
            deg[shared > 0] = -1
            for d in (0, 2, 4, 6, 8):
                for a in (deg == d).nonzero()[:, 0].split((1 << 23) // len(_rule(d)) ** 2):
                    if not len(a):
                        continue
                    y, w = _points(t, j[a], d)
                    xs, wx = _points(t, i[a], d)
                    v = _kernels(y[:, None] - xs[:, :, None], None, t.nrm[j[a]][:, None, None], k, op, False)[op]
                    val[op][a] = (v * w[:, None] * wx[:, :, None]).sum((1, 2))
        for match, count in ((0, 1), (1, 2), (2, 3)):
            rule = _f64(_galerkin_matched(match))
            for a in (shared == count).nonzero()[:, 0].split((1 << 22) // len(rule)):
                if not len(a):
                    continue
                same = eq[i[a]][:, :, None] == eq[j[a]][:, None, :]
                on_i, on_j = same.any(2), same.any(1)
                if match == 2:
                    pi = pj = torch.arange(3, device=DEV)[None].expand(len(a), 3)
                else:
                    # the first common node in cyclic order: its predecessor is not common
                    def first(on):
                        return (on & ~on.roll(1, 1)).to(torch.int64).argmax(1)

                    up = torch.arange(3, device=DEV)[None]
                    pi = (first(on_i)[:, None] + up) % 3
                    pj = (first(on_j)[:, None] + 1 - up) % 3 if match == 1 else (first(on_j)[:, None] + up) % 3
                ci = torch.gather(t.c[i[a]], 1, pi[:, :, None].expand(-1, -1, 3))
                cj = torch.gather(t.c[j[a]], 1, pj[:, :, None].expand(-1, -1, 3))

                def at(c, x, y):
                    return c[:, None, 0] + x[None, :, None] * (c[:, None, 1] - c[:, None, 0]) + y[None, :, None] * (c[:, None, 2] - c[:, None, 0])

                # the difference from the common corner: exact as the points come together
                o = ci[:, :1].clone()
                r = at(cj - o, rule[:, 2], rule[:, 3]) - at(ci - o, rule[:, 0], rule[:, 1])
                v = _kernels(r, None, t.nrm[j[a]][:, None], k, ops, False)
                for op in out:
                    val[op][a] = (v[op] * rule[None, :, 4]).sum(1) * t.J[i[a]] * t.J[j[a]]
        for op in out:
            out[op][j0:j0 + len(cols)] = val[op].view(len(cols), t.n)
    return tuple(out.values())


def exact(case, seed):
    kind = case["kind"]
    if kind == "quads":
        return None  # the polar and Telles schemes of quads have no short restatement
    if kind == "sweep":
        meshes, mesh_of, ks, qs = _sweep_parts(case, seed)
        return torch.cat([_solve_cbie(*meshes[m], k, q) for m, k, q in zip(mesh_of, ks, qs)])
    k = _wave(case, seed)
    nodes, elems = _deformed(case["f"], case.get("drop", 0), seed)
    if kind == "cbie":
        k = _solvable(k)
        return _solve_cbie(nodes, elems, k, _neumann(nodes, elems, k, np.random.default_rng([seed, 3])))
    if kind == "multi":
        k = _solvable(k)
        A = _nystrom(nodes, elems, k, torch.complex64).to(torch.complex128)
        rng = np.random.default_rng([seed, 4])
        B = torch.as_tensor(np.stack([_neumann(nodes, elems, k, rng) for _ in range(case["nrhs"])]), device=DEV)
        return _gmres(lambda v: v @ A, B, tol=1e-11)
    t = Tri(nodes, elems)
    if kind == "galerkin":
        return _galerkin(t, complex(k), case["ops"])
    if kind in ("bm", "pairs"):
        c = -1j / k

        def combine(v, same):
            a, b = v[C.DLP] + c * v[C.HSP], v[C.SLP] + c * v[C.DLPT]
            return a - 0.5 * same, b + c / 2 * same

        if kind == "pairs":
            i, j = (x.to(torch.int64) for x in _near_field(t.cen, case["box"], _pair_count(case)))
            return combine(_entries(t.cen, t.nrm, t, i, j, complex(k), ALL4, True), (i == j).to(torch.float64))
        out = [torch.empty((t.n, t.n), dtype=torch.complex128, device=DEV) for _ in range(2)]

        def fill(j0, v):
            rows = torch.arange(t.n, device=DEV)[None]
            same = (rows == torch.arange(j0, j0 + len(v[C.SLP]), device=DEV)[:, None]).to(torch.float64)
            for o, q in zip(out, combine(v, same)):
                o[j0:j0 + len(q)] = q

        _matrices(t, t, complex(k), ALL4, True, fill)
        return tuple(out)
    test = Tri(*_deformed(case["ft"], case["drop"], seed + 1, radius=1.5)) if kind == "field" else t
    if kind == "host":
        S, D = _dense(t, t, complex(k), 3, True)
        D.diagonal().sub_(0.5)
        return S, D
    kc = None if case["laplace"] else complex(k, case.get("k_im", 0.0))
    return _dense(test, t, kc, case["ops"], kind == "dense")
