"""The calls whose speed this framework is judged by, as its users make them.

``listed()`` are twelve calls over the range in use: a whole boundary solve
(mixed and FP64 forms, one to sixteen excitations, host and device buffers,
with and without symmetry images), a frequency sweep, a batched sweep of
uneven meshes, pressure and pressure gradient at observation points, a design
gradient, and the coupled solver's boundary operators.  ``draw`` gives more
calls of the same ranges.  ``exact`` restates the discretisation in plain
64-bit torch.

A case is a dict of plain values; the fields are

    kind       which call (the ``_run_*`` functions)
    mesh       "ball" (icosphere, radius 0.1 m), "box" (rounded loudspeaker
               enclosure with a piston, 0.2 x 0.3 x 0.25 m) or "half" (the
               x >= 0 half of a sphere, closed by its mirror image)
    faces      triangles asked for
    precision  "mixed" or "fp64"
    columns    excitations (right-hand sides)
    order      order of the triangle and Duffy rules
    hz         frequency, or the lowest of several
    points     observation points or far-field directions (0: none)
    count      frequencies of a sweep, per mesh
"""
import math

import numpy as np
import torch

from beat_engine_b200 import _lib, mesh as meshes

C_AIR = 343.0
PRECISION = {"mixed": _lib.MIXED_FP32_IR, "fp64": _lib.FP64}


def _case(name, kind, mesh, faces, precision, columns, order, hz, points=0, count=1):
    c = {"kind": kind, "mesh": mesh, "faces": faces, "precision": precision, "columns": columns, "order": order,
         "hz": hz, "points": points, "count": count}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call in the tests: a coarse ball, one excitation, host arrays; launches and waits are its cost
        _case("solve_ball320", "solve", "ball", 320, "mixed", 1, 4, 400.0),
        # one frequency of an interactive request: sample-sized enclosure, second-order rules, pressure on an arc
        _case("request_box2776", "solve", "box", 2776, "mixed", 1, 2, 1000.0, points=74),
        # symmetric half model with its image pass, a few excitations, 290 observation points
        _case("symmetric_half3000", "solve", "half", 3000, "mixed", 3, 4, 1500.0, points=290),
        # enclosure in full precision, piston and four other excitations, device buffers
        _case("solve_box1992_fp64", "solve_device", "box", 1992, "fp64", 5, 4, 2000.0),
        # the full-size workload of the benchmark, one frequency alone, in both forms
        _case("solve_ball20480", "solve_device", "ball", 20480, "mixed", 16, 4, 2000.0),
        _case("solve_ball20480_fp64", "solve_device", "ball", 20480, "fp64", 16, 4, 2000.0),
        # the benchmark's own call: a sweep with far fields, frequencies pipelined over the lanes
        _case("sweep_ball20480", "sweep", "ball", 20480, "mixed", 16, 4, 500.0, points=541, count=6),
        # design variants of uneven size as one batched sweep from host arrays
        _case("batch_boxes6000", "batch", "box", 6000, "mixed", 5, 4, 250.0, points=72, count=4),
        # pressure in a plane of observation points for every excitation of a solved problem
        _case("field_box11864", "field", "box", 11864, "fp64", 16, 4, 3000.0, points=2000),
        # pressure and gradient for one excitation, some of the points close to the boundary
        _case("gradient_field_box5228", "field_gradient", "box", 5228, "fp64", 1, 4, 2000.0, points=600),
        # one step of shape optimisation: solve, far field, adjoint with vertex gradients
        _case("design_box5228_fp64", "design", "box", 5228, "fp64", 1, 4, 1000.0, points=72),
        # the coupled solver's boundary operators and their products with sparse and dense maps
        _case("coupled_box4000", "coupled", "box", 4000, "mixed", 4, 4, 700.0),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve_device", "solve_device", "sweep", "batch", "field", "field_gradient",
                       "design", "coupled"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    mesh = rng.choice(["box", "box", "half"]) if kind in ("solve", "solve_device") else "box"
    columns = rng.choice([1, 1, 2, 3, 4, 5, 7, 8, 12, 16])
    order = rng.choice([4, 4, 2])
    hz = round(math.exp(rng.uniform(math.log(100.0), math.log(3000.0))), 3)
    top = {"solve": 12000, "solve_device": 18000, "sweep": 12000, "batch": 5000, "field": 12000,
           "field_gradient": 6000, "design": 5200, "coupled": 4000}[kind]
    faces = size(300, top)
    points = {"solve": rng.choice([0, size(20, 600)]), "sweep": size(20, 541), "batch": size(20, 200),
              "field": size(50, 3000), "field_gradient": size(20, 600), "design": size(10, 150)}.get(kind, 0)
    count = rng.choice([3, 4, 5, 6]) if kind in ("sweep", "batch") else 1
    if kind in ("field_gradient", "design"):
        order = 4
    if kind in ("field", "field_gradient"):
        precision = "fp64"
    if kind in ("field_gradient", "design"):
        columns = min(columns, 4)
    return _case(None, kind, mesh, faces, precision, columns, order, hz, points, count)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _mesh(case, seed, faces=None):
    n = faces or case["faces"]
    if case["mesh"] == "ball":
        return meshes.reference_sphere(0.1, max(0, round(math.log(n / 20.0, 4))))
    if case["mesh"] == "half":
        bands = max(3, round(math.sqrt(n / 2.0)))
        return meshes.uv_sphere_patch(0.1, bands, bands, -math.pi / 2, math.pi / 2)
    return meshes.rounded_box_enclosure(n, seed=seed % 1000003)


def _wavenumbers(case, count):
    top = max(case["hz"], 3000.0)
    return [2 * math.pi * case["hz"] * (top / case["hz"]) ** (i / max(1, count - 1)) / C_AIR for i in range(count)]


def _directions(points):
    return meshes.fibonacci_sphere(points, 1.0)


def _excitations(mesh, columns, k, rng):
    """Neumann data: a piston (or the whole body along z), then random velocities, all times i rho omega."""
    q = rng.standard_normal((mesh.num_faces, columns)) + 1j * rng.standard_normal((mesh.num_faces, columns))
    piston = mesh.physical_tags == 2
    q[:, 0] = piston if piston.any() and (~piston).any() else mesh.normals[:, 2]
    q[:, 0] *= rng.uniform(0.5, 1.5)
    return np.asfortranarray(1j * 1.2 * k * C_AIR * q)


def _waves(mesh, columns, k, rng):
    """Boundary pressure and Neumann data of a few plane waves per column."""
    p = np.zeros((mesh.num_vertices, columns), dtype=complex)
    q = np.zeros((mesh.num_faces, columns), dtype=complex)
    for _ in range(4):
        d = rng.standard_normal((3, columns))
        d /= np.linalg.norm(d, axis=0)
        a = rng.standard_normal(columns) + 1j * rng.standard_normal(columns)
        p += a * np.exp(1j * k * (mesh.vertices @ d))
        q += a * (1j * k * (mesh.normals @ d)) * np.exp(1j * k * (mesh.centroids @ d))
    return np.asfortranarray(p), np.asfortranarray(q)


def _points(case, mesh, rng):
    if case["kind"] == "field_gradient":  # a sphere around the body, one point in sixteen close to a face
        far = meshes.fibonacci_sphere(case["points"], 0.5)
        near = np.arange(0, case["points"], 16)
        f = rng.integers(0, mesh.num_faces, near.size)
        away = np.sqrt(mesh.areas[f]) * rng.uniform(0.3, 2.0, near.size)
        far[near] = mesh.centroids[f] + mesh.normals[f] * away[:, None]
        return far
    if case["mesh"] == "half":
        return meshes.fibonacci_sphere(case["points"], 1.0)
    return meshes.arc_points(case["points"], 1.0) if case["points"] < 200 else \
        meshes.fibonacci_sphere(case["points"], 2.0)


def _inputs(case, seed):
    """Everything the call is given, on the host."""
    rng = np.random.default_rng(seed)
    kind, R = case["kind"], case["columns"]
    if kind == "batch":
        sizes = [max(80, round(case["faces"] * s)) for s in (0.35, 0.6, 1.0)]
        ms = [_mesh(case, seed + 7 * i, n) for i, n in enumerate(sizes)]
        ks = _wavenumbers(case, case["count"])
        q = [np.stack([_excitations(m, R, k, rng) for k in ks], axis=2) for m in ms]
        return {"meshes": ms, "k": ks, "q": [np.asfortranarray(v) for v in q], "dirs": _directions(case["points"])}
    mesh = _mesh(case, seed)
    ks = _wavenumbers(case, case["count"])
    io = {"mesh": mesh, "k": ks}
    if kind in ("field", "field_gradient"):
        io["p"], io["q"] = _waves(mesh, R, ks[0], rng)
        io["points"] = _points(case, mesh, rng)
    elif kind == "coupled":
        F = mesh.num_faces
        rows = np.arange(F)
        ncols = max(1, F // 3)  # interface map: each face's data goes to one interface unknown
        cols = rng.integers(0, ncols, F)
        by = np.argsort(cols, kind="stable")
        io["colptr"] = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=ncols))]).astype(np.int32) + 1
        io["rowval"] = (rows[by] + 1).astype(np.int32)
        io["nzval"] = rng.standard_normal(F) + 0j
        io["motion"] = rng.standard_normal((F, R)) + 1j * rng.standard_normal((F, R))
        io["prescribed"] = rng.standard_normal((F, 2)) + 1j * rng.standard_normal((F, 2))
    else:
        q = np.stack([_excitations(mesh, R, k, rng) for k in ks], axis=2)
        io["q"] = np.asfortranarray(q if kind == "sweep" else q[:, :, 0])
        if kind == "sweep" or kind == "design":
            io["dirs"] = _directions(case["points"])
        elif case["points"]:
            io["points"] = _points(case, mesh, rng)
    return io


def _device(a):
    """A column-major host array as a device tensor with the columns first (the same memory order)."""
    return torch.from_numpy(np.ascontiguousarray(a.T)).cuda()


def _context(case, mesh):
    ctx = _lib.Context(0)
    if case["mesh"] == "half":
        ctx.set_symmetry("x")
    ctx.set_mesh(mesh.vertices, mesh.faces, case["order"], case["order"])
    return ctx


def prepare(case, seed):
    io = _inputs(case, seed)
    kind = case["kind"]
    prec = PRECISION[case["precision"]]
    s = {"case": case, "io": io, "opts": _lib.Context.opts(prec)}
    if kind == "batch":
        s["ctxs"] = [_context(case, m) for m in io["meshes"]]
        return s
    mesh, R = io["mesh"], case["columns"]
    s["ctx"] = _context(case, mesh)
    V, F = mesh.num_vertices, mesh.num_faces
    if kind == "solve_device":
        s["q"], s["p"] = _device(io["q"]), torch.zeros(R, V, dtype=torch.complex128, device="cuda")
    elif kind == "sweep":
        n = case["count"]
        s["q"] = _device(io["q"])
        s["p"] = torch.zeros(n, R, V, dtype=torch.complex128, device="cuda")
        s["ff"] = torch.zeros(n, R, case["points"], dtype=torch.complex128, device="cuda")
    elif kind == "design":  # the adjoint multiplies by the mapping, so the solve keeps it
        s["opts"] = _lib.Context.opts(prec, flags=_lib.FLAG_RHS_CACHED)
    elif kind == "coupled":
        dt = torch.complex128 if case["precision"] == "fp64" else torch.complex64
        z = {"dtype": dt, "device": "cuda"}
        nq = io["colptr"].size - 1
        for key in ("nzval", "motion", "prescribed"):
            s[key] = _device(io[key]).to(dt)
        s["colptr"], s["rowval"] = torch.from_numpy(io["colptr"]).cuda(), torch.from_numpy(io["rowval"]).cuda()
        s["A"], s["C"] = torch.zeros(V, V, **z), torch.zeros(F, V, **z)
        s["interface"], s["moved"], s["rhs"] = torch.zeros(nq, V, **z), torch.zeros(R, V, **z), torch.zeros(2, V, **z)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, io, kind = s["case"], s["io"], s["case"]["kind"]
    if kind == "batch":
        ks = io["k"]
        out = _lib.sweep_batch(s["ctxs"], [ks] * len(s["ctxs"]), [[1.0 / k for k in ks]] * len(s["ctxs"]), io["q"],
                               opts=[s["opts"]] * len(s["ctxs"]), dirs=io["dirs"])
        return [[p, ff] for p, ff, _ in out]
    ctx, k = s["ctx"], io["k"][0]
    if kind == "solve":
        p, _ = ctx.solve(k, 1.0 / k, io["q"], s["opts"])
        return [p, ctx.field(k, io["points"], p, io["q"])] if case["points"] else [p]
    if kind == "solve_device":
        ctx.solve_device(k, 1.0 / k, s["q"].data_ptr(), case["columns"], s["p"].data_ptr(), s["opts"])
        return [s["p"]]
    if kind == "sweep":
        ctx.sweep_device(io["k"], [1.0 / v for v in io["k"]], s["q"].data_ptr(), case["columns"], s["p"].data_ptr(),
                         s["opts"], io["dirs"], s["ff"].data_ptr())
        return [s["p"], s["ff"]]
    if kind == "field":
        return [ctx.field(k, io["points"], io["p"], io["q"])]
    if kind == "field_gradient":
        return [ctx.field_gradient(k, io["points"], io["p"], io["q"])]
    if kind == "design":  # J = sum |p_inf|^2, so dJ / d conj(p_inf) = p_inf
        p, _ = ctx.solve(k, 1.0 / k, io["q"], s["opts"])
        ff = ctx.farfield(k, io["dirs"], p, io["q"])
        w, ga, gx = ctx.adjoint_shape(k, io["dirs"], p, io["q"], ff, s["opts"])
        return [p, ff, w, ga, gx]
    prec = PRECISION[case["precision"]]
    ctx.assemble_coupled_device(k, prec, s["A"].data_ptr(), s["C"].data_ptr())
    ctx.coupled_blocks_device(prec, s["C"].data_ptr(), s["interface"].shape[0], s["colptr"].data_ptr(),
                              s["rowval"].data_ptr(), s["nzval"].data_ptr(), s["nzval"].numel(),
                              s["interface"].data_ptr(), case["columns"], s["motion"].data_ptr(),
                              s["moved"].data_ptr(), 2, s["prescribed"].data_ptr(), s["rhs"].data_ptr())
    return [s["A"], s["C"], s["interface"], s["moved"], s["rhs"]]


def work(case):
    """Inputs read once, outputs written once; flops of the pair integration (72 a point pair), LU and solves."""
    sizes = [round(case["faces"] * s) for s in (0.35, 0.6, 1.0)] if case["kind"] == "batch" else [case["faces"]]
    R, M, n = case["columns"], case["points"], case["count"]
    Q = 6 if case["order"] == 4 else 3
    flops = nbytes = 0.0
    for F in sizes:
        N = F / 2 + 2
        images = 2 if case["mesh"] == "half" else 1
        pairs = 72.0 * Q * Q * F * F * images
        lu = (8 / 3 * N ** 3 + 8 * N * N * R)
        rhs = 8.0 * N * F * R
        eval_ = (40 + 16.0 * R) * M * F * Q * images
        if case["kind"] in ("field", "field_gradient"):
            flops += eval_ * (1 if case["kind"] == "field" else 3)
        elif case["kind"] == "coupled":
            flops += pairs + 8.0 * N * F * (R + 3)
        elif case["kind"] == "design":
            flops += 3 * pairs + lu + 2 * rhs + 8 * N * N * R + 2 * eval_
        else:
            flops += n * (pairs + lu + rhs + eval_)
        nbytes += 24 * N + 12 * F + n * 16 * R * (F + N) + 24 * M + n * 16 * R * M
        if case["kind"] == "coupled":
            nbytes += (8 if case["precision"] == "mixed" else 16) * N * (N + 4 * F / 3 + R + 2)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _triangle_rule(order):
    if order == 4:
        a, b, c, d = 0.4459484909159651, 0.0915762135097700, 0.1081030181680700, 0.8168475729804590
        pts = [(a, a), (0.0915762135097710, b), (c, a), (a, c), (d, b), (0.0915762135097710, 0.8168475729804580)]
        w = [0.2233815896780110, 0.1099517436553220, 0.2233815896780110, 0.2233815896780110, 0.1099517436553220,
             0.1099517436553220]
        w = [0.5 * v for v in w]
    else:
        pts, w = [(1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3)], [1 / 6] * 3
    pts = np.array(pts)
    return np.column_stack([1 - pts.sum(axis=1), pts]), np.array(w)  # basis values, weights (sum 1/2)


def _duffy(order, kind):
    """Points (test xi, eta, trial xi, eta, weight) of a pair sharing 3 (kind 1), 2 or 1 vertices (kind 3)."""
    x, w = np.polynomial.legendre.leggauss(order)
    x, w = (x + 1) / 2, w / 2
    xsi, e1, e2, e3 = (g.ravel() for g in np.meshgrid(x, x, x, x, indexing="ij"))
    bw = np.einsum("i,j,k,l->ijkl", w, w, w, w).ravel()
    e12, e123 = e1 * e2, e1 * e2 * e3
    if kind == 1:
        v = bw * xsi ** 3 * e1 ** 2 * e2
        t = [(xsi, xsi * (1 - e1 + e12), xsi * (1 - e123), xsi * (1 - e1), v),
             (xsi * (1 - e123), xsi * (1 - e1), xsi, xsi * (1 - e1 + e12), v),
             (xsi, xsi * (e1 - e12 + e123), xsi * (1 - e12), xsi * (e1 - e12), v),
             (xsi * (1 - e12), xsi * (e1 - e12), xsi, xsi * (e1 - e12 + e123), v),
             (xsi * (1 - e123), xsi * (e1 - e123), xsi, xsi * (e1 - e12), v),
             (xsi, xsi * (e1 - e12), xsi * (1 - e123), xsi * (e1 - e123), v)]
    elif kind == 2:
        v = bw * xsi ** 3 * e1 ** 2
        t = [(xsi, xsi * e1 * e3, xsi * (1 - e12), xsi * e1 * (1 - e2), v),
             (xsi, xsi * e1, xsi * (1 - e123), xsi * e12 * (1 - e3), v * e2),
             (xsi * (1 - e12), xsi * e1 * (1 - e2), xsi, xsi * e123, v * e2),
             (xsi * (1 - e123), xsi * e12 * (1 - e3), xsi, xsi * e1, v * e2),
             (xsi * (1 - e123), xsi * e1 * (1 - e2 * e3), xsi, xsi * e12, v * e2)]
    else:
        v = bw * xsi ** 3 * e2
        t = [(xsi, xsi * e1, xsi * e2, xsi * e2 * e3, v), (xsi * e2, xsi * e2 * e3, xsi, xsi * e1, v)]
    return np.concatenate([np.column_stack([tx - ty, ty, sx - sy, sy, u]) for tx, ty, sx, sy, u in t])


def _remap(kind, a, b, xy):
    x, y = xy[:, 0], xy[:, 1]
    if kind == 2:
        ref = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
        v0, v1, v2 = ref[a], ref[b], ref[3 - a - b]
        return v0 + x[:, None] * (v1 - v0) + y[:, None] * (v2 - v0)
    if kind == 3 and a == 1:
        return np.column_stack([1 - x - y, y])
    if kind == 3 and a == 2:
        return np.column_stack([x, 1 - x - y])
    return xy


class _Exact:
    """P1 / DP0 Burton-Miller operators of one mesh at one wavenumber, FP64."""

    def __init__(self, mesh, order, symmetry, k):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.F, self.N = mesh.num_faces, mesh.num_vertices
        self.faces_np = np.asarray(mesh.faces, dtype=np.int64)
        verts = np.array(mesh.vertices)
        self.weight = np.ones(self.N)
        if symmetry:
            on = np.abs(verts[:, 0]) <= max(1e-9, 1e-6 * np.linalg.norm(np.ptp(verts, axis=0)))
            verts[on, 0] = 0.0
            self.weight[on] = 2.0
        self.verts_np = verts
        self.X = self.t(verts)
        self.faces = torch.from_numpy(self.faces_np).to(self.dev)
        self.images = [np.ones(3)] + ([np.array([-1.0, 1.0, 1.0])] if symmetry else [])
        self.basis, self.w = _triangle_rule(order)
        self.order, self.k, self.eta = order, k, 1.0 / k
        self.touching = [self._touching(i) for i in range(len(self.images))]

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def geometry(self, X):
        v = X[self.faces]  # F, 3, 3
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        cr = torch.linalg.cross(e1, e2)
        two_a = cr.norm(dim=1)
        n = cr / two_a[:, None]
        # surface curls n x grad phi_b: with grad phi_b = n x (opposite edge) / 2A, minus that edge over 2A
        opp = torch.stack([v[:, 2] - v[:, 1], v[:, 0] - v[:, 2], v[:, 1] - v[:, 0]], dim=1)
        return {"v": v, "n": n, "area2": two_a, "curl": -opp / two_a[:, None, None],
                "pts": torch.einsum("qa,fad->fqd", self.t(self.basis), v)}

    def _touching(self, image):
        """Pairs (test, trial of this image) sharing vertex positions, with their remapped rule's key."""
        F, f = self.F, self.faces_np
        if image == 0:
            it = iv = f
        else:
            both = np.concatenate([self.verts_np, self.verts_np * self.images[image]])
            _, ids = np.unique(np.rint(both / 1e-8).astype(np.int64), axis=0, return_inverse=True)
            ids = ids.reshape(-1)
            it, iv = ids[f], ids[self.N + f]
        trial = iv.ravel()
        by = np.argsort(trial, kind="stable")
        lo, hi = np.searchsorted(trial[by], it.ravel()), np.searchsorted(trial[by], it.ravel(), side="right")
        n = hi - lo
        e = np.repeat(np.arange(3 * F), n)
        o = by[np.repeat(lo, n) + np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n)]
        pair, i, j = (e // 3) * F + o // 3, e % 3, o % 3
        s = np.lexsort((j, i, pair))
        pair, i, j = pair[s], i[s], j[s]
        first = np.flatnonzero(np.concatenate([[True], pair[1:] != pair[:-1]]))
        shared = np.diff(np.concatenate([first, [pair.size]]))
        i2, j2 = i[np.minimum(first + 1, i.size - 1)], j[np.minimum(first + 1, j.size - 1)]
        a, b = i[first], j[first]
        kind = 4 - np.minimum(shared, 3)
        swap = (kind == 2) & (j2 < b)
        a, i2 = np.where(swap, i2, a), np.where(swap, a, i2)
        b, j2 = np.where(swap, j2, b), np.where(swap, b, j2)
        two = kind == 2
        key = kind * 81 + np.where(kind == 1, 0, a * 27 + b * 9) + np.where(two, i2 * 3 + j2, 0)
        return {"t": pair[first] // F, "s": pair[first] % F, "key": key}

    def points_kernel(self, r2, nt, ns, k2n):
        """G, the system kernel -dG/dn_s - i k2n G and the right-hand-side kernel -G - i eta dG/dn_t."""
        k = self.k
        r = torch.sqrt(r2)
        g = torch.polar(1.0 / (4 * math.pi * r), k * r)
        h = g * torch.complex(-1.0 / r2, k / r)  # dG/dr / r
        return g, -(h * ns) - 1j * (k2n * g), -g + (1j * self.eta) * (h * nt)

    def pair_blocks(self, geo, lo, hi, image):
        """3 x 3 blocks, right-hand-side 3-vectors and Green sums of test faces lo..hi against every face."""
        sg = self.t(self.images[image])
        det = float(np.prod(self.images[image]))
        x, nt = geo["pts"][lo:hi], geo["n"][lo:hi]
        y, ns = geo["pts"] * sg, geo["n"] * sg
        skip = torch.zeros(hi - lo, self.F, dtype=torch.bool, device=self.dev)
        tp = self.touching[image]
        m = (tp["t"] >= lo) & (tp["t"] < hi)
        skip[self.t(tp["t"][m] - lo), self.t(tp["s"][m])] = True
        k2n = (self.eta * self.k ** 2) * (nt @ ns.T)
        Q = len(self.w)
        L = R = None
        G = 0
        for qt in range(Q):
            S, U = [0, 0, 0], 0
            for qs in range(Q):
                r = [y[None, :, qs, d] - x[:, None, qt, d] for d in range(3)]
                r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2]
                r2 = torch.where(skip, torch.ones_like(r2), r2)
                rns = r[0] * ns[None, :, 0] + r[1] * ns[None, :, 1] + r[2] * ns[None, :, 2]
                rnt = r[0] * nt[:, None, 0] + r[1] * nt[:, None, 1] + r[2] * nt[:, None, 2]
                g, lhs, rhs = self.points_kernel(r2, rnt, rns, k2n)
                w = float(self.w[qt] * self.w[qs])
                G = G + w * g
                U = U + w * rhs
                S = [S[b] + (w * float(self.basis[qs, b])) * lhs for b in range(3)]
            one = [[float(self.basis[qt, a]) * S[b] for b in range(3)] for a in range(3)]
            two = [float(self.basis[qt, a]) * U for a in range(3)]
            L = one if L is None else [[L[a][b] + one[a][b] for b in range(3)] for a in range(3)]
            R = two if R is None else [R[a] + two[a] for a in range(3)]
        jac = torch.where(skip, 0.0, geo["area2"][lo:hi, None] * geo["area2"][None, :])
        ct, cs = geo["curl"][lo:hi], geo["curl"] * sg * det
        for a in range(3):
            for b in range(3):
                L[a][b] = jac * (L[a][b] + (1j * self.eta) * (ct[:, a] @ cs[:, b].T) * G)
            R[a] = jac * R[a]
        return L, R

    def duffy_blocks(self, geo, image):
        """Per rule key: pair indices, 3 x 3 blocks and right-hand-side 3-vectors of the touching pairs."""
        sg, det, tp = self.t(self.images[image]), float(np.prod(self.images[image])), self.touching[image]
        for key in np.unique(tp["key"]):
            kind, a, b, a2, b2 = key // 81, key // 27 % 3, key // 9 % 3, key // 3 % 3, key % 3
            pts = _duffy(self.order, kind)
            bt = _remap(kind, a, a2, pts[:, 0:2])
            bs = _remap(kind, b, b2, pts[:, 2:4])
            bt = self.t(np.column_stack([1 - bt.sum(axis=1), bt]))
            bs = self.t(np.column_stack([1 - bs.sum(axis=1), bs]))
            w = self.t(pts[:, 4])
            sel = np.flatnonzero(tp["key"] == key)
            for c in range(0, sel.size, 16384):
                t, s = self.t(tp["t"][sel[c:c + 16384]]), self.t(tp["s"][sel[c:c + 16384]])
                r = torch.einsum("qa,pad->pqd", bs, geo["v"][s] * sg) - torch.einsum("qa,pad->pqd", bt, geo["v"][t])
                r2 = (r * r).sum(dim=2)
                ns, nt = geo["n"][s] * sg, geo["n"][t]
                k2n = (self.eta * self.k ** 2) * (ns * nt).sum(dim=1, keepdim=True)
                g, lhs, rhs = self.points_kernel(r2, torch.einsum("pqd,pd->pq", r, nt),
                                                 torch.einsum("pqd,pd->pq", r, ns), k2n)
                btw = (bt * w[:, None]).to(torch.complex128)
                L = torch.einsum("pq,qa,qb->pab", lhs, btw, bs.to(torch.complex128))
                curls = torch.einsum("pad,pbd->pab", geo["curl"][t], geo["curl"][s] * sg * det)
                L = L + (1j * self.eta) * curls * (g @ w.to(torch.complex128))[:, None, None]
                jac = (geo["area2"][t] * geo["area2"][s])[:, None]
                yield t, s, jac[:, :, None] * L, jac * (rhs @ btw)

    def mass(self, geo):
        """Per face: 1/2 of the P1-P1 mass block, and the P1-DP0 column times -i eta / 2."""
        b, w = self.t(self.basis), self.t(self.w)
        half = 0.5 * geo["area2"][:, None, None] * torch.einsum("q,qa,qb->ab", w, b, b)
        return half, (-0.5j * self.eta) * geo["area2"][:, None] * torch.einsum("q,qa->a", w, b)

    def operators(self):
        """A (N x N) and B (N x F) with b = B q."""
        geo, F, N = self.geometry(self.X), self.F, self.N
        z = {"dtype": torch.complex128, "device": self.dev}
        cols = [torch.zeros(N, F, **z) for _ in range(3)]
        B = torch.zeros(N, F, **z)
        step = max(16, min(F, (1 << 22) // F))
        for image in range(len(self.images)):
            part = [torch.zeros(N, F, **z) for _ in range(3)] if image else cols
            for lo in range(0, F, step):
                hi = min(F, lo + step)
                L, R = self.pair_blocks(geo, lo, hi, image)
                for a in range(3):
                    rows = self.faces[lo:hi, a]
                    B.index_add_(0, rows, R[a])
                    for b in range(3):
                        part[b].index_add_(0, rows, L[a][b])
            if image:
                for b in range(3):
                    cols[b] += part[b]
            del part
        A = torch.zeros(N, N, **z)
        for b in range(3):
            A.index_add_(1, self.faces[:, b], cols[b])
        del cols
        for image in range(len(self.images)):
            for t, s, L, R in self.duffy_blocks(geo, image):
                ft, fs = self.faces[t], self.faces[s]
                A.view(-1).index_add_(0, (ft[:, :, None] * N + fs[:, None, :]).reshape(-1), L.reshape(-1))
                B.view(-1).index_add_(0, (ft * F + s[:, None]).reshape(-1), R.reshape(-1))
        half, col = self.mass(geo)
        f = self.faces
        A.view(-1).index_add_(0, (f[:, :, None] * N + f[:, None, :]).reshape(-1), half.reshape(-1) + 0j)
        B.view(-1).index_add_(0, (f * F + torch.arange(F, device=self.dev)[:, None]).reshape(-1), col.reshape(-1))
        w = self.t(self.weight)[:, None]
        return A * w, B * w

    def sources(self, geo, p, q):
        """Weighted pressure and Neumann densities at the rule points (F, Q, R)."""
        w = (geo["area2"][:, None] * self.t(self.w)[None, :])[:, :, None]
        pv = torch.einsum("qa,far->fqr", self.t(self.basis).to(torch.complex128), p[self.faces])
        return w * pv, w * q[:, None, :]

    def far(self, X, dirs, p, q):
        geo = self.geometry(X)
        ps, qs = self.sources(geo, p, q)
        d = self.t(dirs / np.linalg.norm(dirs, axis=1, keepdims=True))
        out = 0
        for sg in self.images:
            y, n = geo["pts"] * self.t(sg), geo["n"] * self.t(sg)
            for f0 in range(0, self.F, 4096):
                f1 = min(self.F, f0 + 4096)
                ph = -self.k * torch.einsum("md,fqd->mfq", d, y[f0:f1])
                e = torch.polar(torch.full_like(ph, 1 / (4 * math.pi)), ph)
                dn = (d @ n[f0:f1].T)[:, :, None]
                out = out + torch.einsum("mfq,fqr->mr", e * (-1j * self.k) * dn, ps[f0:f1]) - \
                    torch.einsum("mfq,fqr->mr", e, qs[f0:f1])
        return out

    @staticmethod
    def point_sums(x, y, n, P, Q, k, gradient):
        """Sums over sources (dim 1) of value (and gradient); x (m, 3), y and n (m or 1, s, 3), P and Q (.., s, R)."""
        r = y - x[:, None, :]
        r2 = (r * r).sum(dim=2)
        rad = torch.sqrt(r2)
        g = torch.polar(1.0 / (4 * math.pi * rad), k * rad)
        a = torch.complex(-1.0 / rad, torch.full_like(rad, k))
        proj = (r * n).sum(dim=2) / rad
        out = [((g * a * proj)[:, :, None] * P - g[:, :, None] * Q).sum(dim=1)]
        if gradient:
            b = torch.complex(3.0 / r2 - k * k, -3.0 * k / rad)
            for d in range(3):
                u = r[:, :, d] / rad
                out.append(((g * a * u)[:, :, None] * Q -
                            (g * (b * proj * u + a / rad * n[:, :, d]))[:, :, None] * P).sum(dim=1))
        return torch.stack(out, dim=1)  # m, 1 or 4, R

    def field(self, points, p, q, gradient=False):
        geo = self.geometry(self.X)
        ps, qs = self.sources(geo, p, q)
        ps, qs = ps.reshape(1, -1, p.shape[1]), qs.reshape(1, -1, p.shape[1])
        x = self.t(points)
        out = torch.zeros(x.shape[0], 4 if gradient else 1, p.shape[1], dtype=torch.complex128, device=self.dev)
        Q = len(self.w)
        for sg in self.images:
            y = (geo["pts"] * self.t(sg)).reshape(1, -1, 3)
            n = (geo["n"] * self.t(sg)).repeat_interleave(Q, dim=0)[None]
            step = max(1, (1 << 25) // (y.shape[1] * (1 + p.shape[1])))
            for m in range(0, x.shape[0], step):
                out[m:m + step] += self.point_sums(x[m:m + step], y, n, ps, qs, self.k, gradient)
        if gradient:
            out += self.near(geo, x, p, q)
        return out

    def near(self, geo, x, p, q):
        """Faces within three diameters of a point: adaptive quadrature in place of the regular rule."""
        def size(v):
            return torch.stack([(v[:, a] - v[:, (a + 1) % 3]).norm(dim=1) for a in range(3)]).amax(dim=0)

        out = torch.zeros(x.shape[0], 4, p.shape[1], dtype=torch.complex128, device=self.dev)
        cen = geo["v"].mean(dim=1)
        away = torch.cdist(x, cen, compute_mode="donot_use_mm_for_euclid_dist")
        m, f = torch.nonzero(away <= 3 * size(geo["v"])[None], as_tuple=True)
        whole = torch.eye(3, dtype=torch.float64, device=self.dev).expand(m.numel(), 3, 3)
        fb, fw = _triangle_rule(4)

        def add(m, f, bary, basis, w, sign):  # bary: the piece's corners in the face's barycentric coordinates
            lam = torch.einsum("qa,nab->nqb", self.t(basis), bary)
            corners = torch.einsum("nab,nbd->nad", bary, geo["v"][f])
            jac = torch.linalg.cross(corners[:, 1] - corners[:, 0], corners[:, 2] - corners[:, 0]).norm(dim=1)
            wt = sign * jac[:, None, None] * self.t(w)[None, :, None]
            P = wt * torch.einsum("nqb,nbr->nqr", lam.to(torch.complex128), p[self.faces[f]])
            got = self.point_sums(x[m], torch.einsum("nqb,nbd->nqd", lam, geo["v"][f]),
                                  geo["n"][f][:, None, :].expand(-1, len(w), -1), P, wt * q[f][:, None, :], self.k,
                                  True)
            out.index_add_(0, m, got)

        add(m, f, whole, self.basis, self.w, -1.0)
        bary = whole
        while m.numel():
            corners = torch.einsum("nab,nbd->nad", bary, geo["v"][f])
            diam = size(corners)
            leaf = (diam <= 0.4 * (x[m] - corners.mean(dim=1)).norm(dim=1)) & (abs(self.k) * diam <= 0.7)
            add(m[leaf], f[leaf], bary[leaf], fb, fw, 1.0)
            m, f, bary = m[~leaf], f[~leaf], bary[~leaf]
            a, b, c = bary[:, 0], bary[:, 1], bary[:, 2]
            ab, bc, ca = (a + b) / 2, (b + c) / 2, (c + a) / 2
            bary = torch.cat([torch.stack(t, dim=1) for t in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))])
            m, f = m.repeat(4), f.repeat(4)
        return out

    def shape_gradient(self, dirs, p, q, g, z):
        """2 Re d/dX of g^H far(X) + z^H (B(X) q - A(X) p), p, q, g and z held."""
        total = torch.zeros_like(self.X)
        zc, f = z.conj(), self.faces

        def backward(part):
            X = self.X.clone().requires_grad_(True)
            part(X).real.mul(2.0).backward()
            total.add_(X.grad)

        def fars(X):
            return (g.conj() * self.far(X, dirs, p, q)).sum()

        def chunk(lo, hi):
            def value(X):
                L, R = self.pair_blocks(self.geometry(X), lo, hi, 0)
                s = 0
                for a in range(3):
                    za = zc[f[lo:hi, a]]
                    s = s + (za.unsqueeze(1) * R[a].unsqueeze(2) * q[None]).sum()
                    for b in range(3):
                        s = s - ((za @ p[f[:, b]].T) * L[a][b]).sum()
                return s
            return value

        def rest(X):
            geo = self.geometry(X)
            s = 0
            for t, tr, L, R in self.duffy_blocks(geo, 0):
                s = s + torch.einsum("par,pa,pr->", zc[f[t]], R, q[tr]) - \
                    torch.einsum("par,pab,pbr->", zc[f[t]], L, p[f[tr]])
            half, col = self.mass(geo)
            return s + torch.einsum("far,fa,fr->", zc[f], col, q) - \
                torch.einsum("far,fab,fbr->", zc[f], half.to(torch.complex128), p[f])

        backward(fars)
        step = max(8, (1 << 19) // self.F)
        for lo in range(0, self.F, step):
            backward(chunk(lo, min(self.F, lo + step)))
        backward(rest)
        return total


def exact(case, seed):
    io, kind = _inputs(case, seed), case["kind"]
    sym = case["mesh"] == "half"

    def solved(e, q):
        A, B = e.operators()
        return torch.linalg.solve(A, B @ q), A, B

    if kind == "batch":
        out = []
        for m, q in zip(io["meshes"], io["q"]):
            p, ff = [], []
            for i, k in enumerate(io["k"]):
                e = _Exact(m, case["order"], sym, k)
                qd = e.t(q[:, :, i])
                p.append(solved(e, qd)[0])
                ff.append(e.far(e.X, io["dirs"], p[-1], qd))
            out.append([torch.stack(p, dim=2).cpu().numpy(), torch.stack(ff, dim=2).cpu().numpy()])
        return out
    mesh = io["mesh"]
    if kind == "sweep":
        p, ff = [], []
        for i, k in enumerate(io["k"]):
            e = _Exact(mesh, case["order"], sym, k)
            qd = e.t(io["q"][:, :, i])
            p.append(solved(e, qd)[0])
            ff.append(e.far(e.X, io["dirs"], p[-1], qd).T)
        return [torch.stack([v.T for v in p]).contiguous(), torch.stack(ff).contiguous()]
    e = _Exact(mesh, case["order"], sym, io["k"][0])
    if kind in ("field", "field_gradient"):
        got = e.field(io["points"], e.t(io["p"]), e.t(io["q"]), kind == "field_gradient")
        return [(got if kind == "field_gradient" else got[:, 0]).cpu().numpy()]
    if kind == "coupled":  # A and C = -B, then C Q, C D and -C D
        A, B = e.operators()
        nq = io["colptr"].size - 1
        ptr = io["colptr"] - 1
        col = np.repeat(np.arange(nq), np.diff(ptr))
        Qm = torch.zeros(e.F, nq, dtype=torch.complex128, device=e.dev)
        Qm[e.t(io["rowval"].astype(np.int64) - 1), e.t(col)] = e.t(io["nzval"])
        out = [A, -B, -(B @ Qm), -(B @ e.t(io["motion"])), B @ e.t(io["prescribed"])]
        return [v.T.contiguous() for v in out]
    q = e.t(io["q"])
    p, A, B = solved(e, q)
    if kind == "solve_device":
        return [p.T.contiguous()]
    if kind == "solve":
        out = [p.cpu().numpy()]
        return out + [e.field(io["points"], p, q)[:, 0].cpu().numpy()] if case["points"] else out
    ff = e.far(e.X, io["dirs"], p, q)
    P = torch.zeros(e.F, e.N, dtype=torch.complex128, device=e.dev)  # face averages of the P1 pressure
    for a in range(3):
        P[torch.arange(e.F, device=e.dev), e.faces[:, a]] = 1 / 3
    rows = [[], []]  # far-field operators of p and of q, by columns
    d = e.t(io["dirs"] / np.linalg.norm(io["dirs"], axis=1, keepdims=True))
    geo = e.geometry(e.X)
    ph = -e.k * torch.einsum("md,fqd->mfq", d, geo["pts"])
    ker = torch.polar(torch.full_like(ph, 1 / (4 * math.pi)), ph) * (geo["area2"][:, None] * e.t(e.w)[None, :])[None]
    dn = (-1j * e.k) * (d @ geo["n"].T)
    Fq = -ker.sum(dim=2)
    Fp = torch.zeros(d.shape[0], e.N, dtype=torch.complex128, device=e.dev)
    for a in range(3):
        Fp.index_add_(1, e.faces[:, a], torch.einsum("mfq,q->mf", ker, e.t(e.basis[:, a]).to(torch.complex128)) * dn)
    z = torch.linalg.solve(A.conj().T, Fp.conj().T @ ff)
    w = B.conj().T @ z + Fq.conj().T @ ff
    ga = -(w * (P @ p).conj()).sum(dim=1)
    gx = e.shape_gradient(io["dirs"], p, q, ff, z)
    return [v.cpu().numpy() for v in (p, ff, w, ga, gx)]
