"""The work users of this framework have it do, as measurable cases.

Every case goes through the public entry points: the remesher classes of
`acvd_gb300.remesh`, `acvd_gb300.Engine` (set-up, minimisation, outputs, curvature,
subdivision), the batched solve and the autograd function of `acvd_gb300.adjoint`.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   float64 values of run()'s computed numbers, where they have any
"""
from __future__ import annotations

import math

import numpy as np
import torch

import acvd_gb300
from acvd_gb300 import adjoint, batch, remesh, synth

REMESHERS = {"iso": remesh.IsotropicDiscreteRemeshing, "qem": remesh.QIsotropicDiscreteRemeshing,
             "aniso": remesh.AnisotropicDiscreteRemeshing}
CLAMP = {"iso": 1e5, "qem": 1e4, "aniso": 1e5}     # weight clamp ratio of each metric
THRESHOLD = 1e-3                                   # relative eigenvalue threshold of the placement


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the drivers' whole call on the smallest usual mesh: a new remesher per mesh, host set-up
        # (rings, weights, sampling) and a solve of a few milliseconds, so allocations and launches count
        {"name": "remesh_icosphere5_iso", "do": "remesh", "mesh": "icosphere", "level": 5, "nu": 0, "nv": 0,
         "metric": "iso", "k": 1000, "gradation": 0.0, "manifold": False, "boundary": False},
        # ACVDQ on an open scan of odd size with every option that is used in earnest: curvature
        # computed by the call, gradation, ForceManifold, BoundaryFixing
        {"name": "remesh_height_251x187_qem", "do": "remesh", "mesh": "heightfield", "level": 0, "nu": 251, "nv": 187,
         "metric": "qem", "k": 1500, "gradation": 1.5, "manifold": True, "boundary": True},
        # minimisations from resident inputs, small to large, one per metric and use: the isotropic
        # icosphere of the configurations ...
        {"name": "solve_icosphere5_iso", "do": "solve", "mesh": "icosphere", "level": 5, "nu": 0, "nv": 0,
         "metric": "iso", "k": 1000, "gradation": 0.0},
        # ... the benchmark's torus ...
        {"name": "solve_torus_1024x512_qem", "do": "solve", "mesh": "torus", "level": 0, "nu": 1024, "nv": 512,
         "metric": "qem", "k": 20000, "gradation": 1.5},
        # ... the slice of the anisotropic heightfield that the full-size tests use ...
        {"name": "solve_height_1024_aniso", "do": "solve", "mesh": "heightfield", "level": 0, "nu": 1024, "nv": 1024,
         "metric": "aniso", "k": 12500, "gradation": 1.5},
        # ... and a ragged one whose colour classes are large (3.7 M items)
        {"name": "solve_height_2047x1801_aniso", "do": "solve", "mesh": "heightfield", "level": 0, "nu": 2047,
         "nv": 1801, "metric": "aniso", "k": 44000, "gradation": 1.5},
        # many meshes of mixed kinds and sizes in one solve
        {"name": "batch_32_qem", "do": "batch", "meshes": 32, "lo": 2000, "hi": 100000, "metric": "qem",
         "per_cluster": 20, "gradation": 0.0},
        # mesh, metric and labels from host arrays into a kept engine, solved, labels back: a stream of meshes
        {"name": "from_host_torus_517x301_qem", "do": "from_host", "mesh": "torus", "level": 0, "nu": 517, "nv": 301,
         "metric": "qem", "k": 6000, "gradation": 1.5},
        # gradients of the clustering energy and of the placed vertices, forward and backward
        {"name": "adjoint_torus_512x512", "do": "adjoint", "mesh": "torus", "level": 0, "nu": 512, "nv": 512,
         "metric": "qem", "k": 10000, "gradation": 1.0, "dtype": "float64"},
        # curvature indicator and principal directions of a whole mesh, to host arrays
        {"name": "curvature_torus_1024x512", "do": "curvature", "mesh": "torus", "level": 0, "nu": 1024, "nv": 512},
        # one level of midpoint subdivision of resident buffers
        {"name": "subdivide_torus_1024x512", "do": "subdivide", "mesh": "torus", "level": 0, "nu": 1024, "nv": 512,
         "indicator": True},
        # the coarse mesh of a clustering: cluster sums and vertices, dual triangles, boundary edges
        {"name": "coarse_torus_1024x512_qem", "do": "coarse", "mesh": "torus", "level": 0, "nu": 1024, "nv": 512,
         "metric": "qem", "k": 20000, "gradation": 1.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, lo, hi, kinds=("icosphere", "torus", "heightfield")):
    """A mesh kind and its dimensions, the vertex count log-uniform in [lo, hi]."""
    kind = rng.choice(kinds)
    n = _log_int(rng, lo, hi)
    if kind == "icosphere":
        level = int(min(8, max(3, round(math.log(n / 10.0, 4)))))
        while level > 3 and 10 * 4 ** level + 2 > hi:
            level -= 1
        return {"mesh": kind, "level": level, "nu": 0, "nv": 0}
    aspect = rng.uniform(0.4, 1.0)
    nv = max(16, int(math.sqrt(n * aspect)))
    return {"mesh": kind, "level": 0, "nu": max(16, n // nv), "nv": nv}


def draw(rng):
    do = rng.choice(("remesh", "solve", "solve", "batch", "from_host", "adjoint", "curvature", "subdivide", "coarse"))
    case = {"do": do}
    if do == "batch":
        return {**case, "meshes": rng.randint(6, 40), "lo": 2000, "hi": _log_int(rng, 8000, 100000),
                "metric": rng.choice(("qem", "iso")), "per_cluster": rng.randint(12, 40), "gradation": 0.0}
    if do == "curvature":
        return {**case, **_draw_mesh(rng, 2000, 1200000)}
    if do == "subdivide":
        return {**case, **_draw_mesh(rng, 2000, 1000000), "indicator": rng.random() < 0.5}
    if do == "adjoint":
        case.update(_draw_mesh(rng, 4000, 400000, ("torus", "heightfield")))
        case.update(metric=rng.choice(("qem", "qem", "iso")), gradation=rng.choice((0.0, 1.0, 1.5)),
                    dtype=rng.choice(("float32", "float64")))
    elif do == "coarse":
        case.update(_draw_mesh(rng, 4000, 1500000, ("torus", "heightfield")))
        case.update(metric=rng.choice(("iso", "qem")), gradation=rng.choice((0.0, 1.5)))
    elif do == "remesh":
        case.update(_draw_mesh(rng, 2500, 90000))
        case.update(metric=rng.choice(("iso", "qem", "qem", "aniso")), gradation=rng.choice((0.0, 1.5)),
                    manifold=rng.random() < 0.4, boundary=rng.random() < 0.4)
    else:
        hi = {"solve": 3000000, "from_host": 600000}[do]
        metric = rng.choice(("iso", "qem", "aniso"))
        case.update(_draw_mesh(rng, 4000, hi if metric == "aniso" else min(hi, 1200000)))
        case.update(metric=metric, gradation=rng.choice((0.0, 1.0, 1.5)))
    n = _vertices(case)
    # below 10 items per cluster the remesher subdivides first (not with the anisotropic metric)
    per = rng.uniform(5, 30) if do == "remesh" and case["metric"] != "aniso" else math.exp(
        rng.uniform(math.log(12), math.log(84)))
    return {**case, "k": max(16, int(n / per))}


# ---------------------------------------------------------------------------
# sizes and inputs
# ---------------------------------------------------------------------------

def _vertices(case):
    return 10 * 4 ** case["level"] + 2 if case["mesh"] == "icosphere" else case["nu"] * case["nv"]


def _faces(case):
    if case["mesh"] == "icosphere":
        return 20 * 4 ** case["level"]
    if case["mesh"] == "torus":
        return 2 * case["nu"] * case["nv"]
    return 2 * (case["nu"] - 1) * (case["nv"] - 1)


def _edges(case):
    n, f = _vertices(case), _faces(case)
    return {"icosphere": n + f - 2, "torus": n + f, "heightfield": n + f - 1}[case["mesh"]]


def _specs(case):
    """Kinds and sizes of a batch's meshes: the same for every seed."""
    return synth.batch_specs(case["meshes"], 0, case["lo"], case["hi"])


def _make_mesh(case, seed):
    """The generators' noise, bumps and octaves follow the seed; positions are float32 values."""
    if case["mesh"] == "icosphere":
        return synth.icosphere(case["level"], seed=seed, with_curvature=False)
    if case["mesh"] == "torus":
        return synth.torus(case["nu"], case["nv"], seed=seed, with_curvature=False)
    return synth.heightfield(case["nu"], ny=case["nv"], seed=seed, with_curvature=False)


def _density(n, seed):
    return np.random.default_rng(seed + 101).uniform(0.5, 2.0, size=n)


def _grid_labels(case, seed):
    """A clustering of a grid-like mesh into about K connected cells: the nearest of jittered
    places, one per block of the parameter grid.  Returns (labels int64 on the GPU, K).  The
    seed numbers the clusters, in no order of place, as the random sampling numbers them; the
    cells stay, so that the coarse mesh has as many triangles for every seed."""
    nu, nv, k = case["nu"], case["nv"], case["k"]
    bu = max(1, min(nu // 2, round(math.sqrt(k * nu / nv))))
    bv = max(1, min(nv // 2, round(k / bu)))
    jit = torch.tensor(np.random.default_rng(7).uniform(0.15, 0.85, size=(bu, bv, 2)), device="cuda")
    number = torch.tensor(np.random.default_rng(seed + 7).permutation(bu * bv), device="cuda")
    su, sv = nu / bu, nv / bv
    i = torch.arange(nu, device="cuda", dtype=torch.float64)
    j = torch.arange(nv, device="cuda", dtype=torch.float64)
    cu, cv = torch.clamp((i / su).long(), max=bu - 1), torch.clamp((j / sv).long(), max=bv - 1)
    best = torch.full((nu, nv), math.inf, device="cuda", dtype=torch.float64)
    lab = torch.zeros((nu, nv), device="cuda", dtype=torch.int64)
    wrap = case["mesh"] == "torus"
    for du in (-1, 0, 1):
        for dv in (-1, 0, 1):
            a, b = cu + du, cv + dv
            ok = torch.ones((nu, nv), device="cuda", dtype=torch.bool)
            if not wrap:
                ok = ((a >= 0) & (a < bu))[:, None] & ((b >= 0) & (b < bv))[None, :]
            am, bm = a % bu, b % bv
            s = jit[am][:, bm]
            pu = (a[:, None] + s[..., 0]) * su - i[:, None]
            pv = (b[None, :] + s[..., 1]) * sv - j[None, :]
            d = torch.where(ok, pu * pu + pv * pv, torch.full_like(best, math.inf))
            near = d < best
            best = torch.where(near, d, best)
            lab = torch.where(near, am[:, None] * bv + bm[None, :], lab)
    return number[lab.reshape(-1)], bu * bv


def _metric_inputs(case, engine, n, seed):
    """(indicator, principal directions) as a program gets them: the engine's curvature of the mesh
    that is set for the metrics that read it, else none."""
    use_ind = case["gradation"] != 0.0
    if not use_ind and case["metric"] != "aniso":
        return None, None
    ind, pd = engine.compute_curvature()
    return ind if use_ind else None, pd if case["metric"] == "aniso" else None


def prepare(case, seed):
    do = case["do"]
    if do == "batch":
        specs = [(kind, {**kw, "seed": seed + i}) for i, (kind, kw) in enumerate(_specs(case))]
        b = batch.batch_from_specs(specs, case["metric"], case["gradation"], case["per_cluster"])
        e = acvd_gb300.Engine()
        row, col, ev = acvd_gb300.build_topology(b.n_points, b.faces)
        e.set_mesh(b.points, b.faces, row, col, ev)
        e.set_batch(b.v_off, b.k_off)
        e.set_metric(b.metric, b.indicator, None, b.gradation)
        e.set_unconstrained_initialization(1)
        e.set_labels(b.k_total, b.labels0)
        return {"do": do, "engine": e}
    m = _make_mesh(case, seed)
    if do == "remesh":
        return {"do": do, "points": m.points, "faces": m.faces, "case": case}
    n = m.n_points
    row, col, ev = acvd_gb300.build_topology(n, m.faces)
    e = acvd_gb300.Engine()
    if do == "subdivide":
        ne, nf = ev.shape[0], m.n_faces
        g = lambda a, dt: torch.tensor(np.ascontiguousarray(a), dtype=dt, device="cuda")
        z = lambda s, dt: torch.zeros(s, dtype=dt, device="cuda")
        use = case["indicator"]
        s = {"do": do, "engine": e, "n": n, "nf": nf, "ne": ne,
             "in": [g(m.points, torch.float64), g(m.faces, torch.int32), g(row, torch.int32), g(col, torch.int32),
                    g(ev, torch.int32)], "ind": g(_density(n, seed), torch.float64) if use else None,
             "points": z((n + ne, 3), torch.float64), "faces": z((4 * nf, 3), torch.int32),
             "p1": z(ne, torch.int32), "p2": z(ne, torch.int32), "out_ind": z(n + ne, torch.float64) if use else None,
             "work": z(e.subdivide_work_bytes(ne), torch.uint8)}
        s["stream"] = torch.cuda.ExternalStream(e.stream())
        torch.cuda.synchronize()
        return s
    e.set_mesh(m.points, m.faces, row, col, ev)
    if do == "curvature":
        return {"do": do, "engine": e}
    if do in ("adjoint", "coarse"):
        lab, k = _grid_labels(case, seed)
        rho = _density(n, seed) if case["gradation"] else None
        e.set_metric(case["metric"], rho, None, case["gradation"])
        e.set_labels(k, lab.to(torch.int32).cpu().numpy())
        if do == "coarse":
            return {"do": do, "engine": e}
        dt = getattr(torch, case["dtype"])
        x = torch.tensor(m.points, dtype=dt, device="cuda").requires_grad_(True)
        r = None if rho is None else torch.tensor(rho, dtype=dt, device="cuda").requires_grad_(True)
        return {"do": do, "engine": e, "x": x, "rho": r, "gradation": case["gradation"], "target": _target(k, seed)}
    ind, pd = _metric_inputs(case, e, n, seed)
    w = acvd_gb300.vertex_weights(case["metric"], m.points, m.faces, ind, case["gradation"])
    lab = acvd_gb300.initial_sampling(row, col, w, case["k"])
    s = {"do": do, "engine": e, "case": case, "mesh": (m.points, m.faces, row, col, ev), "ind": ind, "pd": pd,
         "labels": lab}
    if do == "solve":
        _set_problem(s)
    return s


def _target(k, seed):
    return torch.tensor(np.random.default_rng(seed + 31).normal(size=(k, 3)), device="cuda")


def _set_problem(s):
    e, case = s["engine"], s["case"]
    e.set_metric(case["metric"], s["ind"], s["pd"], case["gradation"])
    e.set_unconstrained_initialization(1)
    e.set_labels(case["k"], s["labels"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _rows(a, rows):
    out = np.zeros((max(rows, a.shape[0]), a.shape[1]), dtype=a.dtype)
    out[:a.shape[0]] = a
    return out


def run(s):
    do = s["do"]
    if do == "remesh":
        case = s["case"]
        r = REMESHERS[case["metric"]]()
        r.SetInput(remesh.Surface(s["points"], s["faces"]))
        r.SetNumberOfClusters(case["k"])
        r.GetMetric().SetGradation(case["gradation"])
        r.SetUnconstrainedInitialization(1)
        r.SetForceManifold(case["manifold"])
        r.SetBoundaryFixing(int(case["boundary"]))
        r.Remesh()
        if case["metric"] == "iso":
            remesh.QuadricPostPlacement(r)     # the ACVD driver's default
        # how many vertices and triangles come out depends on the input: whole, in arrays of one size
        out, k = r.GetOutput(), case["k"]
        return {"labels": r.GetClustering(), "points": _rows(out.points, 2 * k + 64),
                "faces": _rows(out.faces, 6 * k + 64), "energy": r.Energy}
    e = s["engine"]
    if do == "subdivide":
        a = [t.data_ptr() for t in s["in"]]
        p = lambda t: None if t is None else t.data_ptr()
        e.subdivide_device(s["n"], a[0], s["nf"], a[1], a[2], a[3], s["ne"], a[4], p(s["ind"]), p(s["points"]),
                           p(s["faces"]), p(s["p1"]), p(s["p2"]), p(s["out_ind"]), p(s["work"]))
        torch.cuda.current_stream().wait_stream(s["stream"])
        return {k: s[k] for k in ("points", "faces", "p1", "p2", "out_ind")}
    if do == "curvature":
        ind, pd = e.compute_curvature()
        return {"indicator": ind, "directions": pd}
    if do == "adjoint":
        s["x"].grad = None
        if s["rho"] is not None:
            s["rho"].grad = None
        energy, cent = adjoint.ClusteringEnergy.apply(s["x"], s["rho"], e, s["gradation"])
        (energy + (cent * s["target"]).sum()).backward()
        return {"energy": energy.detach(), "centroids": cent.detach(), "grad_x": s["x"].grad,
                "grad_rho": None if s["rho"] is None else s["rho"].grad}
    if do == "coarse":
        c = e.clusters()
        return {"clusters": c, "dual": e.dual_mesh(), "boundary": e.boundary_edges()}
    if do == "from_host":
        e.set_mesh(*s["mesh"])
        _set_problem(s)
    else:
        e.rewind()
    st = e.minimize()
    return {"labels": e.labels(), "energy": e.mesh_energies() if do == "batch" else np.float64(st["energy"])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    do = case["do"]
    if do == "batch":
        n = sum(batch.spec_items(s) for s in _specs(case))
        ne, nf, k = 3 * n, 2 * n, n // case["per_cluster"]
    else:
        n, nf, ne, k = _vertices(case), _faces(case), _edges(case), case.get("k", 0)
    rings = 4 * (n + 1) + 8 * ne                       # CSR of the vertex rings
    mesh = 24 * n + 12 * nf + rings + 8 * ne           # positions, faces, rings, edges
    if do == "subdivide":
        ind = 8 * n + 8 * (n + ne) if case["indicator"] else 0
        return {"bytes": mesh + 24 * (n + ne) + 48 * nf + 8 * ne + ind, "flops": 6 * ne}
    if do == "curvature":
        # 54 faces in a regular 3-ring: frame, local coordinates and normal equations, then a 6 x 6 inverse
        return {"bytes": mesh + 32 * n, "flops": (54 * 110 + 900) * n}
    if do == "adjoint":
        size = 8 if case["dtype"] == "float64" else 4
        rho = 2 * size * n if case["gradation"] else 0
        return {"bytes": 12 * nf + 4 * n + 6 * size * n + rho + 48 * k, "flops": 300 * nf + 150 * n + 2000 * k}
    record = {"iso": 16, "qem": 40, "aniso": 64}[case["metric"]]   # float32 record of an item
    sums = {"iso": 4, "qem": 13, "aniso": 22}[case["metric"]]
    if do == "coarse":
        return {"bytes": (record + 4) * n + 12 * nf + 8 * ne + 8 * (3 + 1 + 9 + 3 + 1) * k + 4 * k + 24 * k + 12 * ne // 4,
                "flops": 2 * sums * n + 500 * k}
    solve = (record + 8) * n + rings + 8 * sums * k    # items, labels in and out, rings, cluster sums
    if do in ("solve", "batch"):
        return {"bytes": solve, "flops": 200 * n}
    host = mesh + (8 * n if case["gradation"] else 0) + (24 * n if case["metric"] == "aniso" else 0) + 4 * n
    if do == "from_host":
        return {"bytes": host + solve, "flops": 400 * n}
    return {"bytes": host + solve + 4 * n + 24 * k + 24 * k, "flops": 500 * n}


# ---------------------------------------------------------------------------
# float64 values
# ---------------------------------------------------------------------------

def exact(case, seed):
    if case["do"] == "subdivide":
        return _exact_subdivide(case, seed)
    if case["do"] == "curvature":
        return _exact_curvature(case, seed)
    if case["do"] in ("adjoint", "coarse"):
        return _exact_fixed(case, seed)
    return None      # a minimisation: its labels are whole numbers, its energy that of its own labels


def _exact_subdivide(case, seed):
    m = _make_mesh(case, seed)
    f = m.faces.astype(np.int64)
    # edges numbered by first appearance over the faces' sides
    sides = np.stack([f, np.roll(f, -1, axis=1)], axis=2).reshape(-1, 2)
    key = sides.min(axis=1) * m.n_points + sides.max(axis=1)
    _, first = np.unique(key, return_index=True)
    ends = sides[np.sort(first)]
    mid = 0.5 * (m.points[ends[:, 0]] + m.points[ends[:, 1]])
    pts = np.concatenate([m.points, mid])
    ind = None
    if case["indicator"]:
        d = _density(m.n_points, seed)
        ind = np.concatenate([d, 0.5 * (d[ends[:, 0]] + d[ends[:, 1]])])
    return {"points": pts.astype(np.float32).astype(np.float64), "faces": None, "p1": None, "p2": None,
            "out_ind": ind}


def _ring_faces(faces, n):
    """The faces of every vertex's 3-ring: (vertex, face) pairs, each once, sorted by vertex.
    They are the faces with a corner at most two edges away."""
    f = torch.tensor(faces, dtype=torch.int64, device="cuda")
    nf = f.shape[0]
    flat = f.reshape(-1)
    order = torch.argsort(flat, stable=True)
    vf = torch.div(order, 3, rounding_mode="floor")
    start = torch.searchsorted(flat[order], torch.arange(n + 1, device="cuda"))

    def expand(owner, vert):
        """Each (owner, vertex) pair into (owner, face of the vertex)."""
        cnt = start[vert + 1] - start[vert]
        own = torch.repeat_interleave(owner, cnt)
        base = torch.repeat_interleave(start[vert] - (torch.cumsum(cnt, 0) - cnt), cnt)
        return own, vf[base + torch.arange(own.numel(), device="cuda")]

    def unique(own, x, top):
        key = torch.unique(own * top + x)
        return torch.div(key, top, rounding_mode="floor"), key % top

    def closure(lo, hi):
        own = torch.arange(lo, hi, device="cuda")
        vert = own.clone()
        for _ in range(2):
            o, g = expand(own, vert)
            own, vert = unique(torch.repeat_interleave(o, 3), f[g].reshape(-1), n)
        return unique(*expand(own, vert), nf)

    for lo in range(0, n, 1 << 17):
        yield lo, min(n, lo + (1 << 17)), closure(lo, min(n, lo + (1 << 17)))


def _exact_curvature(case, seed):
    m = _make_mesh(case, seed)
    n = m.n_points
    p = torch.tensor(m.points, device="cuda")
    f = torch.tensor(m.faces, dtype=torch.int64, device="cuda")
    x1, x2, x3 = p[f[:, 0]], p[f[:, 1]], p[f[:, 2]]
    nrm = torch.linalg.cross(x3 - x2, x1 - x2)
    length = nrm.norm(dim=1, keepdim=True)
    area, nrm, bary = 0.5 * length[:, 0], nrm / length, (x1 + x2 + x3) / 3.0
    ind = torch.zeros(n, dtype=torch.float64, device="cuda")
    dirs = torch.zeros((n, 6), dtype=torch.float64, device="cuda")
    for lo, hi, (own, face) in _ring_faces(m.faces, n):
        c = hi - lo
        own = own - lo
        add = lambda v: torch.zeros((c,) + v.shape[1:], dtype=torch.float64, device="cuda").index_add_(0, own, v)
        cnt = add(torch.ones(own.numel(), dtype=torch.float64, device="cuda"))
        a = area[face]
        origin = add(a[:, None] * bary[face]) / add(a)[:, None]
        f2 = torch.nn.functional.normalize(add(a[:, None] * nrm[face]), dim=1)
        f0 = torch.nn.functional.normalize(torch.linalg.cross(f2[:, [2, 0, 1]], f2), dim=1)
        f1 = torch.linalg.cross(f2, f0)
        q = bary[face] - origin[own]
        x, y, z = ((q * g[own]).sum(1) for g in (f0, f1, f2))
        h = add(torch.sqrt(x * x + y * y)) / cnt
        u, v = x / h[own], y / h[own]
        r = torch.stack([torch.ones_like(u), u, v, u * u, u * v, v * v], 1)
        M = torch.stack([add(r * r[:, j:j + 1]) for j in range(6)], 2)
        rhs = add(r * z[:, None])
        enough = cnt > 6
        M[~enough] = torch.eye(6, dtype=torch.float64, device="cuda")
        w = torch.linalg.solve(M, rhs[:, :, None])[:, :, 0]
        w = w / torch.stack([torch.ones_like(h), h, h, h * h, h * h, h * h], 1)
        E, F, G = 1 + w[:, 1] ** 2, w[:, 1] * w[:, 2], 1 + w[:, 2] ** 2
        s = torch.sqrt(1 + w[:, 1] ** 2 + w[:, 2] ** 2)
        e, ff, g = 2 * w[:, 3] / s, 2 * w[:, 4] / s, 2 * w[:, 5] / s
        det = E * G - F * F
        a00, a01 = -(e * G - ff * F) / det, -(ff * G - g * F) / det
        a11 = -(g * E - ff * F) / det
        # the rotation by at most 45 degrees that makes the symmetric matrix (a00 a01; a01 a11) diagonal
        theta = (a11 - a00) / torch.where(a01 == 0, torch.ones_like(a01), 2 * a01)
        t = torch.where(theta >= 0, 1.0, -1.0) / (theta.abs() + torch.sqrt(theta * theta + 1))
        t = torch.where(a01 == 0, torch.zeros_like(t), t)
        cs = 1 / torch.sqrt(t * t + 1)
        sn = t * cs
        k0, k1 = a00 - t * a01, a11 + t * a01
        d0 = cs[:, None] * f0 - sn[:, None] * f1
        d1 = sn[:, None] * f0 + cs[:, None] * f1
        d0, d1 = torch.sqrt(k0.abs())[:, None] * d0, torch.sqrt(k1.abs())[:, None] * d1
        # the larger |k| first, the larger k where both are alike
        swap = ((k1.abs() > k0.abs()) | ((k1.abs() == k0.abs()) & (k1 > k0)))[:, None]
        both = torch.cat([torch.where(swap, d1, d0), torch.where(swap, d0, d1)], 1)
        ind[lo:hi] = torch.where(enough, torch.sqrt(k0 * k0 + k1 * k1), torch.zeros_like(k0))
        dirs[lo:hi] = torch.where(enough[:, None], both, torch.zeros_like(both))
    return {"indicator": ind, "directions": dirs}


def _exact_fixed(case, seed):
    """Cluster sums, placed vertices and energies of a fixed clustering, and (adjoint) the gradients."""
    m = _make_mesh(case, seed)
    n, grads = m.n_points, case["do"] == "adjoint"
    lab, k = _grid_labels(case, seed)
    f = torch.tensor(m.faces, dtype=torch.int64, device="cuda")
    rho = torch.tensor(_density(n, seed), device="cuda") if case["gradation"] else None
    if grads and case["dtype"] == "float32" and rho is not None:
        rho = rho.float().double()
    x = torch.tensor(m.points, device="cuda").requires_grad_(grads)
    if rho is not None:
        rho.requires_grad_(grads)
    a, b, c = x[f[:, 0]], x[f[:, 1]], x[f[:, 2]]
    cr = torch.linalg.cross(b - a, c - a)
    length = cr.norm(dim=1)
    nrm = cr / length[:, None]
    corners = f.reshape(-1)
    per_vertex = lambda v: torch.zeros((n,) + v.shape[1:], dtype=torch.float64, device="cuda").index_add(
        0, corners, v.repeat_interleave(3, 0))
    dual = per_vertex(length / 6.0)
    Av = per_vertex(nrm[:, :, None] * nrm[:, None, :])
    w = dual if rho is None else dual * rho ** case["gradation"]
    with torch.no_grad():
        mean, ratio = w.mean(), CLAMP[case["metric"]]
    w = torch.clamp(w, min=float(mean) / ratio, max=float(mean) * ratio)
    per_cluster = lambda v: torch.zeros((k,) + v.shape[1:], dtype=torch.float64, device="cuda").index_add(0, lab, v)
    S, W, A = per_cluster(w[:, None] * x), per_cluster(w), per_cluster(Av)
    B = per_cluster((Av @ x[:, :, None])[:, :, 0])
    cent = S / W[:, None]
    if case["metric"] != "iso":
        res = B - (A @ cent[:, :, None])[:, :, 0]
        lam, V = torch.linalg.eigh(A)
        with torch.no_grad():
            keep = lam.abs() > THRESHOLD * lam.abs().max(1, keepdim=True).values
            full = keep.all(1)
        inv = torch.where(keep, 1 / lam, torch.zeros_like(lam))
        part = torch.where(full, torch.zeros_like(W), torch.ones_like(W))[:, None]
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        d = (torch.linalg.solve(torch.where(full[:, None, None], A, eye), (1 - part) * res))
        if bool((~full).any()):
            at = (~full).nonzero()[:, 0]
            lam_p, V_p = torch.linalg.eigh(A[at])
            inv_p = torch.where(keep[at], 1 / lam_p, torch.zeros_like(lam_p))
            d_p = (V_p @ (inv_p[:, :, None] * (V_p.transpose(1, 2) @ res[at][:, :, None])))[:, :, 0]
            d = d.index_put((at,), d_p)
        cent = cent + d
    energy = W * (cent * cent).sum(1) - 2 * (cent * S).sum(1)
    if grads:
        (energy.sum() + (cent * _target(k, seed)).sum()).backward()
        return {"energy": energy.sum().detach(), "centroids": cent.detach(), "grad_x": x.grad,
                "grad_rho": None if rho is None else rho.grad}
    Q = torch.stack([A[:, 0, 0], A[:, 0, 1], A[:, 0, 2], -B[:, 0], A[:, 1, 1], A[:, 1, 2], -B[:, 1], A[:, 2, 2],
                     -B[:, 2]], 1)
    return {"clusters": {"size": None, "S": S, "W": W, "Q": Q * (case["metric"] != "iso"), "centroid": cent,
                         "energy": energy, "energy_total": float(energy.sum())}, "dual": None, "boundary": None}
