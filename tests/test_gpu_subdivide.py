"""Subdivision on device buffers against numpy (needs a GB300): face counts around a warp's 8
and a block's 64 faces, rings longer than 8, buffers at odd element offsets, with and without
an indicator, and faces that are reported instead of subdivided.  All values are exact.
"""
import numpy as np
import pytest
import torch

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _fan(n):
    """n triangles around one vertex: a ring of n + 1 and an open boundary."""
    a = np.linspace(0, 2 * np.pi, n + 1)
    pts = np.concatenate([[[0.0, 0.0, 1.0]], np.stack([np.cos(a), np.sin(a), 0.1 * a], 1)])
    return pts, np.stack([np.zeros(n, int), np.arange(1, n + 1), np.arange(2, n + 2)], 1).astype(np.int32)


def _mesh(name):
    if name.startswith("fan"):
        return _fan(int(name[3:]))
    m = synth.torus(13, 11, seed=3, with_curvature=False) if name == "torus" else synth.icosphere(2, seed=1)
    return m.points, m.faces


def _run(pts, faces, row, col, ev, ind, odd):
    """Device buffers start one element into their allocations when odd."""
    def dev(a, dt):
        t = torch.zeros(a.size + 1, dtype=dt, device="cuda")
        t[odd:odd + a.size] = torch.tensor(a.reshape(-1), dtype=dt)
        return t[odd:odd + a.size]
    nv, nf, ne = pts.shape[0], faces.shape[0], ev.shape[0]
    i32, f64 = torch.int32, torch.float64
    x, t, r, c, e = dev(pts, f64), dev(faces, i32), dev(row, i32), dev(col, i32), dev(ev, i32)
    d = None if ind is None else dev(ind, f64)
    z = lambda n, dt: dev(np.full(n, -7), dt)
    out = [z(3 * (nv + ne), f64), z(12 * nf, i32), z(ne, i32), z(ne, i32), None if ind is None else z(nv + ne, f64)]
    with acvd_gb300.Engine() as g:
        work = torch.zeros(g.subdivide_work_bytes(ne) // 4, dtype=i32, device="cuda")
        p = lambda a: None if a is None else a.data_ptr()
        torch.cuda.synchronize()
        g.subdivide_device(nv, p(x), nf, p(t), p(r), p(c), ne, p(e), p(d), *[p(o) for o in out], p(work))
        torch.cuda.synchronize()
    return [None if o is None else o.cpu().numpy() for o in out] + [int(work[2 * ne].item())]


@pytest.mark.parametrize("name", ["fan1", "fan7", "fan8", "fan9", "fan63", "fan65", "torus", "sphere"])
@pytest.mark.parametrize("with_ind,odd", [(False, 0), (True, 1)])
def test_one_level(name, with_ind, odd):
    pts, faces = _mesh(name)
    nv = pts.shape[0]
    row, col, ev = acvd_gb300.build_topology(nv, faces)
    ind = np.random.default_rng(0).uniform(0.5, 2.0, nv) if with_ind else None
    x, t, p1, p2, oi, missing = _run(pts, faces, row, col, ev, ind, odd)
    a, b = ev[:, 0], ev[:, 1]
    want = np.concatenate([pts, 0.5 * (pts[a] + pts[b])]).astype(np.float32).astype(np.float64)
    np.testing.assert_array_equal(x.reshape(-1, 3), want)
    np.testing.assert_array_equal(p1, a)
    np.testing.assert_array_equal(p2, b)
    if with_ind:
        np.testing.assert_array_equal(oi, np.concatenate([ind, (ind[a] + ind[b]) * 0.5]))
    edge = {frozenset(q): nv + i for i, q in enumerate(ev.tolist())}
    rows = []
    for v1, v2, v3 in faces.tolist():
        v4, v5, v6 = edge[frozenset((v1, v2))], edge[frozenset((v2, v3))], edge[frozenset((v3, v1))]
        rows += [v1, v4, v6, v4, v2, v5, v5, v3, v6, v4, v5, v6]
    np.testing.assert_array_equal(t, rows)
    assert missing == 0


def test_bad_faces_are_reported():
    pts, faces = _fan(20)
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], faces)
    bad = faces.copy()
    bad[3, 1] = pts.shape[0]      # a corner out of range
    bad[9, 2] = -1
    bad[10, 1] = bad[10, 0]       # an inactive face
    bad[15] = [1, 5, 9]           # no such edges
    x, t, p1, p2, oi, missing = _run(pts, bad, row, col, ev, None, 0)
    good = _run(pts, faces, row, col, ev, None, 0)[1].reshape(-1, 12)
    t = t.reshape(-1, 12)
    wrong = [3, 9, 10, 15]
    assert missing == len(wrong)
    assert (t[wrong] == -7).all()
    keep = np.setdiff1d(np.arange(20), wrong)
    np.testing.assert_array_equal(t[keep], good[keep])


def test_rounding_over_the_whole_range():
    """Zeros of both signs, values around the smallest normal and denormal floats, ties, the
    largest float and what rounds past it, infinities and NaN."""
    f = np.float32
    tie = float(np.nextafter(f(1), f(2)))
    v = [0.0, -0.0, 1e-300, 5e-324, 2.0 ** -126, 2.0 ** -126 * (1 - 2.0 ** -25), 2.0 ** -149, 2.0 ** -150, 3e-46,
         1.0 + 2.0 ** -24, tie + 2.0 ** -24, 1.0 + 2.0 ** -24 + 2.0 ** -50, 2.0 ** 126 * 1.9999999, 2.0 ** 127,
         float(np.finfo(f).max), 3.4028235677973366e38, 3.4028235e38, 1e39, 1.7e308, np.inf, -np.inf, np.nan, 0.1, -7.3]
    v += [-x for x in v[:18]]
    pts, faces = _fan(3 * len(v) // 3)
    rng = np.random.default_rng(1)
    pts = np.array(v)[rng.integers(0, len(v), pts.shape)]
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], faces)
    ind = np.array(v)[rng.integers(0, len(v), pts.shape[0])]
    x, t, p1, p2, oi, missing = _run(pts, faces, row, col, ev, ind, 0)
    a, b = ev[:, 0], ev[:, 1]
    with np.errstate(all="ignore"):
        want = np.concatenate([pts, 0.5 * (pts[a] + pts[b])]).astype(np.float32).astype(np.float64)
        want_ind = np.concatenate([ind, (ind[a] + ind[b]) * 0.5])
    np.testing.assert_array_equal(x.reshape(-1, 3), want)
    np.testing.assert_array_equal(np.signbit(x.reshape(-1, 3))[want == 0], np.signbit(want)[want == 0])
    np.testing.assert_array_equal(oi, want_ind)
