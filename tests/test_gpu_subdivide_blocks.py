"""Subdivision at the edges of its kernels' warps and blocks (needs a GB300): a thread takes one
face, and one edge, so that 32 of them are a warp and 256 a block; below, at and above these
the last warp stages and writes a part of its rows.  Fans of n faces have 2 n + 1 edges; an
even number of edges comes from a closed fan (2 n).  All values are exact.
"""
import numpy as np
import pytest

import acvd_gb300
from test_gpu_subdivide import _fan, _run

pytestmark = pytest.mark.gpu


def _closed(n):
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    pts = np.concatenate([[[0.0, 0.0, 1.0]], np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(2 * a)], 1)])
    i = np.arange(1, n + 1)
    return pts, np.stack([np.zeros(n, int), i, np.where(i == n, 1, i + 1)], 1).astype(np.int32)


# faces at a warp and a block; edges: open 15 -> 31, 16 -> 33, 127 -> 255, 128 -> 257, closed 16 ->
# 32, 128 -> 256
@pytest.mark.parametrize("closed,n", [(False, n) for n in (15, 16, 31, 32, 33, 127, 128, 255, 256, 257)] +
                         [(True, n) for n in (16, 32, 128, 256)])
@pytest.mark.parametrize("with_ind,odd", [(False, 1), (True, 0)])
def test_one_level(closed, n, with_ind, odd):
    pts, faces = _closed(n) if closed else _fan(n)
    nv = pts.shape[0]
    row, col, ev = acvd_gb300.build_topology(nv, faces)
    assert len(ev) == 2 * n + (not closed)
    ind = np.random.default_rng(n).uniform(0.5, 2.0, nv) if with_ind else None
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


@pytest.mark.parametrize("n", [31, 32, 33, 255, 256, 257])
def test_reported_faces_at_the_ends_of_a_block(n):
    """Faces that are reported are left unwritten, the first and the last of a warp and a block
    among them, and the others are written."""
    pts, faces = _fan(n)
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], faces)
    wrong = sorted({0, 30, 31, 32, 254, 255, 256, n - 1} & set(range(n)))
    bad = faces.copy()
    bad[wrong, 1] = bad[wrong, 0]
    t, missing = np.array(_run(pts, bad, row, col, ev, None, 0)[1]).reshape(-1, 12), \
        _run(pts, bad, row, col, ev, None, 0)[5]
    good = _run(pts, faces, row, col, ev, None, 0)[1].reshape(-1, 12)
    assert missing == len(wrong) and (t[wrong] == -7).all()
    keep = np.setdiff1d(np.arange(n), wrong)
    np.testing.assert_array_equal(t[keep], good[keep])
