"""Dual triangles, boundary edges and cluster outputs of any labelling against numpy (needs a
GB300): face counts at and around a block of the face bits (32,768), label sets that repeat
thousands of times, more label sets than the first hash table has slots (the second one),
unassigned items, and clusters without items.
"""
import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _dual(faces, lab, k):
    t = lab[faces]
    keep = (t < k).all(1) & (t[:, 0] != t[:, 1]) & (t[:, 1] != t[:, 2]) & (t[:, 0] != t[:, 2])
    at = np.nonzero(keep)[0]
    _, first = np.unique(np.sort(t[at], axis=1), axis=0, return_index=True)
    return t[at[np.sort(first)]]


# 129 x 129: 32,768 faces; k 3: every set thousands of times; 50 and 400: up to 19,600 and
# 65,536 sets for a first table of 4,096 slots; blocks: few sets, in runs
@pytest.mark.parametrize("nu,nv", [(3, 2), (129, 129), (130, 129), (257, 258)])
@pytest.mark.parametrize("k,kind", [(3, "random"), (50, "random"), (400, "random"), (90, "blocks"), (4, "none")])
def test_dual_mesh_and_boundary_edges(nu, nv, k, kind):
    m = synth.heightfield(nu, ny=nv, seed=1, with_curvature=False)
    rng = np.random.default_rng(nu + k)
    if kind == "random":
        lab = rng.integers(0, k + 1, m.n_points)          # some items unassigned (label k)
    elif kind == "blocks":
        i, j = np.divmod(np.arange(m.n_points), nv)
        lab = (i * 9 // nu) * 9 + j * 9 // nv             # clusters 81 .. 89 stay empty
    else:
        lab = np.full(m.n_points, k)
    lab = lab.astype(np.int32)
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    with acvd_gb300.Engine() as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric("iso")
        e.set_labels(k, lab)
        np.testing.assert_array_equal(e.dual_mesh(), _dual(m.faces, lab, k))
        np.testing.assert_array_equal(e.boundary_edges(), np.nonzero(lab[ev[:, 0]] != lab[ev[:, 1]])[0])
        c = e.clusters()
    size = np.bincount(lab, minlength=k + 1)[:k]
    np.testing.assert_array_equal(c["size"], size)
    assert np.isnan(c["centroid"][size == 0]).all() and np.isfinite(c["centroid"][size > 0]).all()
    mean = c["S"][size > 0] / c["W"][size > 0, None]
    np.testing.assert_array_equal(c["centroid"][size > 0], mean)   # the isotropic vertex is S / W
