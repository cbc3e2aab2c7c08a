"""The evaluation's local connectivity test on short and long rings (needs a GB300).

An item with at most 8 neighbours takes the test from a packed adjacency (a byte of ring
slots for each ring slot); a longer ring reads the adjacency words of its CSR slots.  Both
answer the same question, so converged labels are those that the CSR walk alone gave for
every ring (the hashes below), on meshes whose degrees lie on both sides of 8.
"""
import hashlib

import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu

# (grid points per side, share of triangles split at their centre, clusters)
MESHES = [(24, 0.35, 33), (70, 0.2, 257), (70, 0.6, 500)]
LABELS = {
    ("iso", 24, 33): "e09dff400cd6f75d",
    ("iso", 70, 257): "bc0ed801825f2dc7",
    ("iso", 70, 500): "18bbb5241e2dc7f9",
    ("qem", 24, 33): "4ed2f6e73ddc035b",
    ("qem", 70, 257): "cffba1098f0b2993",
    ("qem", 70, 500): "9e1930399fb3d74c",
}


def _mesh(n, share):
    """A height field with some triangles split in three: degrees 3 to 12."""
    m = synth.heightfield(n, ny=n, seed=3)
    pts, tri = np.asarray(m.points, np.float64), np.asarray(m.faces)
    pick = np.random.default_rng(n).random(len(tri)) < share
    s = tri[pick]
    new = len(pts) + np.arange(len(s))
    parts = [np.stack([s[:, a], s[:, (a + 1) % 3], new], 1) for a in range(3)]
    return np.concatenate([pts, pts[s].mean(1)]), np.concatenate([tri[~pick], *parts]).astype(tri.dtype)


def _labels(metric, n, share, k):
    pts, tri = _mesh(n, share)
    row, col, ev = acvd_gb300.build_topology(len(pts), tri)
    deg = np.diff(np.asarray(row))
    assert {4, 7, 8, 9} <= set(deg.tolist())
    w = acvd_gb300.vertex_weights(metric, pts, tri)
    lab = acvd_gb300.initial_sampling(row, col, w, k)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, tri, row, col, ev)
        e.set_metric(metric, None, None, 0.0)
        e.set_labels(k, lab)
        e.minimize()
        return e.labels()


@pytest.mark.parametrize("metric", ["iso", "qem"])
@pytest.mark.parametrize("n,share,k", MESHES)
def test_labels_on_mixed_degrees(metric, n, share, k):
    lab = _labels(metric, n, share, k)
    assert hashlib.sha256(lab.tobytes()).hexdigest()[:16] == LABELS[metric, n, k]
