"""Curvature in several chunks of vertices (needs a GB300), as meshes of more than 524,288 run:
bit for bit the values of one chunk and of the oracle, for chunks of one vertex, below and
above the blocks of the rings (16) and of the fits (32), with and without a short last one;
and a neighbourhood past the kernels' bounds is found in any of them.
"""
import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _curvature(pts, faces, chunk, monkeypatch):
    if chunk is None:
        monkeypatch.delenv("ACVD_CURV_CHUNK", raising=False)
    else:
        monkeypatch.setenv("ACVD_CURV_CHUNK", str(chunk))
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], faces)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, faces, row, col, ev)
        return e.compute_curvature()


# 17 x 13 = 221 vertices; the last chunk holds 1, 11, 23, 29, 110, 1 and 221 of them
@pytest.mark.parametrize("chunk", [1, 15, 33, 32, 111, 220, 221])
def test_chunks(oracle_lib, monkeypatch, chunk):
    m = synth.heightfield(17, ny=13, seed=4, with_curvature=False)
    ref_ind, ref_pd = oracle_lib.Port("iso", m.points, m.faces, 1, 0.0).curvature()
    ind, pd = _curvature(m.points, m.faces, chunk, monkeypatch)
    np.testing.assert_array_equal(ind, ref_ind)
    np.testing.assert_array_equal(pd, np.asarray(ref_pd).reshape(pd.shape))


def test_more_than_one_default_chunk(monkeypatch):
    """1024 x 515 vertices: one chunk of 524,288 and one of 3,072; the values are those of one."""
    m = synth.torus(1024, 515, seed=2, with_curvature=False)
    a = _curvature(m.points, m.faces, None, monkeypatch)
    b = _curvature(m.points, m.faces, 1 << 20, monkeypatch)
    c = _curvature(m.points, m.faces, 100000, monkeypatch)
    for other in (b, c):
        np.testing.assert_array_equal(a[0], other[0])
        np.testing.assert_array_equal(a[1], other[1])


@pytest.mark.parametrize("hub", [0, 150, 300])
def test_a_bad_neighbourhood_in_any_chunk(monkeypatch, hub):
    n = 300
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    rim = np.delete(np.arange(n + 1), hub)
    pts = np.zeros((n + 1, 3))
    pts[rim] = np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(3 * a)], 1)
    faces = np.stack([np.full(n, hub), rim, np.roll(rim, -1)], 1).astype(np.int32)
    with pytest.raises(acvd_gb300.AcvdError):
        _curvature(pts, faces, 64, monkeypatch)
