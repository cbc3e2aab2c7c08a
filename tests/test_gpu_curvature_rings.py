"""Curvature of meshes whose 3-rings have every shape (needs a GB300), bit for bit against the
oracle: rings longer than the 8 lanes of a vertex, isolated corners with few faces (no fit),
vertex counts at the edges of a block (16 vertices for the rings, 32 for the fits), exact
zeros in the coordinates, very small and very large meshes; and neighbourhoods past the
kernel's bounds, which are refused.
"""
import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _fan(n, closed):
    a = np.linspace(0, 2 * np.pi, n + (0 if closed else 1), endpoint=not closed)
    pts = np.concatenate([[[0.0, 0.0, 0.5]], np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(3 * a)], 1)])
    i = np.arange(1, n + 1)
    j = np.where(i == n, 1, i + 1) if closed else i + 1
    return pts, np.stack([np.zeros(n, int), i, j], 1).astype(np.int32)


def _mesh(name):
    if name.startswith("fan"):
        return _fan(int(name[3:].strip("c")), name.endswith("c"))
    kind, nu, nv = name.split("_")
    m = synth.heightfield(int(nu), ny=int(nv), seed=3, with_curvature=False) if kind != "torus" else \
        synth.torus(int(nu), int(nv), seed=3, with_curvature=False)
    p = m.points.copy()
    if kind == "flat":
        p[:, 2] = 0.0
    return p, m.faces


@pytest.mark.parametrize("name", ["fan1", "fan6", "fan7", "fan9c", "fan33", "height_2_2", "height_4_4", "height_3_5",
                                  "height_5_13", "flat_9_7", "torus_16_8", "torus_43_31"])
@pytest.mark.parametrize("scale", [1.0, 1e-120, 3e45])
def test_bits_of_the_oracle(oracle_lib, name, scale):
    pts, faces = _mesh(name)
    pts = pts * scale
    ref_ind, ref_pd = oracle_lib.Port("iso", pts, faces, 1, 0.0).curvature()
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], faces)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, faces, row, col, ev)
        ind, pd = e.compute_curvature()
    np.testing.assert_array_equal(ind, ref_ind)
    np.testing.assert_array_equal(pd, np.asarray(ref_pd).reshape(pd.shape))


@pytest.mark.parametrize("n", [193, 400])   # faces past 192; a ring past 384
def test_too_large_a_ring_is_refused(n):
    pts, faces = _fan(n, True)
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], faces)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, faces, row, col, ev)
        with pytest.raises(acvd_gb300.AcvdError):
            e.compute_curvature()
