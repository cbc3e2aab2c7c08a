"""Curvature where the fits' quotients leave the range in which they share a reciprocal (needs
a GB300), bit for bit against the oracle: meshes squeezed along an axis by powers of two and
ten until products of two coordinates lie at the bottom of the range, below it, or vanish,
and as large.
"""
import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu

SQUEEZE = [(1, 2.0 ** -232, 1), (1, 2.0 ** -233, 1), (1, 1e-80, 1), (1, 1, 1e-90), (1e-75, 1, 1e-75), (1, 1e-110, 1e-40),
           (1, 1e-130, 1), (1, 1e-160, 1), (1e37, 1, 1), (1e60, 1e60, 1e60), (1e-37, 1e-37, 1e-37), (1e-60, 1e10, 1e-60),
           (1, 1e-200, 1e-100), (1e70, 1e70, 1e-60), (1e-100, 1e-100, 1e-100), (1, 1e-300, 1)]


@pytest.mark.parametrize("scale", SQUEEZE, ids=lambda s: "%.3g_%.3g_%.3g" % tuple(s))
@pytest.mark.parametrize("kind", ["height", "grid", "torus"])
def test_bits_of_the_oracle(oracle_lib, kind, scale):
    m = synth.torus(14, 9, seed=3, with_curvature=False) if kind == "torus" else \
        synth.heightfield(9, ny=8, seed=3, with_curvature=False)
    pts = m.points.copy()
    if kind == "grid":   # centred, so that coordinates and their sums are exactly zero
        i, j = np.divmod(np.arange(72), 8)
        pts = np.stack([i - 4.0, j - 4.0, 0.25 * ((i - 4.0) ** 2 - (j - 4.0) ** 2)], 1)
    pts = pts * np.array(scale)
    ref_ind, ref_pd = oracle_lib.Port("iso", pts, m.faces, 1, 0.0).curvature()
    row, col, ev = acvd_gb300.build_topology(pts.shape[0], m.faces)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, m.faces, row, col, ev)
        ind, pd = e.compute_curvature()
    np.testing.assert_array_equal(ind, ref_ind)
    np.testing.assert_array_equal(pd, np.asarray(ref_pd).reshape(pd.shape))
