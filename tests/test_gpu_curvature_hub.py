"""A vertex with tens of thousands of faces (needs a GB300): its neighbourhood is past the
kernels' bounds, which is found from its first 193 faces; listing every one of them in one
thread, each against all before it, took time with the square of their number.
"""
import time

import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def test_a_hub_is_refused_at_once():
    n = 60000
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    pts = np.concatenate([np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(3 * a)], 1), [[0.0, 0.0, 0.5]]])
    i = np.arange(n)
    faces = np.stack([np.full(n, n), i, (i + 1) % n], 1).astype(np.int32)   # the hub is vertex n
    row, col, ev = acvd_gb300.build_topology(n + 1, faces)
    m = synth.heightfield(9, ny=9, seed=1, with_curvature=False)
    with acvd_gb300.Engine() as e:
        r, c, v = acvd_gb300.build_topology(m.n_points, m.faces)
        e.set_mesh(m.points, m.faces, r, c, v)
        e.compute_curvature()                      # the kernels are loaded
        e.set_mesh(pts, faces, row, col, ev)
        t0 = time.monotonic()
        with pytest.raises(acvd_gb300.AcvdError):
            e.compute_curvature()
        # (1.8e9 loads and compares of one thread otherwise: seconds at the least)
        assert time.monotonic() - t0 < 3.0
