"""The cluster schedule in several launches (needs a GB300): a launch returns after a number of
sweeps with its loop state on the device, and the next goes on from there.  Launches of 1 and
3 sweeps give the labels, energies and counts of one launch and of the per-phase graphs.
"""
import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _solve(monkeypatch, metric, run, limit, loops=20000):
    monkeypatch.setenv("ACVD_CLUSTER_MAX", limit)
    if run is None:
        monkeypatch.delenv("ACVD_CLUSTER_RUN", raising=False)
    else:
        monkeypatch.setenv("ACVD_CLUSTER_RUN", str(run))
    m = synth.heightfield(61, ny=47, seed=6, with_curvature=metric == "aniso")
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    lab = acvd_gb300.initial_sampling(row, col, acvd_gb300.vertex_weights(metric, m.points, m.faces), 140)
    with acvd_gb300.Engine(max_loops=loops) as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric(metric, None, m.principal_dirs, 0.0)
        e.set_unconstrained_initialization(1)
        e.set_labels(140, lab)
        st = e.minimize()
        return e.labels(), e.clusters()["energy"], st


KEYS = ("sweeps", "moves", "relaxed_sweeps", "convergences", "candidates", "visited", "hit_loop_cap", "energy")


@pytest.mark.parametrize("metric", ["iso", "qem", "aniso"])
@pytest.mark.parametrize("run", [1, 3])
@pytest.mark.parametrize("loops", [20000, 5])
def test_same_in_several_launches(monkeypatch, metric, run, loops):
    a, ea, sa = _solve(monkeypatch, metric, None, "0", loops)
    b, eb, sb = _solve(monkeypatch, metric, None, "1000000", loops)
    c, ec, sc = _solve(monkeypatch, metric, run, "1000000", loops)
    for lab, en, st in ((b, eb, sb), (c, ec, sc)):
        np.testing.assert_array_equal(lab, a)
        np.testing.assert_array_equal(en, ea)
        assert {k: st[k] for k in KEYS} == {k: sa[k] for k in KEYS}
    # each run of sweeps between two convergence tests is ceil(its sweeps / run) launches
    extra = sc["kernel_launches"] - sb["kernel_launches"]
    if run == 1:
        assert extra == sc["sweeps"] - sc["convergences"]
    else:
        assert 0 < extra < sc["sweeps"]
