"""The cluster schedule of small meshes against the per-phase graphs (needs a GB300): the same
labels and energies bit for bit, for every metric, at class sizes below, at and above one
tile of 32 items per CTA (16 CTAs), with several rounds of claims, with anchored clusters,
frozen clusters and unassigned items to start from, and at the sweep cap; and the rule that
picks it.
"""
import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _solve(monkeypatch, limit, metric, nu, nv, k, seeds=False, anchors=False, frozen=False, loops=20000, rounds=1):
    monkeypatch.setenv("ACVD_CLUSTER_MAX", limit)
    monkeypatch.setenv("ACVD_MATCH_ROUNDS", str(rounds))
    m = synth.heightfield(nu, ny=nv, seed=6, with_curvature=metric == "aniso")
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    if seeds:
        lab = synth.seed_labels(m.n_points, k, seed=1)
    else:
        lab = acvd_gb300.initial_sampling(row, col, acvd_gb300.vertex_weights(metric, m.points, m.faces), k)
    with acvd_gb300.Engine(max_loops=loops) as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric(metric, None, m.principal_dirs, 0.0)
        e.set_unconstrained_initialization(1)
        e.set_labels(k, lab)
        if anchors:
            e.set_anchor_items(np.where(np.arange(k) % 3 == 0, np.arange(k) * (m.n_points // k), -1))
        if frozen:
            e.set_frozen_clusters(np.arange(k) % 4 == 0)
        st = e.minimize()
        return e.labels(), e.clusters()["energy"], st


@pytest.mark.parametrize("metric", ["iso", "qem", "aniso"])
@pytest.mark.parametrize("nu,nv,k", [(5, 4, 3), (45, 44, 90), (47, 46, 110), (130, 97, 700)])
def test_same_as_the_graphs(monkeypatch, metric, nu, nv, k):
    a, ea, sa = _solve(monkeypatch, "0", metric, nu, nv, k)
    b, eb, sb = _solve(monkeypatch, "1000000", metric, nu, nv, k)
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(ea, eb)
    assert (sa["sweeps"], sa["moves"], sa["relaxed_sweeps"]) == (sb["sweeps"], sb["moves"], sb["relaxed_sweeps"])


@pytest.mark.parametrize("kw", [dict(seeds=True), dict(anchors=True), dict(frozen=True), dict(loops=3), dict(rounds=2)],
                         ids=lambda d: next(iter(d)))
def test_same_with_options(monkeypatch, kw):
    a, ea, sa = _solve(monkeypatch, "0", "qem", 61, 53, 160, **kw)
    b, eb, sb = _solve(monkeypatch, "1000000", "qem", 61, 53, 160, **kw)
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(ea, eb)
    assert sa["hit_loop_cap"] == sb["hit_loop_cap"] and sa["sweeps"] == sb["sweeps"]


def test_small_meshes_take_it(monkeypatch):
    """A cluster launch stands for every sweep between two convergence events."""
    small = _solve(monkeypatch, "3072", "iso", 90, 90, 400)[2]
    graph = _solve(monkeypatch, "0", "iso", 90, 90, 400)[2]
    assert small["kernel_launches"] < graph["kernel_launches"] - 3 * small["sweeps"]
