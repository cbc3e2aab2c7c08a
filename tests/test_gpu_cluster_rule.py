"""Which small problems the cluster schedule takes (needs a GB300): those with at least as many
items as clusters; more clusters than items stay with the per-phase graphs, launch for launch.
"""
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu


def _launches(monkeypatch, k, limit):
    if limit is None:
        monkeypatch.delenv("ACVD_CLUSTER_MAX", raising=False)
    else:
        monkeypatch.setenv("ACVD_CLUSTER_MAX", limit)
    m = synth.heightfield(30, ny=20, seed=6, with_curvature=False)
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    with acvd_gb300.Engine() as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric("iso")
        e.set_labels(k, synth.seed_labels(m.n_points, min(k, m.n_points), seed=1) % k)
        return e.minimize()["kernel_launches"]


@pytest.mark.parametrize("k,cluster", [(60, True), (600, True), (601, False), (5000, False)])
def test_rule(monkeypatch, k, cluster):
    assert (_launches(monkeypatch, k, None) < _launches(monkeypatch, k, "0")) == cluster
