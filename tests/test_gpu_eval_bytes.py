"""The evaluation's algorithmic bytes (needs a GB300): the count of the statistics is the sum of
the per-sweep log's, and both are what the counted items, screens and proposals read and
write; the same from the host loop, the graphs and the cluster.
"""
import json

import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu

RECORDS = {"iso": (16, 16), "qem": (40, 80)}   # bytes of an item's and of a cluster's record


def _solve(monkeypatch, metric, env):
    for k in ("ACVD_SWEEP_LOG", "ACVD_HOST_LOOP", "ACVD_CLUSTER_MAX"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    m = synth.heightfield(73, ny=58, seed=6, with_curvature=False)
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    lab = acvd_gb300.initial_sampling(row, col, acvd_gb300.vertex_weights(metric, m.points, m.faces), 210)
    with acvd_gb300.Engine() as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric(metric)
        e.set_labels(210, lab)
        return e.minimize()


@pytest.mark.parametrize("metric", ["iso", "qem"])
def test_bytes_of_the_counted_work(monkeypatch, tmp_path, metric):
    log = tmp_path / "s.jsonl"
    st = _solve(monkeypatch, metric, {"ACVD_SWEEP_LOG": str(log)})
    rows = [r for r in map(json.loads, log.read_text().splitlines()) if "event" not in r]
    assert {r["connexity"] for r in rows} == {0, 1}
    assert sum(r["eval_bytes"] for r in rows) == st["eval_bytes"]
    total = lambda key, sel=rows: sum(r[key] for r in sel)
    tied = [r for r in rows if r["connexity"]]
    item, cluster = RECORDS[metric]
    want = (st["visited"] + 40 * total("screened") + 32 * total("cached") + 4 * st["slots"] +
            (item + cluster + 4) * st["boundary_items"] + cluster * st["targets"] +
            (16 + 8) * st["candidates"] + 8 * total("screened", tied) + 8 * total("candidates", tied))
    assert st["eval_bytes"] == want
    for env in ({"ACVD_HOST_LOOP": "1"}, {"ACVD_CLUSTER_MAX": "0"}, {"ACVD_CLUSTER_MAX": "100000"}):
        assert _solve(monkeypatch, metric, env)["eval_bytes"] == want
