"""The label hashes of the commit and connectivity tests with every small-mesh schedule (needs a
GB300): meshes below 3,072 items a colour class run in one thread-block cluster by default,
so those tests alone no longer reach the per-phase kernels at these sizes.  Here each is
solved with the graphs, with the cluster, from the host loop and by the persistent kernel.
The anisotropic labels on mixed degrees are those of the CSR walk, as the others are.
"""
import hashlib

import numpy as np
import pytest

import acvd_gb300
import test_gpu_commit
import test_gpu_ring_connectivity as ring

pytestmark = pytest.mark.gpu

ANISO = {(24, 33): "c96407ce06bf3a21", (70, 257): "00ffb06beb412c33", (70, 500): "b0d6e0e370da640d"}
SCHEDULES = {"graphs": {"ACVD_CLUSTER_MAX": "0"}, "cluster": {"ACVD_CLUSTER_MAX": "1000000"},
             "host_loop": {"ACVD_HOST_LOOP": "1"}, "threads256": {"ACVD_CLUSTER_MAX": "0", "ACVD_EVAL_THREADS": "256"},
             "persistent": {}}


@pytest.fixture(params=sorted(SCHEDULES))
def schedule(request, monkeypatch):
    for k, v in SCHEDULES[request.param].items():
        monkeypatch.setenv(k, v)
    if request.param == "persistent":
        init = acvd_gb300.Engine.__init__
        monkeypatch.setattr(acvd_gb300.Engine, "__init__", lambda self, **kw: init(self, persistent=True, **kw))


def _hash(lab):
    return hashlib.sha256(lab.tobytes()).hexdigest()[:16]


@pytest.mark.parametrize("metric", ["iso", "qem", "aniso"])
@pytest.mark.parametrize("nu,nv,k", [s for s in test_gpu_commit.SIZES if s[0] < 1600])
def test_commits(schedule, metric, nu, nv, k):
    assert _hash(test_gpu_commit._labels(metric, nu, nv, k)) == test_gpu_commit.LABELS[metric, nu]


@pytest.mark.parametrize("metric", ["iso", "qem", "aniso"])
@pytest.mark.parametrize("n,share,k", ring.MESHES)
def test_mixed_degrees(schedule, metric, n, share, k):
    if metric != "aniso":
        assert _hash(ring._labels(metric, n, share, k)) == ring.LABELS[metric, n, k]
        return
    pts, tri = ring._mesh(n, share)
    row, col, ev = acvd_gb300.build_topology(len(pts), tri)
    lab = acvd_gb300.initial_sampling(row, col, acvd_gb300.vertex_weights("aniso", pts, tri), k)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, tri, row, col, ev)
        e.set_metric("aniso", None, e.compute_curvature()[1], 0.0)
        e.set_labels(k, lab)
        e.minimize()
        assert _hash(e.labels()) == ANISO[n, k]
