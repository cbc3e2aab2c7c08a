"""The commit kernels over proposal lists of every length class (needs a GB300).

A relaxed step gives one proposal to a lane of warp j % W, or, above 32 W proposals
(77,824 on a 152-SM GB300), runs of 32 proposals to a warp; a class below 128 items has
one block.  How the list is split cannot change a clustering: the moves of a relaxed
step are summed exactly, those of an exact step touch disjoint clusters.  So after four
sweeps the labels are those that one thread per proposal gave (the hashes below), for
every metric; and the isotropic energy tracked through the moves, which has no float32
part, equals a recompute in FP64 up to the records' 2^-47 per update.
"""
import hashlib
import json

import numpy as np
import pytest

import acvd_gb300
from acvd_gb300 import synth

pytestmark = pytest.mark.gpu

# 20^2: classes of 4 to 100 items; 129 x 61: a few blocks; 1600^2: classes of 600,000, the
# first sweeps propose far more than 77,824 moves each
SIZES = [(20, 20, 24), (129, 61, 600), (1600, 1600, 100000)]
# the quadric metric takes the isotropic decisions in its unconstrained first phase
LABELS = {
    ("iso", 20): "1d02cd7e2357e251",
    ("iso", 129): "786dda918557da67",
    ("iso", 1600): "99654b0e6d5976d9",
    ("qem", 20): "1d02cd7e2357e251",
    ("qem", 129): "786dda918557da67",
    ("qem", 1600): "99654b0e6d5976d9",
    ("aniso", 20): "cc0df079c9852e7e",
    ("aniso", 129): "f8357c8bba2b0b99",
    ("aniso", 1600): "72afb17e61530af5",
}


def _labels(metric, nu, nv, k):
    m = synth.heightfield(nu, ny=nv, seed=5, with_curvature=metric == "aniso")
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    w = acvd_gb300.vertex_weights(metric, m.points, m.faces)
    lab = acvd_gb300.initial_sampling(row, col, w, k)
    with acvd_gb300.Engine(max_loops=4) as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric(metric, None, m.principal_dirs, 0.0)
        e.set_unconstrained_initialization(1)
        e.set_labels(k, lab)
        e.minimize()
        return e.labels()


@pytest.mark.parametrize("metric", ["iso", "qem", "aniso"])
@pytest.mark.parametrize("nu,nv,k", SIZES)
def test_labels_after_four_sweeps(metric, nu, nv, k):
    lab = _labels(metric, nu, nv, k)
    assert np.all(lab < k)
    assert hashlib.sha256(lab.tobytes()).hexdigest()[:16] == LABELS[metric, nu]


@pytest.mark.parametrize("nu,nv,k", SIZES)
def test_tracked_energy_equals_recompute(nu, nv, k, tmp_path, monkeypatch):
    log = tmp_path / "sweeps.jsonl"
    monkeypatch.setenv("ACVD_SWEEP_LOG", str(log))
    _labels("iso", nu, nv, k)
    lines = [json.loads(x) for x in log.read_text().splitlines()]
    sweeps = [x for x in lines if "sweep" in x and "mode" in x]
    assert sweeps[0]["mode"] == "relaxed" and sweeps[0]["moves"] > 0
    if nu == 1600:
        assert max(x["candidates"] for x in sweeps) > 7 * 77824   # some class had more than 77,824
    events = [x for x in lines if x.get("event") == "convergence"]
    assert events and events[0]["rel_err"] < 1e-11, events
