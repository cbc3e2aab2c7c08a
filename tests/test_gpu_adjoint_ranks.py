"""The adjoint's eigen-decomposition on clusters of every rank (needs a GB300): nearly flat
(one eigenvalue kept), on a ridge (two), over a corner (three), along the axes and turned,
against the FP64 torch reference; within 1e-6 of the largest component, the full-size test's
bound.  The sheets bend a little, by other radii along the two axes: the reference
differentiates an eigen-decomposition, which has no derivative where eigenvalues coincide.
"""
import numpy as np
import pytest
import torch

import acvd_gb300
from acvd_gb300 import synth
from acvd_gb300.adjoint import ClusteringEnergy, reference_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slope", [1.0, 0.3, 0.0])
@pytest.mark.parametrize("turned", [False, True])
def test_gradients_by_rank(slope, turned):
    n = 36
    m = synth.heightfield(n, ny=n, seed=1)
    p = np.array(m.points, np.float64)
    i, j = np.divmod(np.arange(n * n), n)
    u, v = i / 6.0 - 2.5, j / 6.0 - 2.5   # the ridges run through the middle of a 6 x 6 block
    p[:, 0], p[:, 1], p[:, 2] = u, v, slope * (np.maximum(u, 0.0) + np.maximum(v, 0.0))
    p[:, 2] += 0.004 * u * u + 0.002 * v * v
    if turned:
        q, _ = np.linalg.qr(np.random.default_rng(7).normal(size=(3, 3)))
        p = p @ q.T
    lab = ((i // 6) * 6 + j // 6).astype(np.int32)
    k = 36
    row, col, ev = acvd_gb300.build_topology(len(p), m.faces)
    rng = np.random.default_rng(9)
    rho = rng.uniform(0.5, 2.0, len(p))
    G = torch.tensor(rng.normal(size=(k, 3)), dtype=torch.float64)
    with acvd_gb300.Engine() as e:
        e.set_mesh(p, m.faces, row, col, ev)
        e.set_metric("qem", rho, None, 1.0)
        e.set_labels(k, lab)
        x = torch.tensor(p, dtype=torch.float64, device="cuda", requires_grad=True)
        r = torch.tensor(rho, dtype=torch.float64, device="cuda", requires_grad=True)
        E, C = ClusteringEnergy.apply(x, r, e, 1.0)
        (E + (C * G.cuda()).sum()).backward()
        gx, gr = x.grad.cpu().numpy(), r.grad.cpu().numpy()
    xr = torch.tensor(p, dtype=torch.float64, requires_grad=True)
    rr = torch.tensor(rho, dtype=torch.float64, requires_grad=True)
    Er, Cr = reference_energy(xr, m.faces, lab, k, rr, 1.0, metric="qem")
    (Er + (Cr * G).sum()).backward()
    gxr, grr = xr.grad.numpy(), rr.grad.numpy()
    assert np.isfinite(gxr).all() and np.isfinite(grr).all()
    assert abs(float(E) - float(Er)) <= 1e-9 * abs(float(Er))
    assert np.max(np.abs(C.detach().cpu().numpy() - Cr.detach().numpy())) <= 1e-6
    assert np.max(np.abs(gx - gxr)) <= 1e-6 * np.max(np.abs(gxr))
    assert np.max(np.abs(gr - grr)) <= 1e-6 * np.max(np.abs(grr))
