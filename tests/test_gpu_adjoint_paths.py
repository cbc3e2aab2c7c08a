"""The adjoint's branches against the FP64 torch reference (needs a GB300): density
exponents with and without a power, both metrics, an open mesh, clusters of one to
about forty items (more than a warp), a cluster count that leaves a ragged last block,
and weights that the clamp holds.  Gradients within 1e-6 of the largest component, the
bound the full-size test uses.
"""
import numpy as np
import pytest
import torch

import acvd_gb300
from acvd_gb300 import synth
from acvd_gb300.adjoint import ClusteringEnergy, reference_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["iso", "qem"])
@pytest.mark.parametrize("gradation", [0.5, 1.0, 2.0])
def test_gradients(metric, gradation):
    m = synth.heightfield(53, ny=37, seed=2, with_curvature=False)
    rng = np.random.default_rng(4)
    i, j = np.divmod(np.arange(m.n_points), 37)
    lab = ((i // 6) * 7 + j // 6).astype(np.int32)   # blocks of 6 x 6 ...
    k = int(lab.max()) + 1
    lone = rng.permutation(m.n_points)[:5]
    lab[lone] = k + np.arange(5)                     # ... and clusters of one item
    k += 5
    rho = rng.uniform(0.5, 2.0, m.n_points)
    rho[11] = 1e-9 ** (1.0 / gradation)              # held by the lower clamp
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    G = torch.tensor(rng.normal(size=(k, 3)), dtype=torch.float64)
    with acvd_gb300.Engine() as e:
        e.set_mesh(m.points, m.faces, row, col, ev)
        e.set_metric(metric, rho, None, gradation)
        e.set_labels(k, lab)
        x = torch.tensor(m.points, dtype=torch.float64, device="cuda", requires_grad=True)
        r = torch.tensor(rho, dtype=torch.float64, device="cuda", requires_grad=True)
        E, C = ClusteringEnergy.apply(x, r, e, gradation)
        (E + (C * G.cuda()).sum()).backward()
        gx, gr = x.grad.cpu().numpy(), r.grad.cpu().numpy()
    xr = torch.tensor(m.points, dtype=torch.float64, requires_grad=True)
    rr = torch.tensor(rho, dtype=torch.float64, requires_grad=True)
    Er, Cr = reference_energy(xr, m.faces, lab, k, rr, gradation, metric=metric)
    (Er + (Cr * G).sum()).backward()
    gxr, grr = xr.grad.numpy(), rr.grad.numpy()
    assert grr[11] == 0.0 and gr[11] == 0.0
    assert abs(float(E) - float(Er)) <= 1e-9 * abs(float(Er))
    assert np.max(np.abs(C.detach().cpu().numpy() - Cr.detach().numpy())) <= 1e-6
    assert np.max(np.abs(gx - gxr)) <= 1e-6 * np.max(np.abs(gxr))
    assert np.max(np.abs(gr - grr)) <= 1e-6 * np.max(np.abs(grr))
