"""The adjoint without densities (needs a GB300): rho=None is the plain area weight, whatever
the exponent, against the FP64 torch reference; within the bounds of the tests with densities.
"""
import numpy as np
import pytest
import torch

import acvd_gb300
from acvd_gb300 import synth
from acvd_gb300.adjoint import ClusteringEnergy, reference_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["iso", "qem"])
@pytest.mark.parametrize("gradation", [0.0, 1.5])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-6), (torch.float32, 1e-5)])
def test_gradients_without_rho(metric, gradation, dtype, tol):
    m = synth.heightfield(41, ny=29, seed=2, with_curvature=False)
    # values that both types hold, so that both sides start from the same positions
    pts = m.points.astype(np.float32).astype(np.float64)
    i, j = np.divmod(np.arange(m.n_points), 29)
    lab = ((i // 6) * 5 + j // 6).astype(np.int32)
    k = int(lab.max()) + 1
    row, col, ev = acvd_gb300.build_topology(m.n_points, m.faces)
    G = torch.tensor(np.random.default_rng(4).normal(size=(k, 3)), dtype=torch.float64)
    with acvd_gb300.Engine() as e:
        e.set_mesh(pts, m.faces, row, col, ev)
        e.set_metric(metric)
        e.set_labels(k, lab)
        x = torch.tensor(pts, dtype=dtype, device="cuda", requires_grad=True)
        E, C = ClusteringEnergy.apply(x, None, e, gradation)
        (E + (C * G.cuda()).sum()).backward()
        got = x.grad
        with torch.no_grad():
            E0, _ = ClusteringEnergy.apply(x, None, e, gradation)
    xr = torch.tensor(pts, dtype=torch.float64, requires_grad=True)
    Er, Cr = reference_energy(xr, m.faces, lab, k, None, gradation, metric=metric)
    (Er + (Cr * G).sum()).backward()
    gxr = xr.grad.numpy()
    assert got.dtype == dtype
    assert abs(E.item() - Er.item()) <= 1e-9 * abs(Er.item()) and E0.item() == E.item()
    assert np.max(np.abs(C.detach().cpu().numpy() - Cr.detach().numpy())) <= 1e-6
    assert np.max(np.abs(got.cpu().numpy() - gxr)) <= tol * np.max(np.abs(gxr))
