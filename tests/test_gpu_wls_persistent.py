"""The persistent form of the data term (a shape set by set_persistent) against
the FP64 oracle: with and without weights, small and odd sizes, more bands than
one per view, one and two CTAs per SM, and columns long enough that band rows are
spread under locks (nz >= 128).  Tolerances of test_gpu_wls."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_wls import TOL, _gated_scan, _oracle_wls

from yoricktrtt_b200 import phantoms as P

pytestmark = pytest.mark.gpu

SCANS = [
    # gates, views per gate, n, detector, source distance
    (3, [5, 2, 6], (24, 20, 16), 40, 60.0),
    (2, [3, 4], (17, 21, 13), 37, 60.0),
    (2, [4, 3], (16, 12, 128), 200, 150.0),
]


@pytest.mark.parametrize("scan", SCANS)
@pytest.mark.parametrize("shape", [(32, 1), (16, 2), (7, 1)])
@pytest.mark.parametrize("weighted", [False, True])
def test_persistent(oracle_port, scan, shape, weighted):
    import torch
    from yoricktrtt_b200.projectors import Projector3D, columns_from_xyz, xyz_from_columns
    nt, counts, n, nd, rsc = scan
    sc, t = _gated_scan(nt, counts, n=n, nd=nd, rsc=rsc, rsd=1.5 * rsc, seed=4)
    gates = P.breathing_gates(*n, nt, 1.0, amplitude_mm=3.0, seed=5)
    pr = Projector3D(sc)
    pr.set_gates(nt, t)
    x = columns_from_xyz(torch.tensor(gates, device="cuda"))
    g = torch.Generator(device="cuda").manual_seed(3)
    y = torch.rand(pr.detector_shape(), device="cuda", generator=g) * 2.0 * float(gates.mean()) * n[0]
    w = 0.5 + torch.rand(y.shape, device="cuda", generator=g) if weighted else None
    pr.set_persistent(*shape)
    grad = torch.full_like(x, 0.25)  # added to
    cost = float(pr.wls_grad(x, y, grad, w).item())
    pr.status()
    ref_cost, ref_grad = _oracle_wls(oracle_port, sc, t, nt, gates, y.double().cpu().numpy(),
                                     None if w is None else w.double().cpu().numpy())
    assert abs(cost - ref_cost) <= TOL * ref_cost
    assert rel_l2(xyz_from_columns(grad).double().cpu().numpy() - 0.25, ref_grad) <= TOL
