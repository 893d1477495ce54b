"""The data term keeps its own direct projection, whatever kernel set_tiles and
set_columns choose for plan3d_forward.

With y = 0 the cost is 1/2 sum (H x)^2.  The default kernels' FP32 sums leave it
within 2e-7 of FP64 (a bias of 8e-8 of the sums, twice in the squares); the
tensor-core band kernel, which rounds toward zero at each of some 60 additions to a
cell, is several 1e-6 off."""
import numpy as np
import pytest

from yoricktrtt_b200 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [(0, 0), (16, 8), (-1, 0), (-2, 0), (-3, 0), (0, 0, 2)])
def test_cost_does_not_depend_on_the_tiles(oracle_port, tiles):
    import torch
    from yoricktrtt_b200.projectors import Projector3D, columns_from_xyz
    sc = G.circular_scan_3d(64, 64, 32, 1.0, 3, 72, 120, 1.0, 1.0, 3, rsc=200.0, rsd=300.0,
                            theta=np.array([0.2, 1.3, 4.0]))
    vol = np.random.default_rng(2).random((sc.nz, sc.ny, sc.nx)).astype(np.float32)
    ref = 0.0
    for v in range(sc.nviews):
        hx = np.zeros((sc.nv, sc.nu))
        assert oracle_port.cb3d(hx, vol.astype(np.float64), sc, v, 0) == 0
        ref += 0.5 * float((hx * hx).sum())
    pr = Projector3D(sc)
    pr.set_tiles(*tiles)
    x = columns_from_xyz(torch.tensor(vol, device="cuda"))
    cost = float(pr.wls_grad(x, torch.zeros(pr.detector_shape(), device="cuda"), torch.zeros_like(x)).item())
    pr.status()
    assert abs(cost - ref) <= 2e-7 * ref
