"""The direct projection by line sweeps (closed-form model, one view at a
time and view groups) against the FP64 oracle, where its decomposition can go
wrong: every tile width, footprints of many rows, several u tiles and row
bands, clusters of CTAs, pairs of voxels closer than two cells
(every q-th pair), columns beside the detector, one-voxel columns, both line
axes and sweep directions, gates, and scans that keep the band kernels.

Tolerance: FP32 positions' fractions and weights (a few 2^-24 each) and sums
of some hundred FP32 terms in chains of tens: 2e-6 relative in the 2-norm
(sqrt(400) 2^-24 = 1.2e-6 of random rounding)."""
import math

import numpy as np
import pytest

from conftest import rel_l2

from yoricktrtt_b200 import geometry as G

pytestmark = pytest.mark.gpu

CONE, PAR = G.TRTT_CONE_BEAM, G.TRTT_PARALLEL_BEAM
TOL = 2e-6

SCANS = [
    # mode, nx, ny, nz, nu, nv, voxel, u cell, v cell, offsets (u, v)
    (CONE, 24, 20, 18, 40, 44, 1.0, 1.0, 1.0, (0.0, 0.0)),     # one tile, 8 rows
    (CONE, 20, 24, 40, 300, 60, 1.0, 0.35, 1.0, (0.0, 0.0)),   # two u tiles, fine u cells
    (CONE, 21, 19, 16, 40, 150, 1.0, 1.0, 0.45, (3.3, -2.1)),  # footprints of 12 rows
    (CONE, 18, 18, 33, 60, 260, 1.0, 1.0, 0.30, (0.0, 0.0)),   # footprints of 22 rows
    (CONE, 24, 24, 31, 20, 30, 1.0, 2.6, 2.0, (0.0, 0.0)),     # pairs closer than two cells: q = 2
    (PAR, 25, 22, 37, 41, 40, 1.0, 1.0, 1.0, (0.0, 0.0)),      # pairs exactly two cells apart
    (PAR, 22, 25, 21, 16, 33, 0.7, 3.1, 0.9, (0.0, 0.0)),      # q = 5
    (PAR, 16, 16, 24, 6, 20, 1.0, 40.0, 1.0, (0.0, 0.0)),      # nearly coincident voxels: FP64 path
    (PAR, 20, 20, 70, 30, 24, 1.0, 1.0, 1.0, (-25.0, 9.0)),    # columns beside the detector
    (CONE, 40, 1, 1, 16, 64, 1.0, 1.0, 1.0, (0.0, 0.0)),       # one-voxel columns, one line
    (CONE, 9, 70, 150, 230, 200, 1.0, 1.0, 1.0, (0.0, 0.0)),   # long columns, several bands
]


def _scan(case, views):
    mode, nx, ny, nz, nu, nv, s, us, vs, (uo, vo) = case
    theta = np.linspace(0.1, 2 * math.pi, views, endpoint=False) ** 1.01
    rsc = 4.0 * max(nx, ny, nz) * s + 10.0
    return G.circular_scan_3d(nx, ny, nz, s, 3, nu, nv, us, vs, views, mode=mode, rsc=rsc, rsd=1.5 * rsc,
                              theta=theta, u_off=uo, v_off=vo)


def _oracle(oracle_port, sc, v, vol):
    ref = np.zeros((sc.nv, sc.nu))
    fn = oracle_port.cb3d if sc.mode == CONE else oracle_port.pb3d
    assert fn(ref, np.ascontiguousarray(vol, dtype=np.float64), sc, v, 0) == 0
    return ref


@pytest.mark.parametrize("case", SCANS)
@pytest.mark.parametrize("views", [1, 7, 40])
def test_sweep_forward(oracle_port, case, views):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc = _scan(case, views)
    rng = np.random.default_rng(views)
    vol = rng.random((sc.nz, sc.ny, sc.nx)).astype(np.float32)
    vol[rng.random(vol.shape) < 0.4] = 0.0
    pr = Projector3D(sc)
    pr.set_symmetry(False)
    pre = torch.full(pr.detector_shape(), 0.25, device="cuda")
    got = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    acc = pr.forward(torch.tensor(vol, device="cuda"), out=pre).double().cpu().numpy()
    pr.status()
    for v in range(0, views, 6):
        assert rel_l2(got[v], _oracle(oracle_port, sc, v, vol)) <= TOL
    assert np.abs(acc - 0.25 - got).max() <= 1e-5 * max(1.0, np.abs(got).max())


GROUPED = [
    # mode, n (square), nz, nu, nv, views over 2 pi: quads, pairs, quads and pairs
    (CONE, 24, 20, 50, 60, 8),
    (CONE, 22, 33, 150, 50, 6),
    (PAR, 26, 41, 60, 44, 12),
    (PAR, 18, 17, 40, 40, 2),
    (CONE, 40, 70, 300, 90, 4),
]


@pytest.mark.parametrize("case", GROUPED)
def test_sweep_groups(oracle_port, case):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    mode, n, nz, nu, nv, views = case
    sc = G.circular_scan_3d(n, n, nz, 1.0, 3, nu, nv, 1.0, 1.0, views, mode=mode, rsc=5.0 * n, rsd=8.0 * n)
    vol = np.random.default_rng(n).random((nz, n, n)).astype(np.float32)
    pr = Projector3D(sc)
    assert pr.groups()[1] + pr.groups()[2] > 0
    got = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    pr.status()
    for v in range(views):
        assert rel_l2(got[v], _oracle(oracle_port, sc, v, vol)) <= TOL


def test_sweep_gates(oracle_port):
    """Interpolated gates, an integer gate index, and the data term."""
    import torch
    from yoricktrtt_b200.projectors import Projector3D, columns_from_xyz
    sc = _scan(SCANS[0], 5)
    t = np.array([0.0, 0.4, 1.0, 1.7, 2.9])
    rng = np.random.default_rng(3)
    vol = rng.random((3, sc.nz, sc.ny, sc.nx)).astype(np.float32)
    pr = Projector3D(sc)
    pr.set_gates(3, t)
    x = columns_from_xyz(torch.tensor(vol, device="cuda"))
    got = pr.forward(x, layout="columns")
    y = torch.tensor(rng.random(tuple(got.shape)).astype(np.float32), device="cuda")
    w = torch.tensor(rng.random(tuple(got.shape)).astype(np.float32), device="cuda")
    ref = np.zeros(tuple(got.shape))
    for v in range(5):
        (g0, g1), (w0, w1) = G.gate_weights(t[v], 3)
        ref[v] = _oracle(oracle_port, sc, v, w0 * vol[g0].astype(np.float64) + w1 * vol[g1])
        assert rel_l2(got[v].double().cpu().numpy(), ref[v]) <= TOL
    grad = torch.zeros_like(x)
    cost = float(pr.wls_grad(x, y, grad, w))
    pr.status()
    r = ref - y.double().cpu().numpy()
    assert abs(cost - 0.5 * (w.double().cpu().numpy() * r * r).sum()) <= 1e-5 * cost
    res = (w * (got - y)).contiguous()
    back = pr.backward(res, layout="columns")
    assert rel_l2(grad.double().cpu().numpy(), back.double().cpu().numpy()) <= 1e-5
