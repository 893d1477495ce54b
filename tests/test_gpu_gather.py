"""The transpose projection by column gathering (closed-form model, view by
view) against the FP64 oracle, where its decomposition can go wrong: every
range of k per lane (1 to 5 pairs, one and several ranges), odd detector rows
(no vector loads), lines that four columns do not fill, few columns (views
split over warps), footprints of more rows than a weight table, detectors that
miss columns, gates (integer and wrapped indices) and view sub-ranges.

Tolerance: weights of a few 2^-24 each, sums over the rows and cells of one
footprint in FP32 chains of tens (sqrt(40) 2^-24 = 4e-7 of random rounding),
views summed with compensation: 1e-6 relative in the 2-norm."""
import math

import numpy as np
import pytest

from conftest import rel_l2

from yoricktrtt_b200 import geometry as G

pytestmark = pytest.mark.gpu

CONE, PAR = G.TRTT_CONE_BEAM, G.TRTT_PARALLEL_BEAM
TOL = 1e-6

SCANS = [
    # mode, nx, ny, nz, nu, nv, voxel, u cell, v cell, offsets (u, v)
    (CONE, 24, 20, 16, 40, 44, 1.0, 1.0, 1.0, (0.0, 0.0)),     # 1 pair a lane, vector loads
    (CONE, 23, 21, 30, 43, 40, 1.0, 1.0, 1.0, (0.0, 0.0)),     # 2 pairs, odd rows, nx % 4 = 3
    (PAR, 22, 25, 47, 50, 33, 0.7, 0.7, 0.9, (0.0, 0.0)),      # 3 pairs, one voxel short
    (CONE, 17, 18, 61, 97, 60, 1.0, 1.0, 1.0, (3.3, -2.1)),    # 4 pairs
    (PAR, 18, 17, 77, 300, 40, 1.0, 0.3, 1.0, (0.0, 0.0)),     # 5 pairs, 128 cells and more
    (CONE, 9, 14, 150, 230, 60, 1.0, 1.0, 1.0, (0.0, 0.0)),    # two ranges of k
    (CONE, 12, 13, 20, 24, 300, 1.0, 1.0, 0.12, (0.0, 0.0)),   # footprints of more than 32 rows
    (CONE, 24, 24, 31, 20, 30, 1.0, 2.6, 2.0, (0.0, 0.0)),     # voxels closer than a cell
    (PAR, 20, 20, 70, 30, 24, 1.0, 1.0, 1.0, (-25.0, 9.0)),    # columns beside the detector
    (CONE, 4, 1, 1, 16, 32, 1.0, 1.0, 1.0, (0.0, 0.0)),        # one-voxel columns, one group
]


def _scan(case, views):
    mode, nx, ny, nz, nu, nv, s, us, vs, (uo, vo) = case
    theta = np.linspace(0.1, 2 * math.pi, views, endpoint=False) ** 1.01
    rsc = 4.0 * max(nx, ny, nz) * s + 10.0
    return G.circular_scan_3d(nx, ny, nz, s, 3, nu, nv, us, vs, views, mode=mode, rsc=rsc, rsd=1.5 * rsc,
                              theta=theta, u_off=uo, v_off=vo)


def _oracle(oracle_port, sc, v, det):
    ref = np.zeros((sc.nz, sc.ny, sc.nx))
    fn = oracle_port.cb3d if sc.mode == CONE else oracle_port.pb3d
    assert fn(ref, np.ascontiguousarray(det, dtype=np.float64), sc, v, 1) == 0
    return ref


@pytest.mark.parametrize("case", SCANS)
@pytest.mark.parametrize("views", [1, 5, 41])
def test_gather_transpose(oracle_port, case, views):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc = _scan(case, views)
    rng = np.random.default_rng(views)
    y = rng.random((views, sc.nv, sc.nu)).astype(np.float32)
    pr = Projector3D(sc)
    pr.set_symmetry(False)
    pre = torch.full((sc.nz, sc.ny, sc.nx), 0.25, device="cuda")
    yd = torch.tensor(y, device="cuda")
    got = pr.backward(yd).double().cpu().numpy()
    acc = pr.backward(yd, out=pre).double().cpu().numpy()
    lo = views // 3
    sub = pr.backward(yd[lo:].contiguous(), view0=lo, nview=views - lo).double().cpu().numpy()
    pr.status()
    each = [_oracle(oracle_port, sc, v, y[v]) for v in range(views)]
    assert rel_l2(got, sum(each)) <= TOL
    assert rel_l2(sub, sum(each[lo:])) <= TOL
    assert np.abs(acc - 0.25 - got).max() <= 1e-6 * max(1.0, np.abs(got).max())


@pytest.mark.parametrize("case", [SCANS[0], SCANS[2], SCANS[5]])
def test_gather_gates(oracle_port, case):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc = _scan(case, 9)
    t = np.array([2.5, 0.0, 0.4, 1.0, 1.7, 3.9, 0.6, 3.0, 1.2])
    rng = np.random.default_rng(5)
    y = rng.random((9, sc.nv, sc.nu)).astype(np.float32)
    pr = Projector3D(sc)
    pr.set_gates(4, t)
    got = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    sub = pr.backward(torch.tensor(y[2:7], device="cuda"), view0=2, nview=5).double().cpu().numpy()
    pr.status()
    each = np.zeros((9,) + got.shape)
    for v in range(9):
        (g0, g1), (w0, w1) = G.gate_weights(t[v], 4)
        b = _oracle(oracle_port, sc, v, y[v])
        if g0 != g1:
            each[v, g0] += w0 * b
        each[v, g1] += w1 * b  # a repeated index keeps its second weight
    assert rel_l2(got, each.sum(0)) <= TOL
    assert rel_l2(sub, each[2:7].sum(0)) <= TOL
