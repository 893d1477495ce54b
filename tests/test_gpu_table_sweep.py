"""Tabulated footprint in the sweep and gather kernels against the FP64 oracle,
where they can go wrong: several tiles and bands, lanes that take every q-th
voxel, nearly coincident voxels (atomics), footprints of many cells and rows,
detectors that miss columns, one-voxel columns, other spline degrees, tables
from two entries to more than shared memory takes (general kernels), gates, and
both shapes of the gather (with and without vector loads).

Tolerance: the table slots are the oracle's, weights differences of FP64 values
rounded to FP32 (2^-25); direct: FP32 sums of some hundred terms in chains of
tens, 2e-6; transpose: chains of tens, views compensated, 1e-6 (relative, in
the 2-norm)."""
import math

import numpy as np
import pytest

from conftest import rel_l2

from yoricktrtt_b200 import geometry as G
from yoricktrtt_b200.footprint import make_footprint

pytestmark = pytest.mark.gpu

CONE, PAR = G.TRTT_CONE_BEAM, G.TRTT_PARALLEL_BEAM

SCANS = [
    # mode, nx, ny, nz, nu, nv, voxel, u cell, v cell, offsets (u, v), degree, table size
    (CONE, 24, 20, 18, 40, 44, 1.0, 1.0, 1.0, (0.0, 0.0), 3, 10001),
    (CONE, 19, 22, 40, 301, 60, 1.0, 0.35, 1.0, (0.0, 0.0), 3, 5001),    # two u tiles, many cells
    (CONE, 21, 19, 16, 40, 150, 1.0, 1.0, 0.25, (3.3, -2.1), 3, 10001),  # footprints of 26 rows
    (CONE, 24, 24, 31, 20, 30, 1.0, 2.6, 2.0, (0.0, 0.0), 3, 1001),      # every third voxel
    (PAR, 25, 22, 37, 41, 40, 1.0, 1.0, 1.0, (0.0, 0.0), 3, 10001),      # voxels exactly a cell apart
    (PAR, 16, 16, 24, 6, 20, 1.0, 40.0, 1.0, (0.0, 0.0), 3, 10001),      # nearly coincident: atomics
    (PAR, 20, 20, 70, 30, 24, 1.0, 1.0, 1.0, (-25.0, 9.0), 3, 10001),    # columns beside the detector
    (CONE, 40, 1, 1, 16, 64, 1.0, 1.0, 1.0, (0.0, 0.0), 3, 10001),       # one-voxel columns
    (CONE, 14, 17, 150, 230, 90, 1.0, 1.0, 1.0, (0.0, 0.0), 3, 10001),   # long columns
    (CONE, 20, 21, 22, 44, 40, 1.0, 1.0, 1.0, (0.0, 0.0), 0, 2001),      # other degrees
    (PAR, 20, 21, 22, 44, 40, 0.9, 1.0, 1.0, (0.0, 0.0), 9, 2001),
    (CONE, 20, 21, 22, 44, 40, 1.0, 1.0, 1.0, (0.0, 0.0), 1, 2),         # two entries
    (CONE, 20, 21, 22, 44, 40, 1.0, 1.0, 1.0, (0.0, 0.0), 3, 40001),     # longer than the kernels take
]


def _scan(case, views):
    mode, nx, ny, nz, nu, nv, s, us, vs, (uo, vo), deg, size = case
    theta = np.linspace(0.1, 2 * math.pi, views, endpoint=False) ** 1.01
    rsc = 4.0 * max(nx, ny, nz) * s + 10.0
    return (G.circular_scan_3d(nx, ny, nz, s, deg, nu, nv, us, vs, views, mode=mode, rsc=rsc, rsd=1.5 * rsc,
                               theta=theta, u_off=uo, v_off=vo), make_footprint(deg, size))


def _oracle(oracle_port, sc, v, x, job, table):
    ref = np.zeros((sc.nv, sc.nu) if job == 0 else (sc.nz, sc.ny, sc.nx))
    name = "CB3D" if sc.mode == CONE else "PB3D"
    assert oracle_port._p3d(name, ref, np.ascontiguousarray(x, dtype=np.float64), sc, v, job, table) == 0
    return ref


@pytest.mark.parametrize("case", SCANS)
@pytest.mark.parametrize("views", [1, 23])
def test_table_pair(oracle_port, case, views):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc, table = _scan(case, views)
    rng = np.random.default_rng(views)
    vol = rng.random((sc.nz, sc.ny, sc.nx)).astype(np.float32)
    vol[rng.random(vol.shape) < 0.4] = 0.0
    y = rng.random((views, sc.nv, sc.nu)).astype(np.float32)
    pr = Projector3D(sc, table)
    det = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    back = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    pr.status()
    ref = np.zeros_like(back)
    for v in range(views):
        assert rel_l2(det[v], _oracle(oracle_port, sc, v, vol, 0, table)) <= 2e-6
        ref += _oracle(oracle_port, sc, v, y[v], 1, table)
    assert rel_l2(back, ref) <= 1e-6


def test_table_gates(oracle_port):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc, table = _scan(SCANS[8], 7)
    t = np.array([2.5, 0.3, 0.4, 1.2, 1.7, 2.9, 0.6])
    rng = np.random.default_rng(5)
    vol = rng.random((3, sc.nz, sc.ny, sc.nx)).astype(np.float32)
    y = rng.random((7, sc.nv, sc.nu)).astype(np.float32)
    pr = Projector3D(sc, table)
    pr.set_gates(3, t)
    det = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    back = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    pr.status()
    ref = np.zeros_like(back)
    for v in range(7):
        (g0, g1), (w0, w1) = G.gate_weights(t[v], 3)
        assert rel_l2(det[v], _oracle(oracle_port, sc, v, w0 * vol[g0].astype(np.float64) + w1 * vol[g1], 0,
                                      table)) <= 2e-6
        b = _oracle(oracle_port, sc, v, y[v], 1, table)
        ref[g0] += w0 * b
        ref[g1] += w1 * b
    assert rel_l2(back, ref) <= 1e-6
