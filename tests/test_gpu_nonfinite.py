"""Infinite and NaN values in the 3D projections: one such voxel makes the
detector cells of its own footprint not finite and no others, one such cell the
voxels that it covers.  The sweep and gather kernels sum over neighbouring
columns and voxels with weights of 0, which must not carry such a value over.

The cells are those where the FP64 oracle's projection of the voxel's (or
cell's) indicator is not 0; those of a weight above 1e-4 of the largest must be
hit.  All others are compared with the projection of the finite rest: 2e-6 in
the 2-norm, as the kernels' own tests."""
import math

import numpy as np
import pytest

from conftest import rel_l2

from yoricktrtt_b200 import footprint, geometry as G

pytestmark = pytest.mark.gpu

CONE, PAR = G.TRTT_CONE_BEAM, G.TRTT_PARALLEL_BEAM

SCANS = [
    # mode, nx, ny, nz, nu, nv, u cell, table
    (CONE, 24, 20, 18, 40, 44, 1.0, False),
    (PAR, 21, 22, 30, 51, 40, 0.8, False),
    (PAR, 16, 16, 24, 6, 20, 40.0, False),    # nearly coincident voxels
    (CONE, 20, 21, 16, 34, 40, 1.0, True),
    (PAR, 18, 17, 19, 30, 33, 1.0, True),
    (CONE, 20, 20, 90, 600, 40, 0.25, False),  # several u tiles
]


def _scan(case, views=5, square=False):
    mode, nx, ny, nz, nu, nv, us, table = case
    theta = None if square else np.linspace(0.1, 2 * math.pi, views, endpoint=False) ** 1.01
    rsc = 4.0 * max(nx, ny, nz) + 10.0
    sc = G.circular_scan_3d(nx, ny, nz, 1.0, 3, nu, nv, us, 1.0, views, mode=mode, rsc=rsc, rsd=1.5 * rsc, theta=theta)
    return sc, footprint.make_footprint(3, 2001) if table else None


def _oracle(orc, sc, v, x, job, table):
    out = np.zeros((sc.nv, sc.nu) if job == 0 else (sc.nz, sc.ny, sc.nx))
    fn = orc.cb3d if sc.mode == CONE else orc.pb3d
    args = () if table is None else (table,)
    assert fn(out, np.ascontiguousarray(x, dtype=np.float64), sc, v, job, *args) == 0
    return out


def _check(got, finite, hit):
    """got: the result; finite: FP64 result of the finite rest; hit: largest weight of an odd value."""
    odd = ~np.isfinite(got)
    assert not odd[hit == 0.0].any()
    assert odd[hit > 1e-4 * hit.max()].all()
    assert rel_l2(got[~odd], finite[~odd]) <= 2e-6


def _odd_volume(sc, rng):
    vol = rng.random((sc.nz, sc.ny, sc.nx)).astype(np.float32)
    at = [(sc.nz // 2, sc.ny // 3, sc.nx // 2), (sc.nz // 4, sc.ny // 2, sc.nx // 4)]
    clean = vol.copy()
    for p, x in zip(at, (np.nan, np.inf)):
        vol[p] = x
        clean[p] = 0.0
    return vol, clean, at


@pytest.mark.parametrize("case", SCANS)
def test_forward(oracle_port, case):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc, table = _scan(case)
    vol, clean, at = _odd_volume(sc, np.random.default_rng(7))
    pr = Projector3D(sc, table)
    got = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    pr.status()
    for v in range(sc.nviews):
        hit = np.zeros((sc.nv, sc.nu))
        for p in at:
            one = np.zeros(vol.shape)
            one[p] = 1.0
            hit = np.maximum(hit, _oracle(oracle_port, sc, v, one, 0, table))
        _check(got[v], _oracle(oracle_port, sc, v, clean, 0, table), hit)


@pytest.mark.parametrize("mode,views", [(CONE, 4), (PAR, 2), (CONE, 6)])
def test_forward_groups(oracle_port, mode, views):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc, _ = _scan((mode, 20, 20, 26, 60, 44, 1.0, False), views, square=True)
    vol, clean, at = _odd_volume(sc, np.random.default_rng(8))
    pr = Projector3D(sc)
    assert pr.groups()[1] + pr.groups()[2] > 0
    got = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    for v in range(sc.nviews):
        hit = np.zeros((sc.nv, sc.nu))
        for p in at:
            one = np.zeros(vol.shape)
            one[p] = 1.0
            hit = np.maximum(hit, _oracle(oracle_port, sc, v, one, 0, None))
        _check(got[v], _oracle(oracle_port, sc, v, clean, 0, None), hit)


@pytest.mark.parametrize("case", SCANS)
@pytest.mark.parametrize("gates", [False, True])
def test_transpose(oracle_port, case, gates):
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc, table = _scan(case)
    rng = np.random.default_rng(9)
    y = rng.random((sc.nviews, sc.nv, sc.nu)).astype(np.float32)
    at = [(1, sc.nv // 2, sc.nu // 2), (3, sc.nv // 3, sc.nu // 4)]
    clean = y.copy()
    for p, x in zip(at, (np.nan, np.inf)):
        y[p] = x
        clean[p] = 0.0
    pr = Projector3D(sc, table)
    t = np.array([0.3, 1.6, 2.5, 0.7, 1.2])
    if gates:
        pr.set_gates(3, t)
    got = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    pr.status()
    each, hit = np.zeros(got.shape), np.zeros(got.shape)
    for v in range(sc.nviews):
        b = _oracle(oracle_port, sc, v, clean[v], 1, table)
        one = np.zeros((sc.nv, sc.nu))
        for p in at:
            if p[0] == v:
                one[p[1:]] = 1.0
        h = _oracle(oracle_port, sc, v, one, 1, table)
        if gates:
            (g0, g1), (w0, w1) = G.gate_weights(t[v], 3)
            for g, w in ((g0, w0), (g1, w1)):
                each[g] += w * b
                hit[g] = np.maximum(hit[g], h)
        else:
            each += b
            hit = np.maximum(hit, h)
    _check(got, each, hit)


@pytest.mark.parametrize("mode,views,square,table", [(CONE, 24, False, False), (PAR, 24, False, True),
                                                     (CONE, 24, True, False), (PAR, 22, True, False)])
def test_forward_of_nan_volume(oracle_port, mode, views, square, table):
    """A diverged iterate: every cell that some voxel reaches is NaN, and the call
    takes the time of a finite volume's up to a factor (16; about 5 expected: a
    second pass over the columns, with atomics), not that of a pass voxel by voxel
    (over 100)."""
    import torch
    from yoricktrtt_b200.projectors import Projector3D
    sc, tab = _scan((mode, 64, 64, 60, 120, 96, 1.0, table), views, square=square)
    pr = Projector3D(sc, tab)
    vol = torch.rand(pr.volume_shape("columns"), device="cuda")
    nan = torch.full_like(vol, float("nan"))
    out = torch.zeros(pr.detector_shape(), device="cuda")

    def ms(x):
        best = math.inf
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            out.zero_()
            a.record()
            pr.forward(x, out=out, layout="columns")
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    base = ms(vol)
    took = ms(nan)
    pr.status()
    got = out.cpu().numpy()
    for v in (0, views // 3):
        hit = _oracle(oracle_port, sc, v, np.ones((sc.nz, sc.ny, sc.nx)), 0, tab)
        odd = np.isnan(got[v])
        assert not odd[hit == 0.0].any() and odd[hit > 1e-4 * hit.max()].all()
        assert (got[v][~odd] == 0.0).all()
    assert took <= 16.0 * base, (took, base)
