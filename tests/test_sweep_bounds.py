"""Bounds of the sweep and gather kernels (CPU, host arithmetic): where they
apply every footprint of every voxel must lie inside them, and a scan whose
projection has a pole inside the volume (a tilted detector: the depth of the
detector frame changes sign over the grid, the distance from the source does
not) must be refused, since the grid's corners bound nothing there."""
import ctypes as C

import numpy as np
import pytest

from yoricktrtt_b200 import _lib, geometry as G

CONE, PAR = G.TRTT_CONE_BEAM, G.TRTT_PARALLEL_BEAM


def _info(sc, xsd=None):
    xos = np.ascontiguousarray(sc.xos, dtype=np.float64)
    xsd = np.ascontiguousarray(sc.xsd if xsd is None else xsd, dtype=np.float64)
    info = np.zeros(5, dtype=np.int64)
    _lib.check(_lib.load().trtt_b200_sweep_bounds_info(
        4 if sc.mode == CONE else 3, sc.nx, sc.ny, sc.nz, sc.s_scl, sc.s_deg, sc.nu, sc.nv, sc.u_scl, sc.v_scl,
        sc.nviews, _lib.dptr(xos), _lib.dptr(xsd), info.ctypes.data_as(C.POINTER(C.c_long))), "sweep_bounds_info")
    return info


def _scan(mode, tilt=0.0, **kw):
    sc = G.circular_scan_3d(12, 10, 9, 1.0, 3, 23, 19, 1.0, 0.8, 7, mode=mode, rsc=40.0, rsd=60.0, **kw)
    xsd = np.array(sc.xsd, dtype=np.float64).reshape(sc.nviews, 12).copy()
    xsd[:, 1] = tilt
    return sc, xsd


def _footprints(sc, xsd):
    """Lowest and highest cell position of every voxel's footprint, (u, v), and the largest half support along v."""
    k, j, i = np.meshgrid(np.arange(sc.nz), np.arange(sc.ny), np.arange(sc.nx), indexing="ij")
    hs0 = 0.5 * (sc.s_deg + 1)
    lo, hi, hv = np.full(2, np.inf), np.full(2, -np.inf), 0.0
    for o, s in zip(np.asarray(sc.xos).reshape(-1, 3, 4), xsd.reshape(-1, 3, 4)):
        w, y, z = (o[r, 0] * i + o[r, 1] * j + o[r, 2] * k + o[r, 3] for r in range(3))
        if sc.mode == CONE:
            q = -s[0, 3] / (s[0, 0] * w + s[0, 1] * y + s[0, 2] * z)
            w2, y2, z2 = q * w, q * y, q * z
            magn = -s[0, 3] / w
        else:
            t = -(s[0, 1] * y + s[0, 2] * z + s[0, 3]) / s[0, 0]
            w2, y2, z2, magn = t, y, z, np.ones_like(w)
        v = s[1, 0] * w2 + s[1, 1] * y2 + s[1, 2] * z2 + s[1, 3]
        u = s[2, 0] * w2 + s[2, 1] * y2 + s[2, 2] * z2 + s[2, 3]
        dv = np.sqrt(1 + ((v - s[1, 3]) * sc.v_scl / s[0, 3]) ** 2) if sc.mode == CONE else 1.0
        du = np.sqrt(1 + ((u - s[2, 3]) * sc.u_scl / s[0, 3]) ** 2) if sc.mode == CONE else 1.0
        hsv, hsu = hs0 * sc.s_scl / sc.v_scl * magn * dv, hs0 * sc.s_scl / sc.u_scl * magn * du
        hv = max(hv, float(hsv.max()))
        for a, (p, h) in enumerate(((u, hsu), (v, hsv))):
            lo[a] = min(lo[a], float((p - h).min()))
            hi[a] = max(hi[a], float((p + h).max()))
    return lo, hi, hv


@pytest.mark.parametrize("mode", [CONE, PAR])
@pytest.mark.parametrize("tilt,kw", [(0.0, {}), (0.0, dict(u_off=9.3, v_off=-7.1)), (0.3, {})])
def test_bounds_hold_every_footprint(mode, tilt, kw):
    sc, xsd = _scan(mode, tilt, **kw)
    rows, u0, u1, v0, v1 = _info(sc, xsd)
    lo, hi, hv = _footprints(sc, xsd)
    assert rows >= np.floor(2 * hv) + 1
    assert u0 <= max(0, np.floor(lo[0])) and u1 >= min(sc.nu, np.floor(hi[0]) + 1)
    assert v0 <= max(0, np.floor(lo[1])) and v1 >= min(sc.nv, np.floor(hi[1]) + 1)


@pytest.mark.parametrize("tilt", [8.0, -8.0, 30.0])
def test_pole_inside_the_volume_is_refused(tilt):
    sc, xsd = _scan(CONE, tilt)
    o = np.asarray(sc.xos).reshape(-1, 3, 4)
    w = [v[0] @ np.array([i, j, 0, 1]) for v in o for i in (0, 11) for j in (0, 9)]
    d = [(v[0] + tilt * v[1]) @ np.array([i, j, 0, 1]) for v in o for i in (0, 11) for j in (0, 9)]
    assert min(w) > 0 and min(d) < 0 < max(d)
    assert _info(sc, xsd)[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tilt", [0.3, 8.0])
def test_tilted_detector_against_oracle(oracle_port, tilt):
    """Tolerance: FP32 weights and sums of some hundred terms, 2e-6 in the 2-norm."""
    import torch
    from conftest import rel_l2
    from yoricktrtt_b200.projectors import Projector3D
    sc, xsd = _scan(CONE, tilt)
    sc.xsd = xsd.reshape(np.asarray(sc.xsd).shape)
    rng = np.random.default_rng(5)
    vol = rng.random((sc.nz, sc.ny, sc.nx)).astype(np.float32)
    y = rng.random((sc.nviews, sc.nv, sc.nu)).astype(np.float32)
    pr = Projector3D(sc)
    assert pr.factorized
    got = pr.forward(torch.tensor(vol, device="cuda")).double().cpu().numpy()
    back = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    pr.status()
    ref, refb = np.zeros(got.shape), np.zeros(back.shape)
    for v in range(sc.nviews):
        assert oracle_port.cb3d(ref[v], vol.astype(np.float64), sc, v, 0) == 0
        assert oracle_port.cb3d(refb, np.ascontiguousarray(y[v], dtype=np.float64), sc, v, 1) == 0
    assert rel_l2(got, ref) <= 2e-6
    assert rel_l2(back, refb) <= 2e-6
