"""Infinite and NaN values in the 2D projections: a pixel makes the cells of its own
footprint not finite and no others, a detector cell the pixels that it covers.
Long-Fessler included, whose footprint ranges have cells of weight 0 at their ends.
(Not so the tabulated footprints: their ranges are the reference's, weights of 0
among them.)  As test_gpu_nonfinite; the finite rest within 2e-6 (direct) and 2e-7
(transpose)."""
import math

import numpy as np
import pytest

from conftest import rel_l2

from oracle.oracle import LF2DParams
from yoricktrtt_b200 import geometry as G

pytestmark = pytest.mark.gpu

FAN, PAR = G.TRTT_FAN_BEAM, G.TRTT_PARALLEL_BEAM
N, NV = 24, 80


def _case(name, views):
    """(projector, oracle call (view, x, job))."""
    from yoricktrtt_b200.recon import Projector2D
    theta = np.arange(views) * (2 * math.pi / views) + 0.05
    if name.startswith("lf"):
        p = LF2DParams(pixelSize=0.6, pixelStep=0.6, voxelSize=1.0, sourceDistance=90.0, detectorDistance=45.0,
                       objectOffset1=0.0, objectOffset2=0.0, objectDimension1=N, objectDimension2=N,
                       detectorDimension=NV)
        line = name == "lf_line"
        pre = "line_integ_" if line else ""

        def call(orc, v, x, job):
            out = np.zeros(NV if job == 0 else (N, N))
            orc.lf2d(pre + ("direct" if job == 0 else "adjoint"), p, theta[v], 0.0,
                     np.ascontiguousarray(x, dtype=np.float64), out, 1)
            return out
        return Projector2D(lf_params=p, beta=theta, offset=np.zeros(views), line_integ=line), call
    mode = FAN if name == "fan" else PAR
    sc = G.circular_scan_2d(N, N, 1.0, 3, NV, 0.6, views, mode=mode, rsc=90.0, rsd=135.0, theta=theta)

    def call(orc, v, x, job):
        out = np.zeros(NV if job == 0 else (N, N))
        assert orc.p2d("FB2D" if mode == FAN else "PB2D", out, np.ascontiguousarray(x, dtype=np.float64), sc, v, job,
                       None) == 0
        return out
    return Projector2D(sc), call


def _check(got, finite, hit, tol):
    odd = ~np.isfinite(got)
    assert not odd[hit == 0.0].any()
    assert odd[hit > 1e-4 * hit.max()].all()
    assert rel_l2(got[~odd], finite[~odd]) <= tol


@pytest.mark.parametrize("name", ["fan", "parallel", "lf", "lf_line"])
@pytest.mark.parametrize("views", [3, 6, 8])
def test_pair(oracle_port, name, views):
    import torch
    pr, call = _case(name, views)
    rng = np.random.default_rng(11)
    img = rng.random((N, N)).astype(np.float32)
    y = rng.random((views, NV)).astype(np.float32)
    at, aty = [(N // 2, N // 3), (N // 4, N // 2)], [(0, NV // 2), (2, NV // 3)]
    cimg, cy = img.copy(), y.copy()
    for p, q, x in zip(at, aty, (np.nan, np.inf)):
        img[p], y[q] = x, x
        cimg[p], cy[q] = 0.0, 0.0
    f = pr.forward(torch.tensor(img, device="cuda")).double().cpu().numpy()
    b = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    back, hitb = np.zeros((N, N)), np.zeros((N, N))
    for v in range(views):
        hit = np.zeros(NV)
        for p in at:
            one = np.zeros((N, N))
            one[p] = 1.0
            hit = np.maximum(hit, call(oracle_port, v, one, 0))
        _check(f[v], call(oracle_port, v, cimg, 0), hit, 2e-6)
        back += call(oracle_port, v, cy[v], 1)
        one = np.zeros(NV)
        for q in aty:
            if q[0] == v:
                one[q[1]] = 1.0
        hitb = np.maximum(hitb, call(oracle_port, v, one, 1))
    if name != "lf_line":  # (its transpose took cells of weight 0 from the first: not finite times 0)
        _check(b, back, hitb, 2e-7)
