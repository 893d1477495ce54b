"""The 2D group kernels (views related by turns of the pixel grid, one FP64
footprint per group) against the FP64 oracle, at the sizes where their
decomposition can go wrong: tiles, line ranges and lane strides of the direct
kernel, pixel blocks of the transpose, every group class, one view, clusters
of CTAs, and scans that keep the per-view kernels.

Tolerances.  Transpose: FP64 sums rounded once to FP32, 2^-24 = 6e-8 relative
per value, so 2e-7 in the 2-norm.  Direct: each cell sums some hundred FP32
terms in chains of at most a few hundred additions; random rounding gives
sqrt(400) 2^-24 = 1.2e-6 at most, and a cell sum of positive terms stays below
2e-6."""
import math

import numpy as np
import pytest

from conftest import rel_l2

from oracle.oracle import LF2DParams
from yoricktrtt_b200 import footprint as F, geometry as G

pytestmark = pytest.mark.gpu

TABLE = F.make_footprint(3, 10001)
FAN, PAR = G.TRTT_FAN_BEAM, G.TRTT_PARALLEL_BEAM

SCANS = [
    # mode, nx, ny, nv, views, pixel, cell, angles
    (FAN, 64, 64, 130, 12, 1.0, 1.0, "full"),      # quads
    (FAN, 64, 64, 130, 6, 1.0, 1.0, "full"),       # half-turn pairs
    (FAN, 50, 37, 101, 6, 1.0, 0.9, "full"),       # half-turn pairs, rectangular, odd rows
    (FAN, 37, 50, 700, 6, 1.0, 0.2, "full"),       # several tiles, wide footprints
    (FAN, 33, 33, 64, 5, 1.0, 1.7, "full"),        # odd square: single views, cells wider than pixels
    (PAR, 64, 64, 96, 10, 1.0, 1.0, "half"),       # quarter-turn pairs
    (PAR, 40, 40, 20, 8, 1.0, 1.0, "full"),        # quads, clipped detector
    (PAR, 61, 44, 300, 3, 0.6, 0.25, "random"),    # single views
    (FAN, 17, 200, 333, 1, 1.0, 1.0, "random"),    # one view
    (FAN, 1, 1, 9, 4, 1.0, 1.0, "full"),           # one pixel
    (FAN, 256, 256, 515, 16, 1.0, 1.0, "full"),    # quads, three tiles, several CTAs per tile
]


def _scan(case):
    mode, nx, ny, nv, views, s, d, orbit = case
    arc = math.pi if orbit == "half" else 2 * math.pi
    theta = np.arange(views) * (arc / views)
    if orbit == "random":
        theta = np.sort(np.random.default_rng(views).uniform(0, 2 * math.pi, views))
    rsc = 3.0 * max(nx, ny) * s + 10.0
    return G.circular_scan_2d(nx, ny, s, 3, nv, d, views, mode=mode, rsc=rsc, rsd=1.5 * rsc, theta=theta)


@pytest.mark.parametrize("case", SCANS)
@pytest.mark.parametrize("model", ["cubic", "table"])
def test_orbit_pair(oracle_port, case, model):
    import torch
    from yoricktrtt_b200.recon import Projector2D
    sc = _scan(case)
    table = TABLE if model == "table" else None
    name = "FB2D" if sc.mode == FAN else "PB2D"
    rng = np.random.default_rng(7)
    img = rng.random((sc.ny, sc.nx)).astype(np.float32)
    img[rng.random(img.shape) < 0.3] = 0.0
    y = rng.standard_normal((sc.nviews, sc.nv)).astype(np.float32)
    pr = Projector2D(sc, table)
    f = pr.forward(torch.tensor(img, device="cuda")).double().cpu().numpy()
    b = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    pr.status()
    ref_f, ref_b = np.zeros((sc.nviews, sc.nv)), np.zeros((sc.ny, sc.nx))
    img64, y64 = np.ascontiguousarray(img, dtype=np.float64), np.ascontiguousarray(y, dtype=np.float64)
    for v in range(sc.nviews):
        row = np.zeros(sc.nv)
        assert oracle_port.p2d(name, row, img64, sc, v, 0, table) == 0
        ref_f[v] = row
        assert oracle_port.p2d(name, ref_b, np.ascontiguousarray(y64[v]), sc, v, 1, table) == 0
    assert rel_l2(f, ref_f) <= 2e-6
    assert rel_l2(b, ref_b) <= 2e-7
    # accumulation into a given output
    pre = torch.full((sc.nviews, sc.nv), 0.5, device="cuda")
    pr.forward(torch.tensor(img, device="cuda"), out=pre)
    assert rel_l2(pre.double().cpu().numpy() - 0.5, f) <= 1e-5


LF = [
    # n1, n2, nd, views, voxel, pixel size, pixel step, angles
    (64, 64, 130, 8, 1.0, 1.0, 1.0, "full"),
    (64, 64, 130, 6, 1.0, 1.0, 1.0, "full"),
    (45, 38, 401, 3, 0.7, 0.3, 0.3, "random"),
    (32, 32, 90, 8, 1.0, 0.8, 1.0, "full"),     # cells narrower than their pitch
    (33, 20, 50, 1, 1.0, 1.0, 1.0, "random"),
]


@pytest.mark.parametrize("case", LF)
@pytest.mark.parametrize("line", [False, True])
def test_orbit_long_fessler(oracle_port, case, line):
    import torch
    from yoricktrtt_b200.recon import Projector2D
    n1, n2, nd, views, vox, size, step, orbit = case
    beta = np.arange(views) * (2 * math.pi / views) + 0.013
    if orbit == "random":
        beta = np.random.default_rng(views).uniform(0, 2 * math.pi, views)
    par = LF2DParams(pixelSize=size, pixelStep=step, voxelSize=vox, sourceDistance=300.0,
                     detectorDistance=150.0, objectOffset1=0.0, objectOffset2=0.0, objectDimension1=n1,
                     objectDimension2=n2, detectorDimension=nd)
    pr = Projector2D(lf_params=par, beta=beta, offset=np.zeros(views), line_integ=line)
    rng = np.random.default_rng(8)
    img = rng.random((n2, n1)).astype(np.float32)
    y = rng.standard_normal((views, nd)).astype(np.float32)
    f = pr.forward(torch.tensor(img, device="cuda")).double().cpu().numpy()
    b = pr.backward(torch.tensor(y, device="cuda")).double().cpu().numpy()
    pr.status()
    d, a = ("line_integ_direct", "line_integ_adjoint") if line else ("direct", "adjoint")
    ref_b = np.zeros((n2, n1))
    for v in range(views):
        row = np.zeros(nd)
        oracle_port.lf2d(d, par, beta[v], 0.0, np.ascontiguousarray(img, dtype=np.float64), row, 1)
        assert rel_l2(f[v], row) <= 2e-6
        oracle_port.lf2d(a, par, beta[v], 0.0, np.ascontiguousarray(y[v], dtype=np.float64), ref_b, 0)
    assert rel_l2(b, ref_b) <= 2e-7


def _inside(rsc):
    return G.circular_scan_2d(32, 32, 1.0, 3, 64, 1.0, 2, mode=FAN, rsc=rsc, rsd=60.0,
                              theta=np.array([math.pi, 0.3]))


def test_source_inside_the_grid(oracle_port):
    """A source inside the grid (the depth changes sign, on no pixel) keeps
    the per-view kernels; the scan's result is the oracle's."""
    import torch
    from yoricktrtt_b200.recon import Projector2D
    sc = _inside(10.0)
    img = np.random.default_rng(2).random((32, 32)).astype(np.float32)
    pr = Projector2D(sc)
    f = pr.forward(torch.tensor(img, device="cuda")).double().cpu().numpy()
    pr.status()
    for v in range(2):
        row = np.zeros(sc.nv)
        assert oracle_port.p2d("FB2D", row, img.astype(np.float64), sc, v, 0, None) == 0
        assert rel_l2(f[v], row) <= 1e-5


def test_pixel_on_the_source_line_is_reported():
    import torch
    from yoricktrtt_b200 import _lib
    from yoricktrtt_b200.recon import Projector2D
    pr = Projector2D(_inside(5.5))
    pr.forward(torch.ones(32, 32, device="cuda"))
    with pytest.raises(_lib.TrttError):
        pr.status()
