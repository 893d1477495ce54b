"""Which kernels a plan launches after a shape was asked for, refused or given
back (names from the CUDA activity record)."""
import numpy as np
import pytest

from yoricktrtt_b200 import geometry as G

pytestmark = pytest.mark.gpu


def _plan(views=5, theta=True, n=24, nz=16):
    from yoricktrtt_b200.projectors import Projector3D
    th = np.linspace(0.1, 6.0, views) ** 1.01 if theta else None
    return Projector3D(G.circular_scan_3d(n, n, nz, 1.0, 3, 40, 44, 1.0, 1.0, views, rsc=100.0, rsd=150.0, theta=th))


def _kernels(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        fn()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in p.key_averages())
    if "k_" not in names:
        pytest.skip("no CUDA activity record")
    return names


def _forward(pr):
    import torch
    vol = torch.ones(pr.volume_shape(), device="cuda")
    return _kernels(lambda: pr.forward(vol))


@pytest.mark.parametrize("tiles", [(16, 99), (16, 1), (100000, 0), (100000, 8)])
def test_refused_tiles_leave_the_default_kernel(tiles):
    from yoricktrtt_b200 import _lib
    pr = _plan()
    assert "k_fwd3d_sweep" in _forward(pr)
    assert _lib.load().trtt_b200_plan3d_set_tiles(pr._h, *tiles) == -1
    assert "k_fwd3d_sweep" in _forward(pr)


def test_refused_tiles_leave_the_shape_asked_for():
    from yoricktrtt_b200 import _lib
    pr = _plan()
    pr.set_tiles(-2, 0)
    assert "k_fwd3d_pull" in _forward(pr)
    assert _lib.load().trtt_b200_plan3d_set_tiles(pr._h, 16, 99) == -1
    assert "k_fwd3d_pull" in _forward(pr)
    pr.set_tiles(16, 8)
    assert "k_fwd3d_band" in _forward(pr)
    pr.set_tiles(0, 0)
    assert "k_fwd3d_sweep" in _forward(pr)


@pytest.mark.parametrize("ask", [lambda pr: pr.set_group_shape(16, 32, 2), lambda pr: pr.set_group_tiles(band_rows4=8)])
def test_group_shape_can_be_given_back(ask):
    pr = _plan(views=8, theta=False)
    assert pr.groups() == (0, 0, 2)
    assert "k_fwd3d_sweep" in _forward(pr)
    ask(pr)
    assert "k_fwd3d_group" in _forward(pr)
    pr.set_group_tiles(back_chunk_bytes=1 << 20)  # no shape of the direct kernel
    assert "k_fwd3d_group" in _forward(pr)
    pr.set_group_shape()
    assert "k_fwd3d_sweep" in _forward(pr)


def test_refused_group_tiles_leave_the_default_kernel():
    from yoricktrtt_b200 import _lib
    pr = _plan(views=8, theta=False)
    assert pr.groups() == (0, 0, 2)
    assert _lib.load().trtt_b200_plan3d_set_group_tiles(pr._h, 8, 0, 0, -1) == -1
    assert "k_fwd3d_sweep" in _forward(pr)


def test_persistent_shape_can_be_given_back():
    import torch
    pr = _plan()
    x = torch.rand(pr.volume_shape("columns"), device="cuda")
    y = torch.rand(pr.detector_shape(), device="cuda")
    grad = torch.zeros_like(x)
    names = lambda: _kernels(lambda: pr.wls_grad(x, y, grad))
    assert "k_wls_persistent" not in names()
    pr.set_persistent(16, 1)
    assert "k_wls_persistent" in names()
    pr.set_persistent(wait_seconds=1.0)
    assert "k_wls_persistent" in names()
    pr.set_persistent()
    assert "k_wls_persistent" not in names()
    times, choice = pr.autotune_wls(x, y, reps=1)
    assert (0, 0) in times and (16, 1) in times
    assert ("k_wls_persistent" in names()) == (choice != (0, 0))
