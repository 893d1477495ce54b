"""Plans of the default convolution kernels (host arithmetic of
trtt_b200_conv3_plan_info, CPU): every byte that a copy writes or a tcgen05.mma
descriptor reads lies inside the stage, every accumulator inside the
tensor-memory columns, tiles and chunks cover the output, the partial sums fit
the scratch, and no accumulator of the weight gradient takes more rows than one of
the per-tap kernel."""
import numpy as np
import pytest

from test_conv_layout import NET_FWD, NET_WGRAD, SMEM_MAX, _grid, _plan

DIMS = [(1, 128, 128, 128), (2, 64, 64, 64), (1, 33, 40, 75), (1, 16, 16, 16), (2, 3, 5, 140), (1, 1, 40, 50)]


def _channels(c):
    """Channels of a block: rows of 128, 64 or 32 bytes."""
    return 64 if c % 64 == 0 else 32 if c % 32 == 0 else 16


def _taken(which, cin, cout, dims):
    from yoricktrtt_b200 import _lib
    import ctypes as C
    info = np.zeros(10, dtype=np.int64)
    ok = _lib.load().trtt_b200_conv3_plan_info(which, cin, cout, *dims, info.ctypes.data_as(C.POINTER(C.c_long))) == 0
    return info if ok else None


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("cin,cout", NET_FWD)
def test_forward_z(cin, cout, dims):
    p = _taken(4, cin, cout, dims)
    if p is None:
        assert cout > 16  # 16 outputs with at most 96 inputs always fit
        return
    S, rh, stage, nstg, w, edge, smem, cols, tiles, length = (int(x) for x in p)
    g, ic = _grid(*dims), _channels(cin)
    assert S == (3 if cout == 16 else 1) and nstg >= 2
    assert rh >= 128 * S + 2 * g["wp"]          # rows that the last sub-tile's third dy tap reads
    assert stage >= rh * 2 * ic and stage % 1024 == 0 and w % 1024 == 0 and edge % 1024 == 0
    assert w >= 27 * cin * cout * 2             # all taps
    assert edge >= (2 if S == 1 else 1) * 2 * (4 * S + 2) * 2 * cout * 4
    assert w + edge + nstg * stage <= smem <= SMEM_MAX
    assert (5 if cout == 32 else 3) * S * 3 * cout <= cols <= 512
    assert tiles * (128 * S - 2) >= dims[2] * g["wp"] and 1 <= length <= dims[1]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("cout,cin", NET_WGRAD)
def test_wgrad_rows(cout, cin, dims):
    from yoricktrtt_b200 import _lib
    p = _taken(5, cin, cout, dims)
    g = _grid(*dims)
    if p is None:
        assert g["rows"] < 4096 or g["wp"] > 75 or (2 if cout == 64 else 1) * 3 * cin > 512
        return
    kt, a, stage, nstg, smem, cols, sets, accs, chunks, steps = (int(x) for x in p)
    ic = _channels(cin)
    assert sets == (2 if cout == 64 else 1) and accs in (1, 2) and nstg >= 2 and kt in (128, 256)
    # A: blocks of cout channels along M, one dY row apart, from row 2 set on
    last = kt - 1 + 2 * (sets - 1) + 128 // cout - 1
    assert (last + 1) * 2 * cout <= (kt + 8) * 2 * cout <= a
    # B: blocks along N one X line apart, per block of channels
    block = -(-(kt + 2 * g["wp"]) * 2 * ic // 1024) * 1024
    assert a + cin // ic * block <= stage and a % 1024 == 0 and stage % 1024 == 0
    assert nstg * stage <= smem <= SMEM_MAX
    assert accs * sets * 3 * cin <= cols <= 512
    rows = g["rows"] - 2 * g["plane"]
    assert chunks * steps * kt >= rows and (chunks - 1) * steps * kt < rows
    assert chunks * cout * 27 * cin * 4 <= _lib.load().trtt_b200_conv3_wgrad_scratch(cout, cin, *dims)
    tap = _plan(3, cin, cout, *dims)
    assert -(-steps // accs) * kt <= max(int(tap[0] * tap[9]), 128)
