"""The convolution kernel that streams input planes along z, against float64
convolutions of the same BF16 inputs, where it can go wrong: one and several
planes, z segments and tiles, tiles that end inside a row or past the plane,
batches, row widths of 32, 64 and 128 bytes (16, 32, 48, 64 channels in one or
two tensors), 16 and 32 outputs, both sides of the dispatch, and every output mode.

Tolerance: FP32 sums of up to 1728 products, sqrt(1728) 2^-24 = 2.5e-6 of random
rounding: 1e-5 in the 2-norm; BF16 outputs 2^-9 / sqrt(3) = 1.1e-3 more: 4e-3."""
import numpy as np
import pytest

from conftest import rel_l2
from test_unet import _bf, _conv_ref, _dense, _padded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [
    # c1, c2, n, (nb, d, h, w)
    (16, 0, 16, (2, 1, 7, 9)),       # one plane, one tile larger than the plane
    (32, 16, 16, (1, 5, 9, 130)),    # 64 and 32-byte rows, several tiles
    (48, 0, 16, (1, 2, 30, 30)),     # three stages of one tensor
    (16, 32, 16, (3, 40, 8, 11)),    # many z segments
    (64, 0, 32, (1, 4, 20, 33)),     # 128-byte rows
    (32, 0, 32, (2, 3, 37, 64)),
    (16, 0, 32, (1, 9, 5, 127)),     # one stage a plane: per-tile kernel
    (32, 32, 32, (1, 3, 12, 17)),
    (32, 0, 16, (2, 2, 126, 5)),     # narrow rows
    (32, 0, 32, (1, 2, 6, 149)),     # rows too long for 32 outputs: per-tile kernel
]


@pytest.mark.parametrize("c1,c2,n,dims", CASES)
def test_conv_streamed(lib, c1, c2, n, dims):
    from yoricktrtt_b200._lib import check
    from yoricktrtt_b200.unet import _p, _stream
    nb, d, h, w = dims
    g = torch.Generator().manual_seed(c1 + 3 * c2 + n)
    x1 = _bf(torch.randn(nb, c1, d, h, w, generator=g))
    x2 = _bf(torch.randn(nb, c2, d, h, w, generator=g)) if c2 else None
    cin = c1 + c2
    wt = torch.randn(n, 27, cin, generator=g) / np.sqrt(27 * cin)
    bias = torch.randn(n, generator=g)
    pack = torch.empty(27 * n * cin, dtype=torch.bfloat16, device="cuda")
    check(lib.trtt_b200_conv3_pack(_p(wt.cuda()), n, cin, 0, _p(pack), _stream()), "pack")
    xp1, xp2, bd = _padded(x1), (_padded(x2) if c2 else None), bias.cuda()
    rows = xp1.shape[0]
    ref = _conv_ref(torch.cat([x1, x2], 1) if c2 else x1, _bf(wt), bias.double())
    raw = ref - bias.double().view(1, -1, 1, 1, 1)

    def conv(mode, slope, y, y2=None, n1=0, acc=0, resid=None):
        check(lib.trtt_b200_conv3_forward(_p(xp1), c1, _p(xp2), c2, _p(pack), n, _p(bd), mode, slope, _p(y), _p(y2),
                                          n1, acc, _p(resid), nb, d, h, w, _stream()), "conv")
        check(lib.trtt_b200_unet_status(_stream()), "status")

    y = torch.zeros(rows, n, dtype=torch.float32, device="cuda")
    conv(1, 1.0, y)
    full = y.reshape(nb, d + 2, h + 2, w + 2, n).double().cpu()
    got = full[:, 1:-1, 1:-1, 1:-1].permute(0, 4, 1, 2, 3)
    assert rel_l2(got.numpy(), ref.numpy()) <= 1e-5
    full[:, 1:-1, 1:-1, 1:-1] = 0.0
    assert float(full.abs().max()) == 0.0  # the border stays untouched
    yb = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    conv(0, 0.1, yb)
    assert rel_l2(_dense(yb, nb, d, h, w).numpy(), torch.nn.functional.leaky_relu(ref, 0.1).numpy()) <= 4e-3
    # gradient mode: channels split over two tensors, added to what is there
    n1 = 16 * ((n // 16 + 1) // 2)
    g1 = _padded(torch.ones(nb, n1, d, h, w))
    g2 = _padded(torch.ones(nb, n - n1, d, h, w)) if n1 < n else None
    conv(3, 1.0, g1, g2, n1, 1)
    back = _dense(g1, nb, d, h, w)
    if g2 is not None:
        back = torch.cat([back, _dense(g2, nb, d, h, w)], 1)
    assert rel_l2(back.numpy(), (raw + 1.0).numpy()) <= 4e-3
    resid = torch.randn(rows, generator=g).cuda()
    out = torch.zeros(rows, dtype=torch.float32, device="cuda")
    conv(2, 1.0, out, resid=resid)
    sh = (nb, d + 2, h + 2, w + 2)
    got = (out - resid).reshape(sh)[:, 1:-1, 1:-1, 1:-1].double().cpu()
    assert rel_l2(got.numpy(), ref[:, 0].numpy()) <= 1e-5
