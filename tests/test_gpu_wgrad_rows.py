"""The weight gradient with the taps of a row and a plane in one MMA, against
float64 autograd of the same BF16 tensors, where it can go wrong: 16, 32 and 64
output channels (shifts per MMA), input rows of 32, 64 and 128 bytes in one or
two tensors, ranges that do not fill a stage, one plane, batches, long rows,
and sizes the per-tap kernel keeps.  Bias gradient and chunk sums with it.

Tolerance: FP32 sums of at most 2e4 products in chunks of a few thousand,
sqrt(2e4) 2^-24 = 8e-6 of random rounding: 1e-5 in the 2-norm."""
import numpy as np
import pytest

from conftest import rel_l2
from test_unet import _bf, _conv_ref, _padded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [
    # c1, c2, cout, (nb, d, h, w)
    (16, 0, 16, (1, 1, 40, 50)),     # one plane
    (32, 16, 16, (2, 6, 14, 18)),
    (48, 0, 16, (1, 4, 10, 62)),     # three blocks of one tensor
    (32, 0, 32, (2, 6, 20, 33)),
    (64, 32, 32, (1, 5, 16, 40)),    # 384 columns: one CTA per SM
    (16, 0, 32, (1, 2, 5, 300)),     # long rows
    (64, 0, 64, (1, 10, 18, 20)),     # two shifts per MMA
    (32, 0, 64, (2, 6, 10, 26)),
    (16, 16, 48, (1, 4, 8, 20)),     # 48 outputs: per-tap kernel
    (16, 0, 16, (1, 1, 3, 4)),       # too few rows: per-tap kernel
]


@pytest.mark.parametrize("c1,c2,co,dims", CASES)
def test_wgrad_rows(lib, c1, c2, co, dims):
    from yoricktrtt_b200._lib import check
    from yoricktrtt_b200.unet import _p, _stream
    nb, d, h, w = dims
    cin = c1 + c2
    g = torch.Generator().manual_seed(c1 + 5 * c2 + co)
    x = _bf(torch.randn(nb, cin, d, h, w, generator=g))
    wt = torch.zeros(co, 27, cin, dtype=torch.float64, requires_grad=True)
    gy = _bf(torch.randn(nb, co, d, h, w, generator=g))
    (_conv_ref(x, wt) * gy).sum().backward()
    xp1, xp2, gyp = _padded(x[:, :c1]), (_padded(x[:, c1:]) if c2 else None), _padded(gy)
    need = lib.trtt_b200_conv3_wgrad_scratch(co, cin, nb, d, h, w)
    scratch = torch.full((need // 4 + 1,), float("nan"), device="cuda")
    dw = torch.full((co, 27, cin), float("nan"), device="cuda")
    db = torch.full((co,), float("nan"), device="cuda")
    check(lib.trtt_b200_conv3_wgrad(_p(gyp), co, _p(xp1), c1, _p(xp2), c2, _p(dw), _p(db), _p(scratch),
                                    scratch.numel() * 4, nb, d, h, w, _stream()), "wgrad")
    check(lib.trtt_b200_unet_status(_stream()), "status")
    assert rel_l2(dw.double().cpu().numpy(), wt.grad.numpy()) <= 1e-5
    assert rel_l2(db.double().cpu().numpy(), gy.sum((0, 2, 3, 4)).numpy()) <= 1e-5
