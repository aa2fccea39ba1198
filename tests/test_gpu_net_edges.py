"""Weight and bias gradients at the edges of the kernel's tiles: one pixel,
rows shorter than a 128-pixel tile, and more tiles than CTAs (two per SM), so
that a CTA accumulates several; without a bias gradient too."""
import pytest

import hpm_b200 as hb
from test_gpu_net import _case, _ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(16, 16), (16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("h,w,bias", [(1, 1, True), (3, 17, False), (2, 129, True), (401, 130, True)])
def test_weight_gradient_tiles(cin, cout, h, w, bias):
    import torch

    x, wt, _ = _case(h, w, cin, cout, seed=5 + h + w)
    g = torch.Generator(device="cpu").manual_seed(h * w)
    dy = torch.randn(h, w, cout, generator=g).to(torch.bfloat16).cuda()
    ref = torch.nn.grad.conv2d_weight(x.double().permute(2, 0, 1)[None], wt.shape,
                                      dy.double().permute(2, 0, 1)[None], padding=1)
    dw = torch.zeros_like(wt)
    db = torch.zeros(cout, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert hb.lib().hpm_net_conv_wgrad(_ptr(x), _ptr(dy), h, w, cin, cout, _ptr(dw), _ptr(db) if bias else None,
                                       _ptr(err), None) == hb.HPM_OK
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    # FP32 sums of h * w exact products in blocks of at most a few hundred
    # terms: 256 roundings of the sum of magnitudes bound the error
    mag = torch.nn.grad.conv2d_weight(x.double().abs().permute(2, 0, 1)[None], wt.shape,
                                      dy.double().abs().permute(2, 0, 1)[None], padding=1)
    assert ((dw.double() - ref).abs() <= 256 * 2.0**-24 * mag).all()
    want = dy.double().sum((0, 1)) if bias else torch.zeros(cout, dtype=torch.float64, device="cuda")
    assert ((db.double() - want).abs() <= 256 * 2.0**-24 * dy.double().abs().sum((0, 1))).all()
