"""The weight gradient that marches down image rows (the default engine), at
the edges of its row segments, rings and channel blocks, against torch float64
on the same BF16 inputs."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# n, cin, cout, h, w, dilation, extra channels of the views: rows shorter than
# 16 pixels, not a multiple of 16, longer than one segment; one row; dilations
# up to and beyond what the row ring holds; partial output-channel blocks;
# views inside wider tensors
SHAPES = [(1, 32, 32, 1, 1, 1, 0), (2, 32, 32, 5, 8, 1, 0), (3, 64, 96, 7, 24, 1, 32), (1, 32, 160, 9, 16, 2, 0),
          (2, 96, 32, 16, 112, 1, 64), (1, 32, 64, 6, 200, 1, 0), (1, 32, 128, 12, 128, 4, 0),
          (1, 64, 32, 40, 16, 8, 0), (1, 32, 32, 70, 20, 31, 0), (2, 256, 256, 8, 16, 4, 0), (1, 32, 32, 33, 257, 1, 8)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_weight_and_bias_gradient_match_float64(cuda, shape):
    import torch
    from thesis_gb300 import unet as U
    n, cin, cout, h, w, dil, extra = shape
    g = torch.Generator().manual_seed(cin + 5 * cout + w)
    x = torch.randn(n, h, w, cin + extra, generator=g).to(torch.bfloat16)
    dy = torch.randn(n, h, w, cout + extra, generator=g).to(torch.bfloat16)
    xd, dyd = x.cuda(), dy.cuda()
    dw = torch.full((cout, 9, cin), 0.5, device="cuda")  # accumulates on what is there
    db = torch.full((cout,), 0.5, device="cuda")
    U._chk(U._L().unet_conv3x3_wgrad_engine(ctypes.byref(U.view(xd, extra, cin)), ctypes.byref(U.view(dyd, extra, cout)),
                                            U._p(dw), U._p(db), dil, 0, None, 0, None), "wgrad")
    torch.cuda.synchronize()
    X = x[..., extra:].double().permute(0, 3, 1, 2)
    W = torch.zeros(cout, cin, 3, 3, dtype=torch.float64, requires_grad=True)
    torch.nn.functional.conv2d(X, W, None, padding=dil, dilation=dil).backward(
        dy[..., extra:].double().permute(0, 3, 1, 2))
    ref = W.grad.permute(0, 2, 3, 1).reshape(cout, 9, cin)
    refb = dy[..., extra:].double().sum((0, 1, 2))
    # FP32 sums of at most 8481 exact products: worst case 8481 * 2^-24 of the
    # sum of magnitudes, typically its square root
    assert (dw.cpu().double() - 0.5 - ref).abs().max().item() / ref.abs().max().item() < 1e-4
    assert (db.cpu().double() - 0.5 - refb).abs().max().item() / refb.abs().max().item() < 1e-4
