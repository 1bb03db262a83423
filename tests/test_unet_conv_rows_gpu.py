"""The default 3x3 convolution (row-marching and tiled tcgen05 forms) at the
edges of its tiles, rings and channel blocks: bit for bit the mma.sync engine,
which accumulates in the same order, and near torch float64."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# n, cin, cout, h, w, dilation, extra channels of the views.  At least 304 row
# tiles and rows of more than 64 pixels march: widths around one and two
# segments, dilations, every output block, input channels up to the largest
# that fits; the others are tiled: widths and heights that leave tiles partly
# empty, channels that are multiples of 64 or not.
SHAPES = [(5, 32, 32, 70, 65, 1, 0), (4, 96, 32, 100, 128, 1, 8), (2, 32, 96, 160, 127, 1, 0), (3, 64, 64, 60, 129, 1, 32),
          (2, 32, 128, 80, 256, 1, 0), (4, 32, 64, 90, 100, 2, 0), (1, 160, 32, 310, 72, 1, 0), (1, 32, 256, 320, 80, 3, 0),
          (3, 64, 32, 13, 11, 1, 0), (2, 96, 96, 5, 64, 1, 16), (1, 192, 160, 3, 70, 4, 0), (2, 32, 32, 1, 1, 1, 0),
          (1, 128, 128, 17, 33, 2, 0), (2, 320, 64, 9, 26, 1, 0)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("relu", [0, 1])
def test_default_convolution_matches_mma_and_float64(cuda, shape, relu):
    import torch
    from thesis_gb300 import unet as U
    n, cin, cout, h, w, dil, extra = shape
    g = torch.Generator().manual_seed(cin + 7 * cout + w)
    x = torch.randn(n, h, w, cin + extra, generator=g).to(torch.bfloat16)
    wt = (torch.randn(cout, 9, cin, generator=g) * 0.1).to(torch.bfloat16)
    b = torch.randn(cout, generator=g).float()
    xd, wd, bd = x.cuda(), wt.cuda(), b.cuda()
    outs = []
    for engine in (0, 2):
        y = torch.full((n, h, w, cout + extra), 7.0, dtype=torch.bfloat16, device="cuda")
        U._chk(U._L().unet_conv3x3_fwd_engine(ctypes.byref(U.view(xd, extra, cin)), U._p(wd), U._p(bd),
                                              ctypes.byref(U.view(y, extra, cout)), relu, dil, engine, None), "conv")
        torch.cuda.synchronize()
        assert (y[..., :extra] == 7).all()  # channels outside the view stay
        outs.append(y[..., extra:].cpu())
    assert torch.equal(*outs)
    X = x[..., extra:].double().permute(0, 3, 1, 2)
    W = wt.double().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
    ref = torch.nn.functional.conv2d(X, W, b.double(), padding=dil, dilation=dil).permute(0, 2, 3, 1)
    ref = torch.relu(ref) if relu else ref
    # one rounding to BF16: half an ulp of 8 bits, and the FP32 sum's error
    assert (outs[0].double() - ref).abs().max().item() / ref.abs().max().item() < 2 ** -8
