"""The weight gradient on tcgen05 at dilations whose rows do not fit shared memory
in one march, against torch float64 on the same BF16 inputs."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

# n, cin, cout, h, w, dilation: taps that miss the image, one row, several image
# rows a step, partial segments and output-channel blocks, slices within images
SHAPES = [(1, 32, 32, 1, 32, 24), (1, 32, 32, 70, 32, 24), (2, 64, 96, 60, 64, 31), (1, 32, 160, 50, 96, 40), (3, 96, 64, 48, 32, 100),
          (1, 32, 32, 200, 160, 64), (1, 128, 128, 40, 32, 25), (2, 32, 64, 33, 128, 32)]


def gradients(x, dy, dil, engine):
    import torch
    from thesis_gb300 import unet as U
    xd, dyd = x.cuda(), dy.cuda()
    dw = torch.full((dy.shape[3], 9, x.shape[3]), 0.5, device="cuda")  # accumulates on what is there
    db = torch.full((dy.shape[3],), 0.5, device="cuda")
    need = ctypes.c_size_t()
    L, X, Y = U._L(), ctypes.byref(U.view(xd)), ctypes.byref(U.view(dyd))
    U._chk(L.unet_wgrad_workspace_bytes(X, Y, ctypes.byref(need)), "bytes")
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    U._chk(L.unet_conv3x3_wgrad_engine(X, Y, U._p(dw), U._p(db), dil, engine, U._p(ws), need.value, None), "wgrad")
    torch.cuda.synchronize()
    return dw.cpu().double() - 0.5, db.cpu().double() - 0.5


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("engine", [0, 1])
def test_wide_dilations_match_float64(cuda, shape, engine):
    import torch
    n, cin, cout, h, w, dil = shape
    g = torch.Generator().manual_seed(cin + 5 * cout + w)
    x = torch.randn(n, h, w, cin, generator=g).to(torch.bfloat16)
    dy = torch.randn(n, h, w, cout, generator=g).to(torch.bfloat16)
    dw, db = gradients(x, dy, dil, engine)
    W = torch.zeros(cout, cin, 3, 3, dtype=torch.float64, requires_grad=True)
    torch.nn.functional.conv2d(x.double().permute(0, 3, 1, 2), W, None, padding=dil, dilation=dil).backward(
        dy.double().permute(0, 3, 1, 2))
    ref = W.grad.permute(0, 2, 3, 1).reshape(cout, 9, cin)
    refb = dy.double().sum((0, 1, 2))
    # FP32 sums of at most 32000 exact products: worst case 32000 * 2^-24 of the
    # sum of magnitudes, typically its square root
    assert (dw - ref).abs().max().item() / ref.abs().max().item() < 1e-4
    assert (db - refb).abs().max().item() / refb.abs().max().item() < 1e-4


def test_wide_dilations_run_on_the_chosen_engine(cuda):
    """The engines' bits agree, their times do not: mma.sync takes several times
    as long on a layer of the network's size."""
    import torch
    from thesis_gb300 import unet as U
    x, dy = (torch.randn(64, 128, 128, 32, device="cuda").bfloat16() for _ in range(2))
    dw, db = torch.zeros(32, 9, 32, device="cuda"), torch.zeros(32, device="cuda")
    need = ctypes.c_size_t()
    L, X, Y = U._L(), ctypes.byref(U.view(x)), ctypes.byref(U.view(dy))
    U._chk(L.unet_wgrad_workspace_bytes(X, Y, ctypes.byref(need)), "bytes")
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def ms(engine):
        best = 1e9
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            U._chk(L.unet_conv3x3_wgrad_engine(X, Y, U._p(dw), U._p(db), 32, engine, U._p(ws), need.value, s), "wgrad")
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    slow = ms(2)
    assert ms(1) < 0.7 * slow and ms(0) < 0.7 * slow
