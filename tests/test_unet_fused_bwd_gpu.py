"""The backward passes fused with a ReLU gradient (and a skip gradient): bit
for bit the separate calls; the head's sums against torch float64."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _rand(shape, seed, relu=False):
    import torch
    t = torch.randn(*shape, generator=torch.Generator().manual_seed(seed))
    return (t.relu() if relu else t).to(torch.bfloat16).cuda()


# n, channels in and out of the convolution, h, w, dilation: tiled, tiled with
# partly empty tiles, marching
@pytest.mark.parametrize("shape", [(2, 64, 32, 16, 16, 1), (1, 32, 96, 9, 21, 2), (3, 32, 32, 110, 72, 1)],
                         ids=lambda s: "x".join(map(str, s)))
def test_data_gradient_through_relu(cuda, shape):
    import torch
    from thesis_gb300 import unet as U
    n, cout, cin, h, w, dil = shape
    L, V, R = U._L(), U.view, ctypes.byref
    dy, wt = _rand((n, h, w, cout), 1), _rand((cin, 9, cout), 2)
    wide = _rand((n, h, w, cin + 32), 3, relu=True)  # the gate is a view inside a wider tensor
    got, want = torch.empty(n, h, w, cin, dtype=torch.bfloat16, device="cuda"), torch.empty(
        n, h, w, cin, dtype=torch.bfloat16, device="cuda")
    U._chk(L.unet_conv3x3_dgrad_relu(R(V(dy)), U._p(wt), R(V(wide, 32, cin)), R(V(got)), dil, None), "fused")
    U._chk(L.unet_conv3x3_fwd_dil(R(V(dy)), U._p(wt), None, R(V(want)), 0, dil, None), "dgrad")
    U._chk(L.unet_relu_bwd(R(V(want)), R(V(wide, 32, cin)), None), "relu")
    assert torch.equal(got, want)


def test_pool_and_upsample_gradients_through_relu(cuda):
    import torch
    from thesis_gb300 import unet as U
    L, V, R = U._L(), U.view, ctypes.byref
    x, y = _rand((2, 10, 14, 40), 4, relu=True), torch.empty(2, 5, 7, 40, dtype=torch.bfloat16, device="cuda")
    U._chk(L.unet_maxpool2_fwd(R(V(x)), R(V(y)), None), "pool")
    dy, skip = _rand((2, 5, 7, 40), 5), _rand((2, 10, 14, 48), 6)
    got, want = torch.empty_like(x), torch.empty_like(x)
    U._chk(L.unet_maxpool2_bwd_skip_relu(R(V(x)), R(V(y)), R(V(dy)), R(V(skip, 8, 40)), R(V(got)), None), "fused")
    U._chk(L.unet_maxpool2_bwd(R(V(x)), R(V(y)), R(V(dy)), R(V(want)), None), "pool bwd")
    U._chk(L.unet_add(R(V(want)), R(V(skip, 8, 40)), None), "add")
    U._chk(L.unet_relu_bwd(R(V(want)), R(V(x)), None), "relu")
    assert torch.equal(got, want)
    up, gate = _rand((2, 10, 14, 64), 7), _rand((2, 5, 7, 32), 8, relu=True)
    got, want = torch.empty_like(gate), torch.empty_like(gate)
    U._chk(L.unet_upsample2_bwd_relu(R(V(up, 32, 32)), R(V(gate)), R(V(got)), None), "fused")
    U._chk(L.unet_upsample2_bwd(R(V(up, 32, 32)), R(V(want)), None), "up bwd")
    U._chk(L.unet_relu_bwd(R(V(want)), R(V(gate)), None), "relu")
    assert torch.equal(got, want)


# pixels and channels around the kernel's groups: one chunk, a count that does
# not divide the block, the most it takes
@pytest.mark.parametrize("shape", [(1, 3, 5, 8), (2, 9, 17, 24), (3, 40, 64, 32), (1, 7, 11, 256)],
                         ids=lambda s: "x".join(map(str, s)))
def test_head_gradient(cuda, shape):
    import torch
    from thesis_gb300 import unet as U
    L, V, R = U._L(), U.view, ctypes.byref
    n, h, w, c = shape
    x = _rand((n, h, w, c), 9, relu=True)
    hw = torch.randn(c, generator=torch.Generator().manual_seed(10)).cuda()
    dy = torch.randn(n, h, w, generator=torch.Generator().manual_seed(11)).cuda()
    outs = []
    for name in ("unet_head_bwd", "unet_head_bwd_relu"):
        dx, dw, db = torch.empty_like(x), torch.zeros(c, device="cuda"), torch.zeros(1, device="cuda")
        U._chk(getattr(L, name)(R(V(x)), U._p(hw), U._p(dy), R(V(dx)), U._p(dw), U._p(db), None), name)
        outs.append(dx)
        ref = (x.double() * dy.double()[..., None]).sum((0, 1, 2))
        # FP32 sums of at most 7680 products
        assert (dw.double() - ref).abs().max().item() / ref.abs().max().item() < 1e-5
        assert abs(db.item() - dy.double().sum().item()) / dy.double().abs().sum().item() < 1e-6
    assert torch.equal(outs[0], (dy[..., None] * hw).to(torch.bfloat16))
    U._chk(L.unet_relu_bwd(R(V(outs[0])), R(V(x)), None), "relu")
    assert torch.equal(outs[1], outs[0])


def test_optimizer_step_on_flat_and_rebound_tensors(cuda):
    """The one-pass update equals the per-tensor one, also for a network whose
    parameter the caller has replaced by a tensor of its own."""
    import torch
    from thesis_gb300 import unet as U
    nets = [U.UNet(seed=3), U.UNet(seed=3)]
    nets[1].params["e1a"]["w"] = nets[1].params["e1a"]["w"].clone()
    for step in range(2):
        for net in nets:
            net.zero_grad()
            g = torch.Generator(device="cuda").manual_seed(step)
            for P in [net.params[n] for n, _, _ in U.LAYERS] + [net.head]:
                for k in ("dw", "db"):
                    assert not P[k].any()
                    P[k].copy_(torch.randn(P[k].shape, device="cuda", generator=g))
            net.adam_step(lr=1e-2)
    for n, cin, cout in U.LAYERS:
        for k in ("w", "b", "mw", "vw", "mb", "vb", "wb"):
            assert torch.equal(nets[0].params[n][k], nets[1].params[n][k]), (n, k)
        P = nets[0].params[n]
        assert torch.equal(P["wb"], P["w"].to(torch.bfloat16))
        U._chk(U._L().unet_flip_weights(U._p(P["wb"]), U._p(P["wt"]), cout, cin, None), "flip")
        assert torch.equal(P["wt"], P["wb"].flip(1).permute(2, 1, 0)), n
    for k in ("w", "b", "mw", "vw"):
        assert torch.equal(nets[0].head[k], nets[1].head[k]), k
