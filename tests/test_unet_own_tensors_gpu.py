"""Networks whose tensors a caller has put elsewhere than the library's flat ones:
steps, gradients and conversions act on those."""
import copy
import pickle

import pytest

pytestmark = pytest.mark.gpu


def step(net, f, y):
    net.zero_grad()
    bufs = net.loss_and_grad(f, y)
    net.backward(bufs)
    net.adam_step(lr=1e-2)


def moved(net, how):
    import torch
    if how == "data":  # other storage behind the same tensors
        for P in [*net.params.values(), net.head]:
            for k in ("w", "b", "dw", "db"):
                P[k].data = P[k].clone()
    elif how == "one":
        net.params["e1a"]["w"].data = net.params["e1a"]["w"].clone()
    elif how == "dict":
        net.params["d0b"]["b"] = net.params["d0b"]["b"].clone()
        net.head["mw"] = net.head["mw"].clone()
    elif how == "pickled":
        net = pickle.loads(pickle.dumps(net))
    elif how == "copied":
        net = copy.deepcopy(net)
    torch.cuda.synchronize()
    return net


@pytest.mark.parametrize("how", ["data", "one", "dict", "pickled", "copied"])
def test_a_step_updates_the_tensors_in_use(cuda, how):
    import torch
    from thesis_gb300 import stencil, unet
    f = torch.stack([stencil.init_laplace2d((16, 16), k) for k in range(4)])
    y = unet.coons_fill(f) + 0.1
    plain, net = unet.UNet(seed=3), moved(unet.UNet(seed=3), how)
    for _ in range(3):
        step(plain, f, y), step(net, f, y)
    want, got = plain.state_dict(), net.state_dict()
    start = unet.UNet(seed=3).state_dict()
    for k in want:
        # the same steps but for the order of the gradients' atomic sums
        size = abs(want[k] - start[k]).max()
        assert size > 0 and abs(got[k] - want[k]).max() <= 0.05 * size, k
    net.load_state_dict(start)
    assert all((net.params[n]["wb"] == net.params[n]["w"].bfloat16()).all() for n in net.params)
