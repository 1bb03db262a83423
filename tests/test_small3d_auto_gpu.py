"""Small 3-D grids left to the library, on both sides of the line between one
cluster and the streaming sweeps: bit for bit the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu

GRIDS = [((9, 9, 12), 4), ((3, 3, 4), 1), ((40, 40, 40), 2), ((41, 43, 44), 1), ((48, 48, 48), 1), ((48, 48, 48), 4),
         ((49, 50, 52), 3), ((9, 100, 100), 4), ((20, 20, 128), 3), ((20, 20, 132), 3), ((128, 32, 32), 2), ((32, 32, 128), 1)]


@pytest.mark.parametrize("shape,radius", GRIDS, ids=lambda v: str(v).replace(", ", "x"))
@pytest.mark.parametrize("mode", [O.LEGACY, O.JACOBI], ids=["legacy", "jacobi"])
@pytest.mark.parametrize("iters", [8, 13])
def test_small_grids_match_oracle(cuda, shape, radius, mode, iters):
    import torch
    from thesis_gb300 import stencil as S
    u = O.uniform(shape, seed=radius) - 0.5
    a, b = torch.from_numpy(u).cuda(), torch.from_numpy(u).cuda()
    res = S.sweep(a, b, radius, iters, mode)
    want, other = oracle_pair(u, u, radius, iters, mode)
    assert bits_equal(res.cpu().numpy(), want)
    assert bits_equal((b if res is a else a).cpu().numpy(), other)
    assert S.device_status() == 0
