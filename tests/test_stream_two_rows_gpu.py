"""3-D sweeps at R = 2, 3 and 4 on the tiles with two rows per thread, 128 or 64
cells wide, and on the narrow ones beside them: bit for bit the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu

# last tiles of one row and one column, of all rows, odd heights, grids one
# tile wide, few long and many short chunks
GRIDS = [((60, 181, 128), 3, 3), ((61, 331, 132), 3, 4), ((90, 301, 64), 3, 2), ((300, 121, 68), 3, 2),
         ((200, 90, 252), 3, 3), ((31, 500, 124), 3, 5), ((61, 331, 132), 4, 4), ((90, 301, 64), 4, 3),
         ((300, 121, 68), 4, 2), ((200, 88, 252), 4, 3), ((33, 500, 124), 4, 5), ((250, 221, 192), 4, 2),
         ((90, 301, 64), 2, 3), ((130, 61, 56), 2, 4), ((130, 55, 144), 2, 3), ((200, 121, 60), 2, 2)]


@pytest.mark.parametrize("case", GRIDS, ids=lambda c: "x".join(map(str, c[0])) + "_r%d_i%d" % c[1:])
@pytest.mark.parametrize("mode", [O.LEGACY, O.JACOBI], ids=["legacy", "jacobi"])
def test_two_row_tiles_match_oracle(cuda, case, mode):
    import torch
    from thesis_gb300 import stencil as S
    shape, radius, iters = case
    u = O.uniform(shape, seed=radius) - 0.5
    u[tuple(n // 2 for n in shape)] = -0.0
    if mode == O.JACOBI:
        u[0, shape[1] // 2, shape[2] // 2], u[shape[0] // 2, 0, 9] = np.inf, 1e-38  # the slow division
    a, b = torch.from_numpy(u).cuda(), torch.from_numpy(u).cuda()
    res = S.sweep(a, b, radius, iters, mode)
    want, other = oracle_pair(u, u, radius, iters, mode)
    for got, ref in ((res, want), (b if res is a else a, other)):
        got, nan = got.cpu().numpy(), np.isnan(ref)
        assert np.array_equal(np.isnan(got), nan)
        assert bits_equal(np.where(nan, 0, got), np.where(nan, 0, ref))
    assert S.device_status() == 0


@pytest.mark.parametrize("shape,radius", [((150, 179, 59), 2), ((61, 331, 129), 3), ((90, 301, 63), 4), ((160, 200, 126), 4)])
def test_two_row_tiles_on_pitched_copies(cuda, shape, radius):
    import torch
    from thesis_gb300 import stencil as S
    u = O.uniform(shape, seed=8)
    a, b = torch.from_numpy(u).cuda(), torch.from_numpy(u).cuda()
    bt = S.Batch([(a, b, radius, 3, O.JACOBI)], engine="phased")
    bt.launch()
    torch.cuda.synchronize()
    want, _ = oracle_pair(u, u, radius, 3, O.JACOBI)
    assert bits_equal(bt.result(0).cpu().numpy(), want)
