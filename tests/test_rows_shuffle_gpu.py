"""2-D sweeps by register-queue chunk columns whose x-neighbours come from the
lanes beside: bit for bit the oracle's, both buffers, where a warp spans the
seam of two row blocks, ends past the last item or holds border chunks."""
import numpy as np
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu

# (ny, nx), radius, sweeps: one chunk and two, 31 to 33 chunks a row, chunk
# counts prime to the warp, fewer rows than a block, more items than threads
GRIDS = [((3, 4), 1, 3), ((9, 12), 4, 2), ((5, 8), 2, 3), ((7, 8), 3, 2), ((40, 124), 1, 5), ((37, 128), 2, 4),
         ((41, 132), 3, 3), ((29, 132), 4, 3), ((1301, 1516), 1, 9), ((1117, 1804), 2, 8), ((900, 1204), 3, 8),
         ((1003, 1412), 4, 9), ((9, 70000), 4, 8), ((20000, 68), 1, 8), ((3000, 2900), 1, 3)]


@pytest.mark.parametrize("case", GRIDS, ids=lambda c: "x".join(map(str, c[0])) + "_r%d_i%d" % c[1:])
@pytest.mark.parametrize("mode", [O.LEGACY, O.JACOBI], ids=["legacy", "jacobi"])
@pytest.mark.parametrize("how", ["coop", "coop_l2", "batch"])
def test_rows_sweeps_match_oracle(cuda, monkeypatch, case, mode, how):
    import torch
    from thesis_gb300 import stencil as S
    shape, radius, iters = case
    u = O.uniform(shape, seed=radius) - 0.5
    u[shape[0] // 2, shape[1] // 2] = -0.0
    if mode == O.JACOBI:  # border values that only some neighbours may see
        u[0, shape[1] // 2], u[shape[0] // 2, 0], u[shape[0] // 2, -1] = np.inf, np.nan, -np.inf
    pad = [torch.full((u.size + 64,), 7.0, device="cuda") for _ in range(2)]
    u1, u2 = (p[32:32 + u.size].view(shape) for p in pad)
    u1.copy_(torch.from_numpy(u)), u2.copy_(torch.from_numpy(u))
    if how == "batch":
        b = S.Batch([(u1, u2, radius, iters, mode, {"team": 3})], engine="one_launch")
        b.launch()
        res = b.result(0)
    else:
        monkeypatch.setenv("STENCIL_ROWS_L1", "0" if how == "coop_l2" else "1")
        res = S.sweep(u1, u2, radius, iters, mode, variant="coop")
    torch.cuda.synchronize()
    want, other = oracle_pair(u, u, radius, iters, mode)
    rest = u2 if res is u1 else u1
    for got, ref in ((res, want), (rest, other)):
        got = got.cpu().numpy()
        nan = np.isnan(ref)
        assert np.array_equal(np.isnan(got), nan)
        assert bits_equal(np.where(nan, 0, got), np.where(nan, 0, ref))
    for p in pad:
        assert (p[:32] == 7).all() and (p[-32:] == 7).all()
    assert S.device_status() == 0
