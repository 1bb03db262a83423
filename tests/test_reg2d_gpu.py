"""Small 2-D grids in the registers of one CTA (batches on clusters of one):
bit for bit the oracle's, both buffers, at the edges of the row blocks and lane
groups."""
import numpy as np
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu

# (ny, nx), sweeps: the smallest grid, 64 / 65 wide (16 or 32 lanes a row),
# rows at and around full blocks, widths that are not multiples of 4, the
# largest of each lane group, and one row or column too many (another path)
GRIDS = [((3, 3), 5), ((3, 128), 4), ((25, 64), 1), ((26, 61), 2), ((64, 64), 7), ((73, 65), 0), ((74, 68), 33),
         ((85, 100), 9), ((96, 127), 6), ((109, 125), 3), ((128, 128), 50), ((133, 126), 11), ((255, 64), 8),
         ((265, 63), 5), ((120, 36), 2), ((134, 128), 4), ((128, 132), 4), ((266, 64), 3)]


@pytest.mark.parametrize("border", ["equal", "unequal", "special"])
def test_single_cta_batches_match_oracle(cuda, border):
    import torch
    from thesis_gb300 import stencil as S
    hosts, jobs = [], []
    for k, (shape, iters) in enumerate(GRIDS):
        u = O.uniform(shape, seed=40 + k) - 0.5
        if border == "special":  # signed zeros, infinities and a NaN, in the border and inside
            u[0, 1], u[-1, -2], u[shape[0] // 2, 0] = -np.inf, np.nan, np.inf
            u[1, 1:3] = -0.0
        v = u.copy()
        if border == "unequal":
            v[0, 1] += 1.0
            v[shape[0] // 2, -1] -= 1.0
        hosts.append((u, v))
        jobs.append((torch.from_numpy(u.copy()).cuda(), torch.from_numpy(v.copy()).cuda(), 1, iters, O.JACOBI))
    b = S.Batch(jobs, cluster_size=1, engine="phased")
    b.launch()
    torch.cuda.synchronize()
    for k, (shape, iters) in enumerate(GRIDS):
        res, other = oracle_pair(hosts[k][0], hosts[k][1], 1, iters, O.JACOBI)
        got = b.result(k)
        rest = jobs[k][1] if got is jobs[k][0] else jobs[k][0]
        for t, want in ((got, res), (rest, other)):
            t = t.cpu().numpy()
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(t), nan), (shape, iters)
            assert bits_equal(np.where(nan, 0, t), np.where(nan, 0, want)), (shape, iters)
    b.close()
