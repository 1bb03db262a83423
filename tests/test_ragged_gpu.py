"""Sweeps of grids whose rows are not 16-byte aligned, left to the library: bit
for bit the oracle's, both buffers, at the edges of the tiles and z-chunks."""
import numpy as np
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu

# (nz, ny, nx), radius, sweeps: the smallest grids of each radius, one column
# more and less than a tile, all residues of nx and of nx * ny modulo 4, both
# tile shapes, one sweep
GRIDS_3D = [((3, 3, 3), 1, 4), ((9, 9, 9), 4, 3), ((5, 6, 7), 2, 1), ((7, 8, 7), 3, 6), ((12, 17, 127), 1, 5),
            ((9, 34, 129), 2, 4), ((11, 33, 66), 1, 7), ((10, 40, 65), 3, 2), ((14, 19, 253), 4, 3), ((40, 30, 62), 2, 9),
            ((24, 70, 131), 4, 2), ((33, 21, 58), 3, 5)]
# (ny, nx), radius, sweeps: the temporally blocked engine (one tile per SM) and,
# beyond it, the rows kernel; sweep counts around an exchange; fewer than eight
# sweeps (a launch each)
GRIDS_2D = [((9, 9), 4, 8), ((3, 5), 1, 9), ((67, 67), 3, 8), ((256, 255), 1, 61), ((130, 513), 2, 20), ((70, 66), 4, 13),
            ((1500, 1501), 1, 9), ((900, 2049), 2, 8), ((2050, 701), 3, 8), ((640, 3333), 4, 11), ((300, 301), 1, 5)]


@pytest.mark.parametrize("case", GRIDS_3D + GRIDS_2D, ids=lambda c: "x".join(map(str, c[0])) + "_r%d_i%d" % c[1:])
@pytest.mark.parametrize("mode", [O.LEGACY, O.JACOBI], ids=["legacy", "jacobi"])
def test_ragged_sweeps_match_oracle(cuda, case, mode):
    import torch
    from thesis_gb300 import stencil as S
    shape, radius, iters = case
    u = O.uniform(shape, seed=radius) - 0.5
    u[tuple(n // 2 for n in shape)] = -0.0
    second = O.uniform(shape, seed=9) if mode == O.LEGACY else u
    if mode == O.JACOBI:  # a border infinity and zeros reach the slow division
        u[(0,) * (len(shape) - 1) + (shape[-1] // 2,)] = np.inf
        second = u
    # buffers inside larger ones: nothing outside the grid is written
    pad = [torch.full((u.size + 64,), 7.0, device="cuda") for _ in range(2)]
    u1, u2 = (p[32:32 + u.size].view(shape) for p in pad)
    u1.copy_(torch.from_numpy(u)), u2.copy_(torch.from_numpy(second))
    res = S.sweep(u1, u2, radius, iters, mode)
    want, other = oracle_pair(u, second, radius, iters, mode)
    rest = u2 if res is u1 else u1
    for got, ref in ((res, want), (rest, other)):
        got = got.cpu().numpy()
        nan = np.isnan(ref)
        assert np.array_equal(np.isnan(got), nan)
        assert bits_equal(np.where(nan, 0, got), np.where(nan, 0, ref))
    for p in pad:
        assert (p[:32] == 7).all() and (p[-32:] == 7).all()


def test_ragged_sweeps_replay_in_a_graph_and_side_by_side(cuda):
    import torch
    from thesis_gb300 import stencil as S
    shape, radius, iters = (21, 35, 101), 2, 6
    u = O.uniform(shape, seed=3)
    want, _ = oracle_pair(u, u, radius, iters, O.JACOBI)
    bufs = [[torch.from_numpy(u).cuda() for _ in range(2)] for _ in range(2)]
    s = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for (a, b), st in zip(bufs, s):
        with torch.cuda.stream(st):
            res = S.sweep(a, b, radius, iters, stream=st)
    torch.cuda.synchronize()
    for a, _ in bufs:
        assert bits_equal(a.cpu().numpy(), want)
    a, b = bufs[0]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s[0]):
        S.sweep(a, b, radius, iters, stream=s[0])
    for _ in range(2):
        a.copy_(torch.from_numpy(u)), b.copy_(torch.from_numpy(u))
        g.replay()
        torch.cuda.synchronize()
        assert bits_equal(a.cpu().numpy(), want)


def test_ragged_2d_dispatch_captured_before_any_other(cuda):
    """A graph capture of a grid no earlier call has made an exchange buffer
    for (in a process of its own)."""
    import os
    import subprocess
    import sys
    code = """
import torch, numpy as np
from oracle import oracle as O
from thesis_gb300 import stencil as S
u = O.uniform((66, 71), seed=3)
a, b = torch.from_numpy(u).cuda(), torch.from_numpy(u).cuda()
torch.cuda.synchronize()
s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    S.sweep(a, b, 1, 10, stream=s)
g.replay()
torch.cuda.synchronize()
x, y = u.copy(), u.copy()
want = O.run(x, y, 1, O.JACOBI, 10, threads=4)
assert np.array_equal(a.cpu().numpy().view(np.uint32), want.view(np.uint32))
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], cwd=root, check=True, timeout=300)
