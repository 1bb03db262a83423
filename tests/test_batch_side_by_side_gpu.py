"""Phased batches on clusters of one CTA: the small 2-D grids' launch and the
other grids' run beside one another."""
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu

# many short grids of either kind beside long ones of the other, ragged ones
MIXES = {"long 2-D": [((60, 61), 1, 900)] * 2 + [((50, 40), 2, 8)] * 5 + [((9, 10, 12), 1, 20)],
         "long others": [((60, 64), 1, 12)] * 5 + [((50, 41), 2, 400)] + [((9, 10, 12), 1, 200)],
         "one kind": [((60, 64), 1, 12), ((61, 33), 1, 9)]}


@pytest.mark.parametrize("mix", MIXES)
def test_results_and_replays(cuda, mix):
    import torch
    from thesis_gb300 import stencil as S
    hosts = [O.uniform(shape, seed=60 + k) for k, (shape, _, _) in enumerate(MIXES[mix])]
    jobs = [(torch.from_numpy(u).cuda(), torch.from_numpy(u).cuda(), r, n, O.JACOBI)
            for u, (_, r, n) in zip(hosts, MIXES[mix])]
    b = S.Batch(jobs, cluster_size=1, engine="phased")

    def check():
        torch.cuda.synchronize()
        for k, (_, r, n) in enumerate(MIXES[mix]):
            assert bits_equal(b.result(k).cpu().numpy(), oracle_pair(hosts[k], hosts[k], r, n, O.JACOBI)[0]), k

    b.launch()
    check()
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        b.launch(stream=s)
    for _ in range(2):
        for (x, y, *_), u in zip(jobs, hosts):
            x.copy_(torch.from_numpy(u)), y.copy_(torch.from_numpy(u))
        g.replay()
        check()


def test_neither_launch_waits_for_the_other(cuda):
    import torch
    from thesis_gb300 import stencil as S

    def ms(specs):
        jobs = []
        for shape, n in specs:
            a = S.init_uniform(shape, 1)
            jobs.append((a, a.clone(), 1, n, O.JACOBI))
        t = S.Batch(jobs, cluster_size=1, engine="phased")
        best = 1e9
        for _ in range(3):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(), t.launch(), e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        t.close()
        return best

    flat, deep = [((120, 124), 30000)] * 20, [((20, 32, 32), 3000)] * 20
    one, other = ms(flat), ms(deep)
    # 40 CTAs on 152 SMs: as long as the longer one, with room for the clocks
    assert ms(flat + deep) < 1.2 * max(one, other) + 0.1
    assert min(one, other) > 0.4 * max(one, other)
