"""Persistent launches beside one another: on many streams, captured and replayed
beside other calls, from several threads; bit for bit the oracle's."""
import threading

import numpy as np
import pytest

from oracle import oracle as O
from test_cluster_gpu import bits_equal, oracle_pair

pytestmark = pytest.mark.gpu


def grid(shape, seed):
    import torch
    u = O.uniform(shape, seed=seed) - 0.5
    return u, torch.from_numpy(u).cuda(), torch.from_numpy(u).cuda()


# the 2-D engine on rows that are and are not 16-byte aligned, the rows kernels,
# the 3-D streaming and ragged sweeps
CASES = [((66, 71), 1, 40), ((66, 72), 1, 40), ((1300, 1301), 1, 8), ((1300, 1304), 2, 8), ((40, 61, 72), 2, 9), ((40, 61, 71), 2, 9)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])))
def test_replays_beside_other_calls(cuda, case):
    """A graph captured after a warm-up call, replayed after calls on larger
    grids, after a release and beside hundreds of other launches."""
    import torch
    from thesis_gb300 import lib, stencil as S
    shape, radius, iters = case
    u, a, b = grid(shape, 3)
    want, _ = oracle_pair(u, u, radius, iters, O.JACOBI)
    S.sweep(a, b, radius, iters)
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        res = S.sweep(a, b, radius, iters, stream=s)
    big, small = grid((501, 503), 4), [grid((66, 71), 5 + k) for k in range(3)]
    bigger, _ = oracle_pair(big[0], big[0], 1, 20, O.JACOBI)
    for rep in range(3):
        a.copy_(torch.from_numpy(u)), b.copy_(torch.from_numpy(u))
        for x in (big, *small):
            x[1].copy_(torch.from_numpy(x[0])), x[2].copy_(torch.from_numpy(x[0]))
        if rep == 1:
            lib.check(lib.load().stencil_release(), "stencil_release")
        torch.cuda.synchronize()
        other = [torch.cuda.Stream() for _ in range(4)]
        for k in range(100):
            for st, x in zip(other[1:], small):
                with torch.cuda.stream(st):
                    S.sweep(x[1], x[2], 1, 10, stream=st)
            if k == 20:
                with torch.cuda.stream(s):
                    g.replay()
                with torch.cuda.stream(other[0]):
                    out = S.sweep(big[1], big[2], 1, 20, stream=other[0])
        torch.cuda.synchronize()
        assert bits_equal(res.cpu().numpy(), want)
        assert bits_equal(out.cpu().numpy(), bigger)
        for x in small:
            ref, _ = oracle_pair(x[0], x[0], 1, 1000, O.JACOBI)
            assert bits_equal(x[1].cpu().numpy(), ref)
    assert S.device_status() == 0


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])))
def test_more_streams_than_slots(cuda, case):
    import torch
    from thesis_gb300 import stencil as S
    shape, radius, iters = case
    iters += iters % 2
    n, launches = 20, 3
    grids = [grid(shape, 10 + k) for k in range(n)]
    streams = [torch.cuda.Stream() for _ in range(n)]
    torch.cuda.synchronize()
    for _ in range(launches):
        for (_, a, b), st in zip(grids, streams):
            with torch.cuda.stream(st):
                S.sweep(a, b, radius, iters, stream=st)
    torch.cuda.synchronize()
    for u, a, _ in grids:
        want, _ = oracle_pair(u, u, radius, iters * launches, O.JACOBI)
        assert bits_equal(a.cpu().numpy(), want)
    assert S.device_status() == 0


def test_a_long_launch_beside_hundreds_of_short_ones(cuda):
    """The long launch's barrier counter is nobody else's while it runs."""
    import torch
    from thesis_gb300 import stencil as S
    u, a, b = grid((33, 61, 57), 1)  # both persistent
    v, c, d = grid((45, 46, 47), 2)
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        S.sweep(a, b, 1, 4000, stream=s)
    assert S.last_dispatch() == ("ragged3d-persistent", 1)
    for _ in range(700):
        with torch.cuda.stream(t):
            S.sweep(c, d, 1, 4, stream=t)
    assert S.last_dispatch() == ("ragged3d-persistent", 1)
    torch.cuda.synchronize()
    assert bits_equal(a.cpu().numpy(), oracle_pair(u, u, 1, 4000, O.JACOBI)[0])
    assert bits_equal(c.cpu().numpy(), oracle_pair(v, v, 1, 2800, O.JACOBI)[0])
    assert S.device_status() == 0


def test_threads_on_shared_streams(cuda):
    """Launches that threads enqueue on the same stream interleave in any order."""
    import torch
    from thesis_gb300 import stencil as S
    streams = [torch.cuda.Stream() for _ in range(2)]
    work = [[grid(shape, 20 + k) for shape in ((66, 71), (130, 128), (45, 46, 47))] for k in range(4)]
    torch.cuda.synchronize()
    errors = []

    def run(k):
        try:
            for _ in range(40):
                for _, a, b in work[k]:
                    with torch.cuda.stream(streams[k % 2]):
                        S.sweep(a, b, 1, 10, stream=streams[k % 2])
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    [t.start() for t in threads], [t.join() for t in threads]
    torch.cuda.synchronize()
    assert not errors
    for grids in work:
        for u, a, _ in grids:
            assert bits_equal(a.cpu().numpy(), oracle_pair(u, u, 1, 400, O.JACOBI)[0])
    assert S.device_status() == 0


def test_a_larger_capture_than_any_call_is_refused(cuda):
    """Rows that are 16-byte aligned, as before; others take the rows kernel."""
    import torch
    from thesis_gb300 import lib, stencil as S
    lib.check(lib.load().stencil_release(), "stencil_release")
    _, a, b = grid((66, 72), 1)
    u, c, d = grid((66, 71), 1)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        with pytest.raises(Exception, match="outside the graph capture"):
            S.sweep(a, b, 1, 10, stream=s)
        S.sweep(c, d, 1, 10, stream=s)
    g.replay()
    torch.cuda.synchronize()
    assert bits_equal(c.cpu().numpy(), oracle_pair(u, u, 1, 10, O.JACOBI)[0])


def test_graphs_give_their_buffers_back(cuda):
    import gc
    import torch
    from thesis_gb300 import stencil as S
    a = S.init_uniform((512, 512), 1)
    b = a.clone()
    S.sweep(a, b, 1, 10)
    s = torch.cuda.Stream()

    def capture():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(3):
                S.sweep(a, b, 1, 10, stream=s)
        g.replay()
        torch.cuda.synchronize()

    capture()
    gc.collect()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(60):
        capture()
    gc.collect()
    # two slots of 8 bytes a cell each time would be 250 MB
    assert before - torch.cuda.mem_get_info()[0] < 100 << 20


def test_launches_in_other_threads_during_a_capture(cuda):
    """A capture does not stop other threads' calls, nor do they end it."""
    import ctypes
    import torch
    from thesis_gb300 import lib, stencil as S
    lib.check(lib.load().stencil_release(), "stencil_release")
    u, a, b = grid((66, 71), 1)
    S.sweep(a, b, 1, 10)
    a.copy_(torch.from_numpy(u)), b.copy_(torch.from_numpy(u))
    other = [grid(shape, 30 + k) for k, shape in enumerate([(301, 304), (401, 399), (45, 46, 47), (90, 91, 92), (66, 71)])]
    torch.cuda.synchronize()
    s, g, errors = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []

    def run():
        try:
            t = torch.cuda.Stream()
            for _, x, y in other[:4]:
                for _ in range(3):
                    with torch.cuda.stream(t):
                        S.sweep(x, y, 1, 10, stream=t)
            _, x, y = other[4]  # the thread's own default stream
            p = lib.make_params((66, 71), 1, 30, lib.MODE_JACOBI)
            lib.check(lib.load().stencil_dispatch_ex(ctypes.byref(p), ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()),
                                                     ctypes.c_void_p(2), None), "dispatch")
        except Exception as e:
            errors.append(e)

    with torch.cuda.graph(g, stream=s):
        S.sweep(a, b, 1, 10, stream=s)
        t = threading.Thread(target=run)
        t.start(), t.join()
        S.sweep(a, b, 1, 10, stream=s)
    assert not errors, errors
    g.replay()
    torch.cuda.synchronize()
    assert bits_equal(a.cpu().numpy(), oracle_pair(u, u, 1, 20, O.JACOBI)[0])
    for v, x, _ in other:
        assert bits_equal(x.cpu().numpy(), oracle_pair(v, v, 1, 30, O.JACOBI)[0])
    assert S.device_status() == 0
