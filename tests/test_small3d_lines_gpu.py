"""Which engine small 3-D grids left to the library take, on both sides of each
line, and that they stay out of one another's way on several streams."""
import pytest

pytestmark = pytest.mark.gpu


# held in one cluster's shared memory; not held, swept by a cluster from the L2;
# by the streaming sweeps
@pytest.mark.parametrize("shape,radius,engine", [((64, 64, 64), 1, "cluster"), ((48, 48, 48), 1, "cluster"), ((56, 56, 56), 2, "cluster"),
                                                 ((68, 64, 64), 1, "stream3d-persistent"), ((40, 40, 40), 4, "cluster"),
                                                 ((64, 64, 64), 2, "stream3d-persistent"), ((52, 52, 52), 4, "stream3d-persistent")])
def test_engine(cuda, shape, radius, engine):
    from thesis_gb300 import stencil as S
    a = S.init_uniform(shape, 1)
    S.sweep(a, a.clone(), radius, 8)
    assert S.last_dispatch()[0] == engine


@pytest.mark.parametrize("shape,radius", [((64, 64, 64), 1), ((56, 56, 56), 2)])
def test_grids_on_several_streams_run_side_by_side(cuda, shape, radius):
    """Eight grids on clusters of 16 of the GPU's SMs: well under half of eight
    launches in a row."""
    import torch
    from thesis_gb300 import stencil as S
    grids = [(S.init_uniform(shape, k), S.init_uniform(shape, k)) for k in range(8)]
    streams = [torch.cuda.Stream() for _ in grids]

    def ms(n):
        best = 1e9
        for _ in range(4):
            torch.cuda.synchronize()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for (a, b), s in list(zip(grids, streams))[:n]:
                s.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(s):
                    S.sweep(a, b, radius, 2000, stream=s)
            for s in streams[:n]:
                torch.cuda.current_stream().wait_stream(s)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best

    assert ms(8) < 0.4 * 8 * ms(1)
