"""3-D grids whose rows are not 16-byte aligned, on both sides of the line between
a launch per sweep and the persistent sweeps: which one takes them, and the
oracle's bits at the edges of the persistent sweeps' tiles and z-chunks."""
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (nz, ny, nx), radius: a tile more and less along x and y, all residues of nx and
# nx * ny modulo 4, both tile shapes, few and many planes
PERSISTENT = [((44, 43, 43), 1), ((9, 97, 127), 1), ((150, 17, 33), 1), ((12, 65, 129), 1), ((37, 35, 38), 2), ((6, 70, 131), 2),
              ((7, 34, 254), 2), ((120, 20, 21), 2), ((49, 48, 49), 3), ((10, 90, 131), 3), ((200, 24, 26), 3), ((55, 53, 54), 4),
              ((13, 93, 130), 4), ((11, 110, 127), 4), ((330, 22, 21), 4)]
LAUNCHES = [((42, 43, 43), 1), ((35, 36, 35), 2), ((46, 47, 47), 3), ((52, 53, 53), 4), ((17, 65, 129), 4), ((9, 9, 9), 4)]


@pytest.mark.parametrize("shape,radius", PERSISTENT, ids=lambda v: str(v).replace(", ", "x"))
@pytest.mark.parametrize("mode", [O.LEGACY, O.JACOBI], ids=["legacy", "jacobi"])
def test_persistent(cuda, shape, radius, mode):
    from test_ragged_gpu import test_ragged_sweeps_match_oracle
    from thesis_gb300 import stencil as S
    test_ragged_sweeps_match_oracle(cuda, (shape, radius, 5), mode)
    assert S.last_dispatch() == ("ragged3d-persistent", 1)


@pytest.mark.parametrize("shape,radius", LAUNCHES, ids=lambda v: str(v).replace(", ", "x"))
def test_a_launch_per_sweep(cuda, shape, radius):
    from test_ragged_gpu import test_ragged_sweeps_match_oracle
    from thesis_gb300 import stencil as S
    test_ragged_sweeps_match_oracle(cuda, (shape, radius, 9), O.JACOBI)
    assert S.last_dispatch() == ("base", 9)


def test_few_sweeps_of_a_large_grid(cuda):
    from test_ragged_gpu import test_ragged_sweeps_match_oracle
    from thesis_gb300 import stencil as S
    test_ragged_sweeps_match_oracle(cuda, ((162, 161, 161), 2, 1), O.JACOBI)
    assert S.last_dispatch() == ("ragged3d-persistent", 1)
