"""Team sizes of the one-launch batch engine: chosen for the whole batch, hints
kept, every grid swept once whatever its team, bit for bit the oracle's."""
import pytest

from oracle import oracle as O
from test_batch_one_launch_gpu import _check, _make, _wants

pytestmark = pytest.mark.gpu

BATCHES = {
    # a lone grid and one with most of the work: no other grid to leave CTAs to
    "one": [((96, 120, 128), 2, 12, "jacobi")],
    "one_2d": [((1301, 1304), 1, 8, "jacobi")],
    "long_and_short": [((120, 100, 96), 1, 40, "jacobi")] + [((20 + 3 * k, 33 + k), 1 + k % 4, 2, "jacobi") for k in range(24)],
    # equal grids, more and fewer than the CTAs; some with no sweep
    "equal": [((40, 44), 2, 5, "jacobi")] * 200,
    "few": [((150, 131), 3, 7, "legacy"), ((30, 33, 37), 4, 5, "jacobi"), ((64, 64), 1, 0, "jacobi")],
    # either tile at R <= 2: widths around 64, 128 and 192, heights around 60
    "narrow_tiles": [((40, 93, 42), 2, 4, "jacobi"), ((21, 61, 63), 2, 3, "legacy"), ((30, 121, 150), 2, 3, "jacobi"),
                     ((33, 59, 190), 2, 2, "jacobi"), ((9, 64, 200), 2, 5, "jacobi"), ((26, 163, 176), 2, 3, "legacy"),
                     ((17, 31, 66), 1, 4, "jacobi"), ((12, 91, 129), 1, 3, "jacobi")],
    "no_sweeps": [((16, 16), 1, 0, "jacobi"), ((12, 12, 12), 2, 0, "jacobi")],
}


@pytest.mark.parametrize("hint", [0, 5])
@pytest.mark.parametrize("name", BATCHES)
def test_planned_teams_match_oracle(cuda, name, hint):
    import torch
    from thesis_gb300 import stencil as S
    specs = BATCHES[name]
    hosts, jobs, modes = _make(specs, 40)
    if hint:  # the first grid's own team size: the next smaller of the ladder
        jobs[0] = jobs[0] + ({"team": hint},)
    b = S.Batch(jobs, engine="one_launch")
    teams = b.teams()
    assert sum(n for _, n in teams) == len(specs)
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    ladder = [ctas >> k for k in range(ctas.bit_length())]
    assert all(t in ladder for t, _ in teams)
    if hint and len(specs) == 1:
        assert teams == [(max(t for t in ladder if t <= hint), 1)]
    if not hint and name in ("one", "one_2d", "long_and_short"):
        assert teams[0][0] > ctas // 4  # beyond the rule by cells
    b.launch()
    torch.cuda.synchronize()
    _check(b, specs, _wants(specs, hosts, modes), jobs)
    b.close()
    assert S.device_status() == 0
