"""Kernel launches that a solve reports: residual checks of large 3-D grids take
three, others two."""
import pytest

pytestmark = pytest.mark.gpu


# the streaming residual pass from 2^23 cells on
@pytest.mark.parametrize("shape,check", [((64, 256, 512), 3), ((63, 256, 512), 2), ((512, 512), 2), ((210, 201, 203), 2)])
def test_residual_checks_are_counted(cuda, shape, check):
    from thesis_gb300 import stencil as S
    u = S.init_uniform(shape, 1)
    if shape[-1] % 8 == 0:
        r = S.ir_solve_ex(u, 1, 12, "bf16", inner_sweeps=6, tol=1e-30, engine="launches")
        # an outer step: two residual passes, five sweeps, the update, the check
        assert r["outer_steps"] == 2 and r["kernel_launches"] == 2 * (8 + check)
    S.solve(u, u.clone(), 1, 16, 0.0, check_every=8, variant="base")
    assert S.last_dispatch() == ("base", 16 + 3 * check)
