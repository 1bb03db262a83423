"""The residual norm and the refinement's residual of 3-D grids, read by the
streaming sweep's code: partial tiles and chunks, narrow grids, each radius."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from oracle import ir_oracle as IRO

pytestmark = pytest.mark.gpu


# at least 2^23 cells (the rule's line), tile edges in x and y, one grid just
# below the line, one so narrow that both border bands meet
@pytest.mark.parametrize("shape,radius", [((70, 331, 364), 1), ((210, 200, 204), 2), ((203, 211, 200), 3),
                                          ((205, 205, 204), 4), ((1200, 900, 12), 4), ((9, 1000, 1000), 4),
                                          ((64, 256, 512), 1), ((63, 256, 512), 1)])
@pytest.mark.parametrize("alloc", [True, False])
def test_residual_norm_matches_oracle(cuda, shape, radius, alloc):
    import torch
    from thesis_gb300 import lib as L, stencil as S
    # border values of one sign and size, interior near the mean of them
    u = O.uniform(shape, seed=radius) * np.float32(0.01) + np.float32(1)
    want = O.rel_residual(u, radius, threads=8)
    d = torch.from_numpy(u).cuda()
    if alloc:
        got = S.residual(d, radius)
    else:
        p, out = L.make_params(shape, radius, 1, L.MODE_JACOBI), ctypes.c_double()
        L.check(L.load().stencil_residual_noalloc(ctypes.byref(p), ctypes.c_void_p(d.data_ptr()),
                                                  ctypes.byref(out), None), "stencil_residual_noalloc")
        got = out.value
    # FP32 per cell: 6R terms and as many roundings of relative 2^-24
    assert got == pytest.approx(want, rel=6 * radius * 2.0 ** -23)
    assert S.device_status() == 0


@pytest.mark.parametrize("storage", ["bf16", "fp16"])
@pytest.mark.parametrize("shape,radius", [((3, 3, 8), 1), ((40, 35, 136), 1), ((21, 33, 264), 2), ((9, 9, 16), 4),
                                          ((50, 49, 120), 4), ((100, 100, 128), 2)])
def test_refinement_step_of_one_sweep_is_exact(cuda, storage, shape, radius):
    """u + s * E(r / s) with r = (M u + c) - u in the sweep's order, bit for bit."""
    import torch
    from thesis_gb300 import stencil as S
    u = O.uniform(shape, seed=5) - np.float32(0.5)
    a, b = u.copy(), u.copy()
    swept = O.run(a, b, radius, O.JACOBI, 1)
    inner = (slice(radius, -radius),) * 3
    r = swept[inner] - u[inner]
    s = np.float32(np.ldexp(1.0, int(np.frexp(np.abs(r).max())[1])))
    want = u.copy()
    want[inner] = s * IRO.ROUND[storage](r * (np.float32(1) / s)).astype(np.float32) + u[inner]
    d = torch.from_numpy(u).cuda()
    S.ir_solve_ex(d, radius, 1, storage, inner_sweeps=1)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("storage,ulp", [("bf16", 2.0 ** -8), ("fp16", 2.0 ** -11)])
@pytest.mark.parametrize("shape", [(9, 9, 16), (10, 41, 24), (22, 40, 136), (35, 9, 264), (300, 33, 128), (64, 300, 152)],
                         ids=lambda s: "x".join(map(str, s)))
def test_tensor_core_correction_sweeps(cuda, storage, ulp, shape):
    """R = 4, three sweeps: z ranges shorter and longer than the plane ring, one
    and several chunks, partial tiles.  Sums in FP64 here, so a cell's rounding
    to 16 bits may fall the other way: one unit of the largest e (at most 1.5,
    M being a mean) per sweep, and e is read as 16 bits once more at the end."""
    import torch
    from thesis_gb300 import stencil as S
    R = 4
    u = O.uniform(shape, seed=6) - np.float32(0.5)
    swept = O.run(u.copy(), u.copy(), R, O.JACOBI, 1)
    inner = (slice(R, -R),) * 3
    r = swept[inner] - u[inner]
    s = np.float32(np.ldexp(1.0, int(np.frexp(np.abs(r).max())[1])))
    rhs = np.zeros(shape, np.float64)
    rhs[inner] = IRO.ROUND[storage](r * (np.float32(1) / s))
    e = rhs.copy()
    for _ in range(2):
        m = np.zeros(shape, np.float64)
        for ax in range(3):
            for o in (-4, -3, -2, -1, 1, 2, 3, 4):
                m += np.roll(e, -o, ax)
        nxt = np.zeros(shape, np.float64)
        nxt[inner] = IRO.ROUND[storage]((m[inner] / 24 + rhs[inner]).astype(np.float32))
        e = nxt
    d = torch.from_numpy(u).cuda()
    S.ir_solve_ex(d, R, 3, storage, inner_sweeps=3)
    got = d.cpu().numpy()
    assert np.abs(got - (u + s * e)).max() <= s * np.abs(e).max() * 3 * ulp
    border = np.ones(shape, bool)
    border[inner] = False
    assert np.array_equal(got[border], u[border])
