"""The 2-D register engine's barriers in tiles where some rows lie outside the
grid: warps differ in the row arithmetic, where __syncthreads() is not allowed."""
import os
import re

import pytest

from oracle import oracle as O

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "thesis_gb300", "csrc", "k_tb2d.cu")


def braces(text, start):
    """The text of the block that opens at or after start."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if not depth:
            return text[i:j]


def test_no_cta_wide_barrier_where_warps_differ():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    kernel = braces(text, text.index("k_tb2d_reg(float *g0"))
    row_arithmetic = braces(kernel, kernel.index("auto whole)"))
    assert "__shfl" in row_arithmetic and "__syncthreads" not in row_arithmetic


@pytest.mark.gpu
@pytest.mark.parametrize("shape,radius", [((67, 128), 1), ((131, 96), 1), ((254, 250), 1), ((67, 120), 2), ((200, 203), 2)])
def test_tiles_with_rows_outside_the_grid(cuda, shape, radius):
    """Warps with and without rows beyond the update region in one tile."""
    from test_ragged_gpu import test_ragged_sweeps_match_oracle
    for mode in (O.LEGACY, O.JACOBI):
        test_ragged_sweeps_match_oracle(cuda, (shape, radius, 41 if mode == O.JACOBI else 8), mode)
