"""The reverse step's launches at the edges of their blocks: stages of several
parts in one grid (128 items to a block), the array-wide first stage, the
one-launch reductions (256 cells to a block, 296 blocks at most), against the
same stages run one after the other on the host (tests/hostcheck).

Sizes: a part of full blocks and one an item short of that, one row and one column
of blocks, fewer cells than one block, and more cells than the reductions have
threads (75776).  Per item both sides do the same operations in the same order;
the gradient differs by the order of the sum that forms dt's adjoint (relative
1e-16 sqrt(cells), amplified by the steps) and by the device's fused
multiply-adds against the host's, which round alike: 1e-10 of the largest entry
is the bound the small cases of the adjoint are held to.
"""
from __future__ import annotations

import numpy as np
import pytest

import adjoint_host as ah
from athena_cuda_b200 import Grid, Params, configs, problem_state

pytestmark = pytest.mark.gpu

# a PLM part has (nx1 + 4)(nx2 + 4) items: 256 at 12 x 12, 255 at 13 x 11, 1024 at 124 x 4
SIZES = {
    "plm_two_full_blocks": (12, 12, "roe", (4, 4, 4, 4), 3),
    "plm_one_under": (13, 11, "roe", (1, 2, 2, 1), 3),
    "row_of_blocks": (124, 4, "roe", (4, 4, 1, 1), 3),
    "column_of_blocks": (4, 124, "hlle", (2, 2, 4, 4), 3),
    "under_one_block": (5, 4, "roe", (1, 1, 1, 1), 3),
    "more_cells_than_reduction_threads": (304, 251, "roe", (4, 4, 4, 4), 2),
}


@pytest.mark.parametrize("name", sorted(SIZES))
def test_reverse_launches_match_host(name):
    nx1, nx2, flux, bc, n = SIZES[name]
    p = Params.from_blocks(configs.blast(nx1, nx2, bc=bc, flux=flux, tlim=100.0))
    S0 = problem_state("blast", p)
    g = Grid.create(p.config())
    g.upload(S0)
    J, grad, st = g.adjoint_gradient(n)
    again = g.adjoint_gradient(n)
    g.close()
    Jh, gh, steps, _ = ah.adjoint(p.config(), S0, n, n + 1)
    assert st["steps"] == steps == n
    assert abs(J - Jh) <= (1e-13 + 1e-17 * nx1 * nx2) * abs(Jh)   # a tree of partials against one running sum
    scale = np.max(np.abs(gh))
    assert scale > 0
    assert np.max(np.abs(grad - gh)) <= 1e-10 * scale, np.max(np.abs(grad - gh)) / scale
    assert again[0] == J and np.array_equal(again[1], grad)
