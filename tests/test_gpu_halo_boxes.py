"""The TMA apply's boxes, which hold a halo along y or z only for the stencils
that reach there, against the per-thread-load apply.

Both form every product and sum in the same order, so the solves agree bit for
bit. A wait limit of the default size (tpicb200_set_wait_limit) keeps the solve
on the step's kernels on these small grids. The grids end inside a tile, on
its last node, and one node beyond it, on each axis.
"""
from __future__ import annotations

import numpy as np
import pytest

from tpic_b200 import _lib
from tpic_b200.plasma import GridSpec
from test_gpu_tiled_apply import assert_same_result, contexts, random_mass, solve_backward, solve_inputs
from fieldutil import periodic_node_field, smooth_random_unique

pytestmark = pytest.mark.gpu

# Tiles are 32 x 4 x 2 nodes, 32 x 8 x 1 on grids one cell thick along z.
GRIDS = [(32, 4, 2), (31, 3, 3), (33 + 2, 5, 1), (64, 9, 4), (6, 8, 1), (2, 1, 2), (3, 2, 1)]


@pytest.mark.parametrize("shape", GRIDS, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", [0, 1])
def test_boxes_equal_the_per_thread_loads(torch_cuda, shape, precision):
    import torch
    nx, ny, nz = shape
    g = GridSpec(nx, ny, nz, 0.2 * nx, 0.2 * ny, 0.2 * nz)
    rng = np.random.default_rng(29)
    sm, tl = contexts(g, precision)
    for ctx in (sm, tl):
        _lib.check(ctx.lib.tpicb200_set_wait_limit(ctx.ctx, 1 << 22))
    m = random_mass(g, rng)
    e, b, j = solve_inputs(g, rng)
    etheta_bar = torch.from_numpy(periodic_node_field(g, smooth_random_unique(g, rng, 1.0))).cuda()
    out = []
    for ctx in (sm, tl):
        et, res = ctx.field_solve(ctx.field(e), ctx.field(b), ctx.field(j), ctx.mass_from_records(m))
        lam, e_bar, b_bar, back = solve_backward(ctx, ctx.mass_from_records(m), etheta_bar)
        torch.cuda.synchronize()
        assert ctx.invalid_count() == 0
        out.append((et, lam, e_bar, b_bar, res, back))
        ctx.close()
    for x, y in zip(out[0][:4], out[1][:4]):
        assert torch.equal(x, y)
    assert_same_result(out[0][4], out[1][4])
    assert_same_result(out[0][5], out[1][5])
