"""The smoothing passes over shared-memory tiles (tpicb200_smooth) against the
oracle bit for bit, ghosts and duplicates included, where tiles, halos and
launches meet the grid: axes of one to three cells (a halo wraps several
times), partial tiles, exact tiles, flat grids and boxes, pass counts on both
sides of what one launch takes (8 passes, one on grids thicker than a cell on
every axis)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle as O
from fieldutil import periodic_node_field
from reference_fixtures import ogrid
from tpic_b200.plasma import GridSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (33, 1, 1), (1, 9, 1), (1, 1, 17), (3, 2, 1), (32, 8, 1),
                                   (45, 19, 1), (1, 20, 11), (2, 3, 2), (16, 8, 8), (17, 9, 10)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("passes,alpha,op", [(1, 0.5, 0), (3, 0.5, 1), (4, 0.25, 0), (6, 0.5, 0), (7, 0.0, 1),
                                             (9, 0.75, 0), (17, 0.5, 0)])
def test_tiled_passes_match_the_oracle(torch_cuda, shape, passes, alpha, op):
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    rng = np.random.default_rng(11)
    f = periodic_node_field(g, rng.normal(size=(3, g.nz, g.ny, g.nx)))
    want = np.zeros_like(f)
    O.load().oracle_smooth(C.byref(ogrid(g)), passes, alpha, op, O.ptr(f), O.ptr(want))
    ctx = StageContext(g, 0, smoothing=(passes, alpha, op))
    src = ctx.field(f, np.float64)
    out = torch_cuda.full_like(src, np.nan)
    assert ctx.lib.tpicb200_smooth(ctx.ctx, src.data_ptr(), out.data_ptr(), ctx.stream) == 0
    assert np.array_equal(out.cpu().numpy(), want)
    ctx.close()
