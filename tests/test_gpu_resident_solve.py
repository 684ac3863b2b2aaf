"""The field solve's resident kernels (whole GMRES restart cycles of small grids
in one launch) against the step graph on the same inputs.

A context with a wait bound set takes the step graph (the bound acts on its
applies), so one context gives both. Their sums run in other orders, so two
converged solutions agree to the solve's tolerance; iteration counts may
differ by one where an estimate falls on the tolerance. The step graph's two
applies (per-thread loads, and mass boxes by TMA on the tiled layout) form
every sum in the same order: bit for bit.

Grids: one cell and two per axis (every neighbour a periodic copy), partial
tiles on each axis, lines, planes and boxes, tiles of every size (1 to 256
threads a node), bases in shared memory and out of it, one to three tiles a CTA,
and grids too large for the resident kernels.
"""
from __future__ import annotations

import numpy as np
import pytest

from fieldutil import interior_nodes, periodic_cell_field, periodic_node_field, smooth_random_unique
from tpic_b200 import _lib
from tpic_b200.plasma import GridSpec
from test_gpu_tiled_apply import random_mass

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 1), (3, 2, 1), (2, 2, 2), (33, 1, 1), (200, 1, 1), (1, 70, 1), (31, 9, 1), (40, 24, 1),
          (150, 90, 1), (256, 130, 1), (5, 6, 7), (17, 16, 15), (33, 20, 18), (30, 40, 26), (48, 44, 40), (48, 48, 44),
          (64, 38, 63)]


def solve(ctx, inputs, adjoint):
    import torch
    e, b, j, m = inputs
    if not adjoint:
        return ctx.field_solve(e, b, j, m)
    lam = torch.zeros(3 * ctx.layout.node_count, dtype=torch.float64, device="cuda")
    ebar, bbar = torch.zeros_like(lam), torch.zeros(3 * ctx.layout.cell_count, dtype=torch.float64, device="cuda")
    res = _lib.GmresResult()
    _lib.check(ctx.lib.tpicb200_field_solve_backward(ctx.ctx, m.data_ptr(), e.double().data_ptr(), lam.data_ptr(),
                                                     ebar.data_ptr(), bbar.data_ptr(), res, ctx.stream))
    return lam, res


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("adjoint", [False, True])
def test_resident_solve_equals_the_step_graph(torch_cuda, shape, precision, adjoint):
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    rng = np.random.default_rng(sum(shape))
    tol = 1e-10
    e = periodic_node_field(g, smooth_random_unique(g, rng, 0.01))
    b = periodic_cell_field(g, smooth_random_unique(g, rng, 0.05))
    j = periodic_node_field(g, smooth_random_unique(g, rng, 0.02))
    mass = random_mass(g, rng, dt=0.1)
    stepped = {}
    for layout in (0, 1, 2):
        ctx = StageContext(g, precision=precision, dt=0.1, tol=tol, mass_layout=layout, max_iterations=300, restart=20)
        inputs = (ctx.field(e), ctx.field(b), ctx.field(j), ctx.mass_from_records(mass))
        got, res = solve(ctx, inputs, adjoint)
        again, _ = solve(ctx, inputs, adjoint)
        assert torch.equal(got, again)  # fixed summation order
        _lib.check(ctx.lib.tpicb200_set_wait_limit(ctx.ctx, 1 << 22))
        want, ref = solve(ctx, inputs, adjoint)
        stepped[layout] = want
        assert res.converged and ref.converged
        assert abs(res.iterations - ref.iterations) <= 1, (res.iterations, ref.iterations)
        assert res.rhs_norm == pytest.approx(ref.rhs_norm, rel=1e-12 if precision == 0 or adjoint else 1e-6)
        # Ghosts and duplicates included. A is within a few of the identity
        # here, so the error is at most that times the accepted residual.
        scale = np.abs(interior_nodes(g, want.cpu().numpy())).max()
        assert float((got - want).abs().max()) <= 20 * tol * max(res.rhs_norm, scale)
        ctx.close()
    assert torch.equal(stepped[1], stepped[2]) and torch.equal(stepped[0], stepped[1])


def system(ctx, g, rng):
    return (ctx.field(periodic_node_field(g, smooth_random_unique(g, rng, 0.01))),
            ctx.field(periodic_cell_field(g, smooth_random_unique(g, rng, 0.05))),
            ctx.field(periodic_node_field(g, smooth_random_unique(g, rng, 0.02))),
            ctx.mass_from_records(random_mass(g, rng, dt=0.1)))


@pytest.mark.parametrize("shapes", [((1024, 1, 1), (2, 1, 1)), ((96, 96, 1), (12, 12, 12)), ((150, 90, 1), (256, 130, 1)),
                                    ((30, 40, 26), (33, 20, 18))], ids=lambda s: "x".join(map(str, s[0])))
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("adjoint", [False, True])
def test_two_live_contexts_solve_in_turn(torch_cuda, shapes, precision, adjoint):
    """The kernels' shared memory limit is one for all contexts: plans of different sizes, forward and adjoint."""
    import torch
    from gpu_helpers import StageContext
    rng = np.random.default_rng(1)
    pairs = []
    for shape in shapes:
        g = GridSpec(*shape, *(0.1 * n for n in shape))
        ctx = StageContext(g, precision=precision, dt=0.1, tol=1e-10, mass_layout=1, max_iterations=300, restart=20)
        pairs.append((ctx, system(ctx, g, rng)))
    first = [solve(ctx, inputs, adjoint)[0] for ctx, inputs in pairs]
    for order in (0, 1, 1, 0):
        got, res = solve(*pairs[order], adjoint)
        assert res.converged and torch.equal(got, first[order])
    for ctx, _ in pairs:
        ctx.close()


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 1), (70, 1, 1), (5, 3, 1), (40, 24, 1), (1, 33, 1), (150, 90, 1)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("smoothing", [(1, 0.5, 0), (6, 0.5, 0), (3, 0.25, 1), (8, 0.75, 0)])
def test_resident_smoothed_solve_equals_the_step_graph(torch_cuda, shape, precision, smoothing):
    """Halos wider than the grid (every pass reads periodic copies of copies) and of several tiles."""
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    rng = np.random.default_rng(sum(shape))
    tol = 1e-10
    ctx = StageContext(g, precision=precision, dt=0.1, tol=tol, mass_layout=1, max_iterations=300, restart=20,
                       smoothing=smoothing)
    inputs = system(ctx, g, rng)
    got, res = ctx.field_solve(*inputs)
    _lib.check(ctx.lib.tpicb200_set_wait_limit(ctx.ctx, 1 << 22))
    want, ref = ctx.field_solve(*inputs)
    assert res.converged and ref.converged and abs(res.iterations - ref.iterations) <= 1
    scale = np.abs(interior_nodes(g, want.cpu().numpy())).max()
    assert float((got - want).abs().max()) <= 20 * tol * max(res.rhs_norm, scale)
    ctx.close()
