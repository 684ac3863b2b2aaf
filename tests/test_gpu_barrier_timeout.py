"""The bounded grid barriers of the cooperative kernels, tested without a fault:
tpicb200_inject_stall makes one wait of the sort's first CTA, or the first wait of
all CTAs of a solve's launch, expect arrivals that nothing makes,
tpicb200_set_wait_limit makes the bound short. In the sort the first CTA gives up
there; the others pass and run out at their next wait, or finish.

What each path then does, and that the next call on the context is right: the
binned sort's plan leaves the work to the general sort; the general sort's bins
come out empty, so that nothing is read through them; the solve fails."""
from __future__ import annotations

import numpy as np
import pytest

from fieldutil import periodic_node_field, smooth_random_unique
from test_gpu_resident_solve import system
from test_gpu_sort_launches import bins_of, check, moved, records
from tpic_b200 import _lib
from tpic_b200.plasma import Case, FieldInit, GridSpec, SpeciesSpec

pytestmark = pytest.mark.gpu
SORT_BIT = 1 << 22
POLLS = 1 << 13


def stall(lib, ctx, site, index):
    _lib.check(lib.tpicb200_set_wait_limit(ctx, POLLS if site else 0))
    _lib.check(lib.tpicb200_inject_stall(ctx, site, index))


def sort_case(torch, n, precision, far, rng, ctx, crowded=False):
    g = ctx.g
    d = records(g, n, rng, precision, crowded)
    counts, offsets = (torch.from_numpy(a).cuda() for a in bins_of(g, d["cell"]))
    if not crowded:
        d["cell"] = moved(g, d["cell"], rng, False)
    if far:  # bins that do not describe the records
        counts[int(counts.argmax())] -= 1
    return d, ctx.upload_particles(d), counts, offsets


@pytest.mark.parametrize("shape,n,crowded", [((4, 3, 1), 37, False), ((9, 8, 7), 20000, False),
                                             ((60, 52, 51), 300000, False), ((61, 1, 1), 50000, True)])
@pytest.mark.parametrize("precision", [0, 1])
def test_sort_barriers_that_give_up(torch_cuda, shape, n, crowded, precision):
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(1.0 * m for m in shape))
    rng = np.random.default_rng(n)
    ctx = StageContext(g, precision=precision, max_particles=n)
    assert ctx.lib.tpicb200_inject_stall(ctx.ctx, _lib.STALL_SORT, 0) == _lib.INVALID_ARGUMENT

    def sorted_right(far):
        d, src, c, o = sort_case(torch, n, precision, far, rng, ctx, crowded and far)
        out, counts, offsets = ctx.sort_binned(src, n, c, o)
        assert ctx.invalid_count() == 0
        check(g, d, out, counts, offsets, n)

    for wait in (1, 2):  # the plan's
        stall(ctx.lib, ctx.ctx, _lib.STALL_PLAN, wait)
        sorted_right(False)
        stall(ctx.lib, ctx.ctx, _lib.STALL_NONE, 0)
        sorted_right(False)
    bn = ctx.field(periodic_node_field(g, smooth_random_unique(g, rng, 0.1)))
    j, m = ctx.moments()
    # The general sort's: seven, and one a merge pass of the 40,000 records of one cell and one behind them.
    for wait in range(1, 12 if crowded else 8):
        d, src, c, o = sort_case(torch, n, precision, True, rng, ctx, crowded)
        stall(ctx.lib, ctx.ctx, _lib.STALL_SORT, wait)
        out, counts, offsets = ctx.sort_binned(src, n, c, o)
        assert ctx.invalid_count() == SORT_BIT, wait
        assert not counts.any() and not offsets.any()
        ctx.deposit(-1.0, src, n, bn, j, m, counts, offsets)
        assert not j.any() and not m.any()
        ctx.invalid.zero_()
        stall(ctx.lib, ctx.ctx, _lib.STALL_NONE, 0)
        sorted_right(True)
        sorted_right(False)
    ctx.close()


def simulation(fast):
    from tpic_b200.simulation import Simulation
    g = GridSpec(12, 10, 8, 6.0, 5.0, 4.0)
    sp = [SpeciesSpec(qom=-64.0, npcel=(3, 3, 3), vth=((9.0 if fast else 0.045),) * 3),
          SpeciesSpec(qom=1.0, npcel=(3, 3, 3), vth=(0.0056,) * 3)]
    sim = Simulation(Case(g, sp, dt=0.15, theta=0.5, gmres_tol=1e-8, fields=FieldInit(b0=(0.0, 0.0, 0.0195))),
                     precision="mixed", keep_ids=True)
    sim.prepare()
    return sim


def test_a_cycle_whose_plan_gives_up_is_the_same_cycle(torch_cuda):
    import torch
    results = []
    for site in (_lib.STALL_NONE, _lib.STALL_PLAN):
        sim = simulation(False)
        _lib.check(sim.lib.tpicb200_set_wait_limit(sim.ctx, POLLS))  # the same solve in both
        _lib.check(sim.lib.tpicb200_inject_stall(sim.ctx, site, 1))
        sim.run(2)
        results.append([sim.e, sim.j, sim.mass, *sim.bins[0], *sim.bins[1]])
    for a, b in zip(*results):
        assert torch.equal(a, b)


def test_a_cycle_whose_general_sort_gives_up_reports_invalid_data(torch_cuda):
    sim = simulation(True)
    stall(sim.lib, sim.ctx, _lib.STALL_SORT, 3)
    with pytest.raises(_lib.TpicError) as error:
        sim.run(1)
    assert error.value.status == _lib.INVALID_DATA


@pytest.mark.parametrize("shape", [(150, 90, 1), (17, 16, 15), (48, 48, 44)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("precision", [0, 1])
def test_solve_barriers_that_give_up(torch_cuda, shape, precision):
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    rng = np.random.default_rng(2)
    ctx = StageContext(g, precision=precision, dt=0.1, tol=1e-10, mass_layout=1, max_iterations=300, restart=20)
    inputs = system(ctx, g, rng)
    want, res = ctx.field_solve(*inputs)
    for launch in (1, 2):  # the start and the first restart cycle
        stall(ctx.lib, ctx.ctx, _lib.STALL_SOLVE, launch)
        with pytest.raises(_lib.TpicError) as error:
            ctx.field_solve(*inputs)
        assert error.value.status == _lib.BACKEND_FAILURE
        stall(ctx.lib, ctx.ctx, _lib.STALL_NONE, 0)
        got, again = ctx.field_solve(*inputs)
        assert torch.equal(got, want) and again.iterations == res.iterations
    ctx.close()
