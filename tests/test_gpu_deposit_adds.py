"""The deposition adds to what J and the mass hold, in every mass form, also
right behind tpicb200_clear_moments: values that the caller put there after the
clear, another context's deposition into the same buffers, and the replays of a
graph that recorded the deposition and not the clear.

There are records enough for the scalar forms to deposit cell moments: an entry's
sum over the records is the same number each time and is added in one rounding, so
the comparisons with the sum added on the host are exact."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from fieldutil import periodic_node_field, smooth_random_unique
from test_gpu_scalar_moments import QOM, bins, ragged_species
from tpic_b200 import _lib
from tpic_b200.plasma import GridSpec

pytestmark = pytest.mark.gpu

FORMS = [(0, _lib.MASS_SCALAR), (0, _lib.MASS_SCALAR_F64), (0, _lib.MASS_MOMENTS_F64), (1, _lib.MASS_SCALAR),
         (1, _lib.MASS_SCALAR_F64), (1, _lib.MASS_TF32), (1, _lib.MASS_BF16X3)]
SHAPES = [(8, 6, 4), (5, 3, 2)]  # the assembly by quads of cells and by nodes


class Species:
    def __init__(self, ctx, g, s, precision):
        rng = np.random.default_rng(s)
        d = ragged_species(g, s, rng, precision, 0.5)
        self.n, self.qom = len(d["cell"]), QOM[s]
        self.parts = ctx.upload_particles(d)
        self.bins = bins(ctx, d)

    def into(self, ctx, bn, j, m, kind):
        ctx.deposit(self.qom, self.parts, self.n, bn, j, m, *self.bins, kind=kind)


def clear(ctx, j, m):
    _lib.check(ctx.lib.tpicb200_clear_moments(ctx.ctx, j.data_ptr(), m.data_ptr(), ctx.stream))


def unique(ctx, t):
    """The values at the unique nodes (the stored order of the layout's other axes kept)."""
    g = ctx.g
    nodes = t.numel() // (g.nx + 3) // (g.ny + 3) // (g.nz + 3)
    return t.reshape(nodes, g.nz + 3, g.ny + 3, g.nx + 3)[:, 1:g.nz + 1, 1:g.ny + 1, 1:g.nx + 1]


def setting(precision, shape):
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    ctx = StageContext(g, precision=precision, dt=0.2, mass_layout=1)
    rng = np.random.default_rng(5)
    return g, ctx, ctx.field(periodic_node_field(g, smooth_random_unique(g, rng, 0.9)))


@pytest.mark.parametrize("shape", SHAPES, ids=["8x6x4", "5x3x2"])
@pytest.mark.parametrize("precision,kind", FORMS)
def test_values_put_there_after_the_clear_stay(torch_cuda, precision, kind, shape):
    import torch
    g, ctx, bn = setting(precision, shape)
    s = Species(ctx, g, 0, precision)
    j, m = ctx.moments()
    external = [torch.rand_like(t) * 1e-3 for t in (j, m)]
    alone = ctx.moments()
    s.into(ctx, bn, *alone, kind)
    ctx.fold(*alone)
    clear(ctx, j, m)
    for t, x in zip((j, m), external):
        t += x
    s.into(ctx, bn, j, m, kind)
    ctx.fold(j, m)
    assert ctx.invalid_count() == 0
    for t, x, a in zip((j, m), external, alone):
        assert torch.equal(unique(ctx, t), unique(ctx, x) + unique(ctx, a))
    ctx.close()


@pytest.mark.parametrize("precision,kind", FORMS)
def test_another_contexts_species_stays(torch_cuda, precision, kind):
    import torch
    g, ctx, bn = setting(precision, SHAPES[0])
    _, other, _ = setting(precision, SHAPES[0])
    first, second = Species(ctx, g, 0, precision), Species(ctx, g, 1, precision)
    alone = [ctx.moments() for _ in range(2)]
    for s, a in zip((first, second), alone):
        s.into(ctx, bn, *a, kind)
        ctx.fold(*a)
    j, m = ctx.moments()
    clear(ctx, j, m)
    first.into(other, bn, j, m, kind)
    other.fold(j, m)
    second.into(ctx, bn, j, m, kind)
    ctx.fold(j, m)
    for t, a, b in zip((j, m), *alone):
        assert torch.equal(unique(ctx, t), unique(ctx, a) + unique(ctx, b))
    ctx.close()
    other.close()


@pytest.mark.parametrize("precision,kind", FORMS)
def test_replays_of_the_deposition_alone_add(torch_cuda, precision, kind):
    import torch
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        g, ctx, bn = setting(precision, SHAPES[0])
        s = Species(ctx, g, 0, precision)
        alone, (j, m) = ctx.moments(), ctx.moments()
        s.into(ctx, bn, *alone, kind)
        ctx.fold(*alone)
        clear(ctx, j, m)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            s.into(ctx, bn, j, m, kind)
            ctx.fold(j, m)
        for _ in range(2):
            graph.replay()
        for t, a in zip((j, m), alone):
            assert torch.equal(unique(ctx, t), unique(ctx, a) + unique(ctx, a))
        del graph
        ctx.close()


def test_two_contexts_on_two_streams_into_the_same_buffers(torch_cuda):
    """The scalar form's atomic additions of depositions that run at the same time."""
    import torch
    g, ctx, bn = setting(0, (23, 21, 20))
    _, other, _ = setting(0, (23, 21, 20))
    first, second = Species(ctx, g, 0, 0), Species(ctx, g, 1, 0)
    alone = [ctx.moments() for _ in range(2)]
    for s, a in zip((first, second), alone):
        s.into(ctx, bn, *a, 0)
    streams = [torch.cuda.Stream() for _ in range(2)]
    ctx.stream, other.stream = (C.c_void_p(s.cuda_stream) for s in streams)
    j, m = ctx.moments()
    torch.cuda.synchronize()
    rounds = 8
    for _ in range(rounds):
        first.into(ctx, bn, j, m, 0)
        second.into(other, bn, j, m, 0)
    torch.cuda.synchronize()
    for t, a, b in zip((j, m), *alone):
        want = rounds * (a + b)
        # Sixteen additions of the two sums in any order: 16 eps of their magnitudes.
        assert float((t - want).abs().max()) <= 16 * 2.0**-52 * rounds * float((a.abs() + b.abs()).max())
    ctx.close()
    other.close()
