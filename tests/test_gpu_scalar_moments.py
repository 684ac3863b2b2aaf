"""The scalar mass forms' deposition of sorted records through per-cell moments,
at the sizes where its kernels change path: empty cells, counts around the
32-record chunks and the 4-record steps, cells whose two species share a chunk,
one to three species, grids taken cell by cell and in batches of four cells
with a partial last batch, rows that are and are not multiples of 4; invalid
and nonfinite records; and the calls that keep the per-cell atomics.

Bound: a node's value is a sum of at most 8 cells' n records of the form's
arithmetic, each product within a few roundings: (n + 40) eps of the sum of
the terms' magnitudes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from fieldutil import interior_nodes, interior_records, periodic_node_field, smooth_random_unique
from reference_fixtures import oracle_moments
from tpic_b200 import _lib
from tpic_b200.plasma import GridSpec

pytestmark = pytest.mark.gpu

COUNTS = np.array([0, 1, 2, 3, 4, 5, 31, 32, 33, 35, 63, 64, 65, 0, 97, 130])
QOM = (-4.0, 1.0, -1.0)


def ragged_species(g, s, rng, precision, scale):
    cells = g.nx * g.ny * g.nz
    per = (COUNTS[(np.arange(cells) * (3 + 2 * s) + s) % len(COUNTS)] / scale).astype(int)
    lin = np.repeat(np.arange(cells), per)
    n = len(lin)
    vt = np.float64 if precision == 0 else np.float32
    d = {k: rng.random(n) for k in ("rx", "ry", "rz")}
    d.update({k: (0.2 * rng.normal(size=n)).astype(vt) for k in ("u", "v", "w")})
    d["q"] = np.sign(QOM[s]) * (0.5 + rng.random(n)) * 1e-3
    d["cell"] = g.encode(lin % g.nx, (lin // g.nx) % g.ny, lin // (g.nx * g.ny)).astype(np.int32)
    return d


def bins(ctx, d):
    import torch
    counts = np.bincount(d["cell"], minlength=ctx.layout.bin_count)
    offsets = np.concatenate([[0], np.cumsum(counts)])
    return torch.from_numpy(counts.astype(np.int32)).cuda(), torch.from_numpy(offsets.astype(np.int32)).cuda()


def check(g, ctx, j, m, want, size, precision, records):
    rel = (records + 40) * (2.0**-53 if precision == 0 else 2.0**-24)
    jg, mg = j.cpu().numpy().astype(np.float64), ctx.records(m)
    for got, w, a, pick in ((jg, want[0], size[0], interior_nodes), (mg, want[1], size[1], interior_records)):
        assert np.abs(pick(g, got) - pick(g, w)).max() <= rel * np.abs(pick(g, a)).max()


@pytest.mark.parametrize("shape", [(5, 3, 2), (8, 3, 1), (23, 21, 20)], ids=["5x3x2", "8x3x1", "23x21x20"])
@pytest.mark.parametrize("nspecies", [1, 2, 3])
@pytest.mark.parametrize("precision,kind", [(0, 0), (1, 0), (1, 1)])
def test_ragged_cells_match_the_oracle(torch_cuda, shape, nspecies, precision, kind):
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    rng = np.random.default_rng(nspecies)
    scale = 1 if np.prod(shape) < 1000 else 4
    ctx = StageContext(g, precision=precision, dt=0.2, mass_layout=1)
    bnode = periodic_node_field(g, smooth_random_unique(g, rng, 0.9)).astype(ctx.np_fdt)
    bn = ctx.field(bnode)
    j, m = ctx.moments()
    keep, structs, want, size = [], [], [0.0, 0.0], [0.0, 0.0]
    bad_records = 0
    for s in range(nspecies):
        d = ragged_species(g, s, rng, precision, scale)
        n = len(d["cell"])
        if s == 0:  # out of range and nonfinite: counted, nothing deposited
            d["rx"][n // 2], d["q"][n // 3], d["q"][n // 4] = 1.25, np.nan, np.inf
        good = (d["rx"] < 1) & np.isfinite(d["q"])
        bad_records += int(np.count_nonzero(~good))
        parts = ctx.upload_particles(d)
        keep.append((parts, *bins(ctx, d)))
        structs.append(ctx.struct(parts, n))
        kept = {k: np.ascontiguousarray(v[good]) for k, v in d.items()}
        js, ms, _ = oracle_moments(g, precision, QOM[s], 0.2, kept, bnode)
        ja, ma, _ = oracle_moments(g, precision, QOM[s], 0.2,
                                   {**kept, **{k: np.abs(kept[k]) for k in ("u", "v", "w", "q")}}, bnode)
        for total, values in ((want, (js, ms)), (size, (np.abs(ja), np.abs(ma)))):
            total[0], total[1] = total[0] + values[0], total[1] + values[1]
    arrays = ((C.c_double * nspecies)(*QOM[:nspecies]), (_lib.Particles * nspecies)(*structs),
              (C.c_void_p * nspecies)(*[k[1].data_ptr() for k in keep]),
              (C.c_void_p * nspecies)(*[k[2].data_ptr() for k in keep]))

    def deposit():
        _lib.check(ctx.lib.tpicb200_deposit_species(ctx.ctx, nspecies, *arrays, bn.data_ptr(), j.data_ptr(),
                                                    m.data_ptr(), kind, ctx.invalid.data_ptr(), ctx.stream))

    records = int(8 * COUNTS.max() * nspecies / scale)
    # A second deposition adds.
    _lib.check(ctx.lib.tpicb200_clear_moments(ctx.ctx, j.data_ptr(), m.data_ptr(), ctx.stream))
    deposit()
    ctx.fold(j, m)
    assert ctx.invalid_count() == bad_records
    check(g, ctx, j, m, want, size, precision, records)
    deposit()
    ctx.fold(j, m)
    check(g, ctx, j, m, [2 * w for w in want], [2 * a for a in size], precision, records)
    # J or the mass alone: the per-cell atomics.
    alone = ctx.moments()
    for s in range(nspecies):
        ctx.deposit(QOM[s], keep[s][0], structs[s].count, bn, alone[0], None, keep[s][1], keep[s][2], kind=kind)
        ctx.deposit(QOM[s], keep[s][0], structs[s].count, bn, None, alone[1], keep[s][1], keep[s][2], kind=kind)
    ctx.fold(*alone)
    check(g, ctx, alone[0], alone[1], want, size, precision, records)
    ctx.close()


def test_scalar_deposition_leaves_waiting_moments_alone(torch_cuda):
    """A scalar deposition between a tensor-core one and its fold: both in J and the mass after it."""
    from gpu_helpers import StageContext
    g = GridSpec(8, 6, 4, 0.8, 0.6, 0.4)
    rng = np.random.default_rng(7)
    ctx = StageContext(g, precision=1, dt=0.2, mass_layout=1)
    bnode = periodic_node_field(g, smooth_random_unique(g, rng, 0.9)).astype(np.float32)
    bn = ctx.field(bnode)
    j, m = ctx.moments()
    jw = mw = 0.0
    for s, kind in ((0, 3), (1, 0)):
        d = ragged_species(g, s, rng, 1, 1)
        parts = ctx.upload_particles(d)
        counts, offsets = bins(ctx, d)
        ctx.deposit(QOM[s], parts, len(d["cell"]), bn, j, m, counts, offsets, kind=kind)
        js, ms, _ = oracle_moments(g, 1, QOM[s], 0.2, d, bnode)
        jw, mw = jw + js, mw + ms
    ctx.fold(j, m)
    assert ctx.invalid_count() == 0
    jg, mg = j.cpu().numpy().astype(np.float64), ctx.records(m)
    assert np.abs(interior_nodes(g, jg) - interior_nodes(g, jw)).max() <= 1e-4 * np.abs(interior_nodes(g, jw)).max()
    assert np.abs(interior_records(g, mg) - interior_records(g, mw)).max() <= 1e-4 * np.abs(mw).max()


@pytest.mark.parametrize("shape,per_cell", [((12, 12, 12), 48), ((16, 16, 16), 16), ((16, 16, 16), 1), ((21, 20, 20), 1)])
@pytest.mark.parametrize("precision,kind", [(0, 0), (1, 0), (1, 1)])
def test_both_sides_of_the_rule_agree(torch_cuda, shape, per_cell, precision, kind):
    """With one record less than the rule asks for the cell-tile kernel runs (one launch), else the moments
    (two): the same deposition within the sums' rounding."""
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(0.1 * n for n in shape))
    cells = g.nx * g.ny * g.nz
    rng = np.random.default_rng(per_cell)
    ctx = StageContext(g, precision=precision, dt=0.2, mass_layout=1)
    bn = ctx.field(periodic_node_field(g, smooth_random_unique(g, rng, 0.9)))
    fp32 = precision == 1 and kind == 0
    least = 48 if cells < 148 * 16 else 16 if fp32 and cells < 8192 else 1
    vt = np.float64 if precision == 0 else np.float32
    n = per_cell * cells
    lin = np.arange(n) // per_cell
    d = {k: rng.random(n) for k in ("rx", "ry", "rz")}
    d.update({k: np.abs(0.2 * rng.normal(size=n)).astype(vt) for k in ("u", "v", "w")})
    d["q"] = 1e-3 * (0.5 + rng.random(n))
    d["cell"] = g.encode(lin % g.nx, (lin // g.nx) % g.ny, lin // (g.nx * g.ny)).astype(np.int32)
    results = []
    for count in (n, n - 1):
        e = {k: v[:count] for k, v in d.items()}
        if count == n:  # the last record deposits nothing, so that both calls deposit the same
            e = {**e, "q": e["q"].copy()}
            e["q"][-1] = 0.0
        parts = ctx.upload_particles(e)
        counts, offsets = bins(ctx, e)
        j, m = ctx.moments()
        before = ctx.lib.tpicb200_launch_count()
        ctx.deposit(-1.0, parts, count, bn, j, m, counts, offsets, kind=kind)
        assert ctx.lib.tpicb200_launch_count() - before == (2 if count >= least * cells else 1)
        results.append((j.double(), m.double()))
    assert ctx.invalid_count() == 0
    # Sums of 8 cells' records, each term within a few roundings, of terms up to the largest entry's size.
    rel = (8 * per_cell + 40) * (2.0**-53 if precision == 0 else 2.0**-24)
    for a, b in zip(*results):
        assert float((a - b).abs().max()) <= rel * float(b.abs().max())
    ctx.close()
