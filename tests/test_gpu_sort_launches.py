"""The binned sort's cooperative kernels: the plan (counts, scan, bases) on grids
of one CTA to several tiles of the scan a CTA, and the fallback sort, on one context
one after the other (each must leave the flags and the barrier as it found
them): neighbour moves, far moves, bins that do not describe the records, an
invalid key, bins of one record to several merge passes of all CTAs;
and both recorded in a CUDA graph. Against a stable sort on the host, bit for
bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tpic_b200 import _lib
from tpic_b200.plasma import GridSpec

pytestmark = pytest.mark.gpu


def records(g, n, rng, precision, heavy):
    c = [rng.integers(0, m, n) for m in (g.nx, g.ny, g.nz)]
    if heavy:  # most records in one cell
        crowd = rng.random(n) < 0.8
        for a in range(3):
            c[a][crowd] = 0
    vt = np.float64 if precision == 0 else np.float32
    d = {k: rng.random(n) for k in ("rx", "ry", "rz", "q")}
    d.update({k: rng.normal(size=n).astype(vt) for k in ("u", "v", "w")})
    d["cell"] = np.sort(g.encode(*c)).astype(np.int32)
    d["id"] = np.arange(n, dtype=np.uint64)
    return d


def bins_of(g, key):
    counts = np.bincount(key, minlength=(g.nx + 4) * (g.ny + 4) * (g.nz + 4))
    return counts.astype(np.int32), np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)


def moved(g, key, rng, far):
    ex, ey = g.nx + 4, g.ny + 4
    k = key.astype(np.int64)
    c = [k % ex - 2, (k // ex) % ey - 2, k // (ex * ey) - 2]
    step = [rng.integers(-1, 2, len(k)) for _ in range(3)]
    if far:
        step[0][rng.random(len(k)) < 0.01] = 2
    return g.encode(*((a + s) % m for a, s, m in zip(c, step, (g.nx, g.ny, g.nz)))).astype(np.int32)


def check(g, src, out, counts, offsets, n):
    order = np.argsort(src["cell"], kind="stable")
    want_counts, want_offsets = bins_of(g, src["cell"])
    assert np.array_equal(counts.cpu().numpy(), want_counts)
    assert np.array_equal(offsets.cpu().numpy(), want_offsets)
    for k, v in src.items():
        got = out[k][:n].cpu().numpy()
        assert np.array_equal(got.view(v.dtype) if k == "id" else got, v[order]), k


@pytest.mark.parametrize("shape,n,heavy", [((4, 3, 1), 1, False), ((4, 3, 1), 37, False), ((9, 8, 7), 20000, False),
                                           ((9, 8, 7), 30000, True), ((61, 1, 1), 4000, True),
                                           ((60, 52, 51), 30000, False), ((70, 52, 50), 30000, False)])
@pytest.mark.parametrize("precision", [0, 1])
def test_binned_sorts_in_a_row(torch_cuda, shape, n, heavy, precision):
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(*shape, *(1.0 * m for m in shape))
    rng = np.random.default_rng(n)
    ctx = StageContext(g, precision=precision, max_particles=n)
    for far, wrong_bins in ((False, False), (True, False), (False, True), (False, False), (True, True), (False, False)):
        d = records(g, n, rng, precision, heavy)
        counts, offsets = (torch.from_numpy(a).cuda() for a in bins_of(g, d["cell"]))
        if wrong_bins:
            counts[int(d["cell"][0])] -= 1
        d["cell"] = moved(g, d["cell"], rng, far)
        src = ctx.upload_particles(d)
        out, c, o = ctx.sort_binned(src, n, counts, offsets, alias=far)
        assert ctx.invalid_count() == 0
        check(g, d, out, c, o, n)
    # An invalid key stops the sort and is counted; the next sort works.
    d = records(g, n, rng, precision, heavy)
    counts, offsets = (torch.from_numpy(a).cuda() for a in bins_of(g, d["cell"]))
    bad = dict(d, cell=d["cell"].copy())
    bad["cell"][n // 2] = -7
    ctx.sort_binned(ctx.upload_particles(bad), n, counts, offsets)
    assert ctx.invalid_count() == 1
    d["cell"] = moved(g, d["cell"], rng, False)
    out, c, o = ctx.sort_binned(ctx.upload_particles(d), n, counts, offsets)
    check(g, d, out, c, o, n)
    ctx.close()


@pytest.mark.parametrize("cells", [(8192,), (8193,), (16384, 300), (16385, 8192, 257, 256, 1), (0, 70000, 33000, 8200, 12),
                                   (32769, 9000, 65536, 20000), (300,) * 700], ids=lambda c: f"{c[0]}of{len(c)}")
def test_fallback_of_crowded_cells(torch_cuda, cells):
    """Bins on both sides of what a warp, a block and the merge passes of all blocks take, of several pass
    counts in one sort, scrambled by a far move."""
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(len(cells), 1, 1, 1.0 * len(cells), 1.0, 1.0)
    rng = np.random.default_rng(len(cells))
    n = int(sum(cells))
    d = records(g, n, rng, 1, False)
    d["cell"] = np.sort(d["cell"])  # the old cells: evenly
    counts, offsets = (torch.from_numpy(a).cuda() for a in bins_of(g, d["cell"]))
    counts[int(d["cell"][0])] -= 1  # bins that do not describe the records
    d["cell"] = rng.permutation(np.repeat(g.encode(np.arange(len(cells)), 0, 0), cells)).astype(np.int32)
    ctx = StageContext(g, precision=1, max_particles=n)
    for _ in range(2):
        out, c, o = ctx.sort_binned(ctx.upload_particles(d), n, counts, offsets)
        assert ctx.invalid_count() == 0
        check(g, d, out, c, o, n)
    ctx.close()


def test_binned_sort_in_a_graph(torch_cuda):
    import torch
    from gpu_helpers import StageContext
    g = GridSpec(9, 8, 7, 9.0, 8.0, 7.0)
    n = 20000
    rng = np.random.default_rng(3)
    d = records(g, n, rng, 1, False)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = StageContext(g, precision=1, max_particles=n)
        counts, offsets = (torch.from_numpy(a).cuda() for a in bins_of(g, d["cell"]))
        src, dst = ctx.upload_particles(d), ctx.empty_particles(n, True)
        c, o = torch.zeros_like(counts), torch.zeros_like(offsets)
        pin, pout = ctx.struct(src, n), ctx.struct(dst, n)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            _lib.check(ctx.lib.tpicb200_sort_binned(ctx.ctx, C.byref(pin), counts.data_ptr(), offsets.data_ptr(),
                                                    C.byref(pout), c.data_ptr(), o.data_ptr(),
                                                    ctx.invalid.data_ptr(), ctx.stream))
        key = d["cell"]
        for far in (False, True, False):
            d["cell"] = moved(g, key, rng, far)
            src["cell"].copy_(torch.from_numpy(d["cell"]))
            graph.replay()
            assert ctx.invalid_count() == 0
            check(g, d, dst, c, o, n)
        del graph
        ctx.close()
