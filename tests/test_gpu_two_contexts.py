"""Two contexts on two streams from two host threads: their cooperative kernels (resident solves that fill the
device, the sort's plan and general sort) run beside each other, and every result is the one a context alone gives."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

from test_gpu_resident_solve import system
from test_gpu_sort_launches import bins_of, check, moved, records
from tpic_b200.plasma import GridSpec

pytestmark = pytest.mark.gpu


def test_cooperative_kernels_of_two_contexts_at_once(torch_cuda):
    import torch
    from gpu_helpers import StageContext
    failures = []
    results = {}

    def work(k, shape, go):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                rng = np.random.default_rng(k)
                g = GridSpec(*shape, *(0.1 * n for n in shape))
                n = 60000
                ctx = StageContext(g, precision=0, dt=0.1, tol=1e-10, mass_layout=1, restart=20, max_iterations=300,
                                   max_particles=n)
                ctx.stream = C.c_void_p(stream.cuda_stream)
                inputs = system(ctx, g, rng)
                d = records(g, n, rng, 0, False)
                counts, offsets = (torch.from_numpy(a).cuda() for a in bins_of(g, d["cell"]))
                near, far = (dict(d, cell=moved(g, d["cell"], rng, f)) for f in (False, True))
                uploaded = [(x, ctx.upload_particles(x)) for x in (near, far)]
                want, _ = ctx.field_solve(*inputs)
                stream.synchronize()
                go.wait()
                for _ in range(40):
                    got, res = ctx.field_solve(*inputs)
                    outs = [(x, *ctx.sort_binned(src, n, counts, offsets)) for x, src in uploaded]
                stream.synchronize()
                results[k] = (torch.equal(got, want), bool(res.converged), int(ctx.invalid.item()))
                for x, out, c, o in outs:
                    check(g, x, out, c, o, n)
                ctx.close()
        except Exception as e:  # noqa: BLE001
            failures.append((k, repr(e)))
            go.abort()

    go = threading.Barrier(2)
    threads = [threading.Thread(target=work, args=(k, s, go)) for k, s in enumerate([(48, 44, 40), (36, 40, 41)])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    assert results == {0: (True, True, 0), 1: (True, True, 0)}
