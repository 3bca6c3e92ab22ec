"""Two contexts on two host threads, transforming fields of different sizes whose
stages need more than 48 KB of shared memory: each call succeeds and gives what
it gives alone."""
import ctypes as C
import threading

import numpy as np
import pytest

from tests.spectral_cases import std_base

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _call(ctx, shape, batch, seed):
    from kadath_frontera_gb300._lib import TransformDesc
    nc = (shape[0], shape[1], shape[2] + 2)
    br, bt, bp = std_base("nucleus", nc[1], nc[2])
    x = torch.randn((batch,) + shape, device="cuda", dtype=torch.float64,
                    generator=torch.Generator(device="cuda").manual_seed(seed))
    y = torch.zeros((batch,) + nc, device="cuda", dtype=torch.float64)
    r = (C.c_int * (nc[1] * nc[2]))(*[b for row in br for b in row])
    t = (C.c_int * nc[2])(*bt)
    d = TransformDesc()
    d.nbr_points[:], d.nbr_coefs[:] = shape, nc
    d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), bp
    d.batch, d.in_, d.out = batch, x.data_ptr(), y.data_ptr()
    keep = (x, y, r, t, d)
    torch.cuda.synchronize()
    return keep, lambda: ctx.lib.kd_coef_many(ctx.h, 1, C.byref(d))


@pytest.mark.parametrize("batch", [2, 100])
def test_two_threads(batch):
    from kadath_frontera_gb300._lib import Context
    sizes = [(25, 13, 14), (21, 11, 8)]
    ctxs = [Context(0) for _ in sizes]
    calls = [_call(c, s, batch, q) for q, (c, s) in enumerate(zip(ctxs, sizes))]
    alone = []
    for c, (keep, call) in zip(ctxs, calls):
        assert call() == 0
        c.synchronize()
        alone.append(keep[1].clone())
    failed = [0, 0]
    go = threading.Barrier(2)

    def loop(q):
        go.wait()
        for _ in range(3000):
            failed[q] += calls[q][1]() != 0

    threads = [threading.Thread(target=loop, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.synchronize()
    assert failed == [0, 0]
    for (keep, _), ref in zip(calls, alone):
        assert torch.equal(keep[1], ref)
    assert np.isfinite(alone[0].cpu().numpy()).all()
