"""The launch shape that line passes take by themselves is about as fast as the
best of all shapes, at the ends of the rule's ranges."""
import ctypes as C
import json
import time

import pytest

from tests.spectral_cases import std_base

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _desc(shape, batch):
    from kadath_frontera_gb300._lib import TransformDesc
    nc = (shape[0], shape[1], shape[2] + 2)
    br, bt, bp = std_base("shell", nc[1], nc[2])
    r = (C.c_int * (nc[1] * nc[2]))(*[b for row in br for b in row])
    t = (C.c_int * nc[2])(*bt)
    x = torch.randn((batch,) + nc, device="cuda", dtype=torch.float64)
    y = torch.empty((batch,) + shape, device="cuda", dtype=torch.float64)
    d = TransformDesc()
    d.nbr_points[:], d.nbr_coefs[:] = shape, nc
    d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), bp
    d.batch, d.in_, d.out = batch, x.data_ptr(), y.data_ptr()
    return d, (r, t, x, y)


def _time(fn, ctx):
    for _ in range(5):
        fn()
    best = float("inf")
    for _ in range(7):
        ctx.synchronize()
        t = time.perf_counter()
        for _ in range(30):
            fn()
        ctx.synchronize()
        best = min(best, (time.perf_counter() - t) / 30)
    return best


@pytest.mark.parametrize("shape,batch", [((33, 17, 16), 8), ((33, 17, 16), 9), ((33, 17, 16), 12), ((21, 11, 14), 12),
                                         ((33, 17, 16), 16), ((13, 9, 4), 32), ((5, 5, 4), 300), ((5, 5, 4), 1200),
                                         ((5, 5, 4), 3600), ((9, 5, 4), 3600), ((13, 9, 4), 300)])
def test_rule(ctx, tmp_path, shape, batch):
    d, keep = _desc(shape, batch)
    table = tmp_path / "table.json"

    def fn():
        ctx.check(ctx.lib.kd_coef_i_many(ctx.h, 1, C.byref(d)))
    try:
        ctx.autotune(None, mode=0)
        rule = _time(fn, ctx)
        ctx.autotune(table, mode=2)
        fn()
        keys = list(json.loads(table.read_text())["line_passes"])
        best = float("inf")
        for cluster, threads in ([(8, 128), (4, 128)] if batch <= 64 else []) + [(1, 128), (1, 256)]:
            table.write_text(json.dumps({"line_passes": {k: {"cluster": cluster, "threads": threads, "us": 1.0}
                                                         for k in keys}}))
            ctx.autotune(table, mode=1)
            best = min(best, _time(fn, ctx))
    finally:
        ctx.autotune(None, mode=0)
    # (launches come in steps of 2 us)
    assert rule <= 1.1 * best + 1.5e-6, (rule, best)
