"""kd_coef_host_noalloc is for code between an application's steps: a call costs
about what kd_coef_host costs, and nothing is compiled or sorted again for a
shape met before."""
import ctypes as C
import time

import numpy as np
import pytest

from tests.test_zz_no_alloc import _declare, _desc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,shape", [("nucleus", (13, 9, 4)), ("shell", (21, 11, 14))])
def test_call_costs_about_what_the_allocating_one_does(ctx, kind, shape):
    _declare(ctx.lib)
    nc = (shape[0], shape[1], shape[2] + 2)
    x, y = np.random.default_rng(0).standard_normal((1,) + shape), np.zeros((1,) + nc)
    d, keep = _desc(kind, shape, 1, x, y)
    best = []
    for fn in (ctx.lib.kd_coef_host, ctx.lib.kd_coef_host_noalloc):
        times = []
        for _ in range(300):
            t = time.perf_counter()
            ctx.check(fn(ctx.h, C.byref(d)))
            times.append(time.perf_counter() - t)
        best.append(np.median(times[50:]))
    # one more small copy and, per line, the matrix's zeros: less than as much again
    assert best[1] <= 2.0 * best[0], best
