"""A regrid runs each domain's passes once: it compiles nothing for them, so it
costs about what one transform a domain costs."""
import ctypes as C
import time

import numpy as np
import pytest

from tests.test_zz_no_alloc import _desc

pytestmark = pytest.mark.gpu


def _median(fn, n=60):
    times = []
    for _ in range(n):
        t = time.perf_counter()
        fn()
        times.append(time.perf_counter() - t)
    return np.median(times[n // 4:])


@pytest.mark.parametrize("old,new", [((13, 9, 4), (21, 11, 14))])
def test_regrid_costs_a_transform_a_domain(ctx, old, new):
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Scalar, Space_spheric
    bounds = (3.5, 7.0, 12.0)
    coarse, fine = (Space_spheric(CHEB_TYPE, (0, 0, 0), r, bounds, ctx=ctx) for r in (old, new))
    f, g = Scalar(coarse), Scalar(fine)
    for d in range(4):
        r = coarse.get_radius(d)
        f.set_domain(d, np.where(np.isfinite(r), 1.0 / (1.0 + np.where(np.isfinite(r), r, 0.0) ** 2), 0.0))
    f.std_base()
    x, y = np.zeros((1,) + new), np.zeros((1, new[0], new[1], new[2] + 2))
    desc, keep = _desc("shell", new, 1, x, y)
    one = _median(lambda: ctx.check(ctx.lib.kd_coef_host(ctx.h, C.byref(desc))))
    # (a regrid's four domains are transformed and evaluated on the device alone)
    assert _median(lambda: g.regrid_from(f)) <= 1.5 * 4 * one
