"""Infinities and NaN in the line passes: an output is a sum over its whole line,
the matrix's zeros included, so a non-finite entry makes every output of the
lines it lies on non-finite (0 * Inf is NaN), in the slots of basis functions
that vanish on the grid and under the zeros of a triangular operator too."""
import ctypes as C

import numpy as np
import pytest

from tests.spectral_cases import std_base

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _desc(kind, shape, batch, x, y):
    from kadath_frontera_gb300._lib import TransformDesc
    nc = (shape[0], shape[1], shape[2] + 2)
    br, bt, bp = std_base(kind, nc[1], nc[2])
    r = (C.c_int * (nc[1] * nc[2]))(*[b for row in br for b in row])
    t = (C.c_int * nc[2])(*bt)
    d = TransformDesc()
    d.nbr_points[:], d.nbr_coefs[:] = shape, nc
    d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), bp
    d.batch, d.in_, d.out = batch, x.data_ptr(), y.data_ptr()
    return d, (r, t)


def _apply(ctx, fn, kind, shape, src, out_shape):
    x = torch.tensor(src, device="cuda")
    y = torch.full((len(src),) + out_shape, 7.0, device="cuda", dtype=torch.float64)
    d, keep = _desc(kind, shape, len(src), x, y)
    torch.cuda.synchronize()
    ctx.check(fn(ctx, d))
    ctx.synchronize()
    return y.cpu().numpy()


@pytest.mark.parametrize("kind", ["nucleus", "shell"])
@pytest.mark.parametrize("shape,batch", [((9, 5, 4), 1), ((9, 5, 4), 40), ((21, 11, 14), 3), ((21, 11, 14), 90)])
@pytest.mark.parametrize("junk", [np.nan, np.inf])
def test_transforms(ctx, kind, shape, batch, junk):
    nc = (shape[0], shape[1], shape[2] + 2)
    rng = np.random.default_rng(batch)
    at = batch // 2
    others = np.arange(batch) != at
    for inverse in (False, True):
        i_shape, o_shape = (nc, shape) if inverse else (shape, nc)
        name = "kd_coef_i_many" if inverse else "kd_coef_many"
        fn = lambda c, d: getattr(c.lib, name)(c.h, 1, C.byref(d))  # noqa: E731
        src = rng.standard_normal((batch,) + i_shape)
        clean = _apply(ctx, fn, kind, shape, src, o_shape)
        places = [(0, 0, 0), (shape[0] - 1, 2, 3)] + ([(3, 1, 1), (2, 0, nc[2] - 1)] if inverse else [])
        for place in places:
            bad = src.copy()
            bad[(at,) + place] = junk
            got = _apply(ctx, fn, kind, shape, bad, o_shape)
            assert not np.isfinite(got[at]).any()
            # the other fields do not notice
            assert np.array_equal(got[others], clean[others])


@pytest.mark.parametrize("shape,batch", [((9, 5, 4), 1), ((13, 9, 4), 60)])
@pytest.mark.parametrize("junk", [np.nan, np.inf])
def test_derivative_along_r(ctx, shape, batch, junk):
    """The radial derivative of Chebyshev coefficients: a triangular matrix with
    a parity, on the line of one (theta, phi)."""
    nc = (shape[0], shape[1], shape[2] + 2)
    src = np.random.default_rng(1).standard_normal((batch,) + nc)

    def fn(c, d):
        p = C.c_int()
        r, t = (C.c_int * (nc[1] * nc[2]))(), (C.c_int * nc[2])()
        return c.lib.kd_ope_1d(c.h, 2, 0, C.byref(d), r, t, C.byref(p))  # KD_OP_DER
    clean = _apply(ctx, fn, "shell", shape, src, nc)
    bad = src.copy()
    bad[batch - 1, 0, 2, 3] = junk  # T_0, whose derivative is zero
    got = _apply(ctx, fn, "shell", shape, bad, nc)
    line = np.zeros((batch,) + nc, bool)
    line[batch - 1, :, 2, 3] = True
    assert not np.isfinite(got[line]).any()
    # (the sums of the others may take the zeros of the matrix along)
    assert np.abs(got[~line] - clean[~line]).max() <= 1e-13 * np.abs(clean).max()


def test_collected_passes(ctx):
    """A NaN among the values of one domain: the same rows of the residual are
    NaN whether the pass is collected into levels or launched one by one, and the
    Newton step is refused."""
    from kadath_frontera_gb300 import KadathError, workloads
    from kadath_frontera_gb300.kadath import profile_enable
    wl = workloads.star(res=(9, 5, 4), ctx=ctx)
    wl.syst.sec_member()
    f = wl.unknowns[0][1]
    v = f.get_domain(1)
    v[3, 2, 1] = np.nan
    f.set_domain(1, v)
    collected = np.isnan(wl.syst.sec_member())
    profile_enable(ctx, True)
    try:
        single = np.isnan(wl.syst.sec_member())
    finally:
        profile_enable(ctx, False)
    assert collected.sum() > 9 * 5 * 4 and np.array_equal(collected, single)
    with pytest.raises(KadathError):
        wl.syst.do_newton(1e-10)
