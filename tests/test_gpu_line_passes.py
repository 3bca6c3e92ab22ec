"""Line passes where their lists change form: transforms of few fields (plain
matrices) and of many (mirrored entries combined), even and odd line lengths
(a middle entry or none), fields too large for a padded stage or for matrices
beside the stages, and the zero lines of the phi basis."""
import ctypes as C

import numpy as np
import pytest

from oracle import spectral as S
from tests.spectral_cases import std_base

pytestmark = pytest.mark.gpu


def _many(ctx, kind, shape, batch, inverse, seed, anti=False):
    import torch

    from kadath_frontera_gb300._lib import TransformDesc
    nr, nt, np_ = shape
    nc = (nr, nt, np_ + 2)
    br, bt, bp = std_base(kind, nt, nc[2], anti)
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((batch,) + shape)
    if inverse:  # coefficients of real fields: what the forward transform gives
        ref_in = np.stack([S.coef_3d(x, br, bt, bp, nc) for x in v[:2]])
        src = np.concatenate([ref_in, np.repeat(ref_in[:1], batch - 2, 0)]) if batch > 2 else ref_in[:batch]
        ref = [S.coef_i_3d(x, br, bt, bp, shape) for x in src[:2]]
    else:
        src, ref = v, [S.coef_3d(x, br, bt, bp, nc) for x in v[:2]]
    x = torch.tensor(src, device="cuda")
    y = torch.full((batch,) + (shape if inverse else nc), 7.0, device="cuda", dtype=torch.float64)
    r = (C.c_int * (nt * nc[2]))(*[b for row in br for b in row])
    t = (C.c_int * nc[2])(*bt)
    d = TransformDesc()
    d.nbr_points[:] = shape
    d.nbr_coefs[:] = nc
    d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), bp
    d.batch, d.in_, d.out = batch, x.data_ptr(), y.data_ptr()
    torch.cuda.synchronize()
    ctx.check((ctx.lib.kd_coef_i_many if inverse else ctx.lib.kd_coef_many)(ctx.h, 1, C.byref(d)))
    ctx.synchronize()
    return y.cpu().numpy(), ref


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("kind,anti", [("nucleus", False), ("shell", False), ("shell", True)])
@pytest.mark.parametrize("shape,batch", [((5, 3, 4), 1), ((9, 5, 4), 32), ((9, 5, 4), 33), ((13, 9, 4), 40),
                                         ((11, 7, 6), 100), ((9, 5, 14), 77), ((21, 11, 14), 33), ((25, 13, 14), 2)])
def test_transforms_of_few_and_many_fields(ctx, kind, anti, shape, batch, inverse):
    got, ref = _many(ctx, kind, shape, batch, inverse, 3, anti)
    for g, o in zip(got, ref):
        # three passes of at most 25-term sums of O(1) matrices: the parity
        # bound of the transforms, 1e-13 relative
        assert np.linalg.norm(g - o) <= 1e-13 * np.linalg.norm(o)


@pytest.mark.parametrize("shape,batch", [((33, 17, 20), 1), ((33, 17, 24), 40)])
def test_fields_that_fill_shared_memory(ctx, shape, batch):
    """33 x 17 x 22 coefficients pad to a stage of 12,903 doubles (the matrices
    find no room beside two of them); 33 x 17 x 26 do not fit and are refused."""
    if shape[2] == 20:
        got, ref = _many(ctx, "shell", shape, batch, False, 4)
        for g, o in zip(got, ref):
            assert np.linalg.norm(g - o) <= 1e-13 * np.linalg.norm(o)
    else:
        from kadath_frontera_gb300 import KadathError
        with pytest.raises(KadathError):
            _many(ctx, "shell", shape, batch, False, 4)


def test_coefficients_without_collocation_values_are_ignored(ctx):
    """sin(0) and the sine at the highest frequency vanish on the grid: what
    their slots hold does not reach the values."""
    import torch

    from kadath_frontera_gb300._lib import TransformDesc
    shape, nc, batch = (9, 5, 4), (9, 5, 6), 3
    br, bt, bp = std_base("shell", 5, 6)
    c = np.random.default_rng(0).standard_normal((batch,) + nc)
    out = []
    for junk in (0.0, 5.0):
        c[..., 1] = c[..., 5] = junk
        x, y = torch.tensor(c, device="cuda"), torch.zeros((batch,) + shape, device="cuda", dtype=torch.float64)
        r = (C.c_int * 30)(*[b for row in br for b in row])
        t = (C.c_int * 6)(*bt)
        d = TransformDesc()
        d.nbr_points[:], d.nbr_coefs[:] = shape, nc
        d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), bp
        d.batch, d.in_, d.out = batch, x.data_ptr(), y.data_ptr()
        torch.cuda.synchronize()
        ctx.check(ctx.lib.kd_coef_i_many(ctx.h, 1, C.byref(d)))
        ctx.synchronize()
        out.append(y.cpu().numpy())
    assert np.array_equal(out[0], out[1])
