"""A one-dimensional operator's bases, asked for without fields, whatever the size."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

CHEB, COSSIN, COS_EVEN = 1, 4, 6
DER = 2  # KD_OP_DER


def _desc(nc):
    from kadath_frontera_gb300._lib import TransformDesc
    r, t = (C.c_int * (nc[1] * nc[2]))(*[CHEB] * (nc[1] * nc[2])), (C.c_int * nc[2])(*[COS_EVEN] * nc[2])
    d = TransformDesc()
    d.nbr_points[:] = d.nbr_coefs[:] = nc
    d.base_r, d.base_t, d.base_p = C.cast(r, C.POINTER(C.c_int)), C.cast(t, C.POINTER(C.c_int)), COSSIN
    d.batch = 0
    return d, (r, t)


def _der(ctx, d, nc):
    p, r, t = C.c_int(), (C.c_int * (nc[1] * nc[2]))(), (C.c_int * nc[2])()
    ctx.check(ctx.lib.kd_ope_1d(ctx.h, DER, 0, C.byref(d), r, t, C.byref(p)))
    return list(r), list(t), p.value


@pytest.mark.parametrize("nc", [(9, 5, 6), (61, 33, 18)])
def test_bases_without_fields(ctx, nc):
    """No fields, so nothing has to fit an SM's shared memory."""
    d, keep = _desc(nc)
    assert _der(ctx, d, nc) == ([CHEB] * (nc[1] * nc[2]), [COS_EVEN] * nc[2], COSSIN)
