"""Point evaluation where its kernels change: few points (eight lanes each), the
number that switches to grouped chunks, fields with different bases and zero
fields in one call, a resolution whose tables do not fit, points at infinity,
on the axis and in no domain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(space, n):
    from kadath_frontera_gb300.kadath import Scalar
    out = []
    for q in range(n):
        f = Scalar(space)
        for d in range(space.get_nbr_domains()):
            x, y, z = (space.get_cart(d, c) for c in (1, 2, 3))
            r = space.get_radius(d)
            with np.errstate(invalid="ignore", divide="ignore"):
                v = np.where(np.isfinite(r), _value(q, x, y, z), 0.0)
            f.set_domain(d, v)
        out.append(f.std_base_cart(3) if q % 5 == 4 else f.std_base())
    return out


# x y holds the sine of 2 phi, which needs more than four phi points
def _value(q, x, y, z):
    r2 = x * x + y * y + z * z
    with np.errstate(invalid="ignore"):
        if q % 5 == 4:  # odd in z
            return (q + 1) * z / (4.0 + r2) ** 2
        return (q + 1 + x * y - 0.5 * z * z) / (4.0 + r2) ** 2


def _check(ctx, res, nf, npts, tol=1e-6):
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Space_spheric, val_points
    space = Space_spheric(CHEB_TYPE, (0, 0, 0), res, (1.0, 2.0, 4.0), ctx=ctx)
    fields = _fields(space, nf)
    rng = np.random.default_rng(npts)
    pts = rng.uniform(-6, 6, (npts, 3))
    special = np.array([[0, 0, 0], [0, 0, 0.7], [0, 0, -3.0], [1.0, 0, 0], [0, 2.0, 0], [np.inf, 0, 0], [0, 0, np.inf]])
    k = min(npts, len(special))
    pts[:k] = special[:k]
    got = val_points(fields, pts)
    whole = val_points(fields, np.vstack([pts] * (1 + 70000 // npts)))[:, :npts]
    for q in range(nf):
        v = _value(q, *pts.T)
        v = np.where(np.isfinite(pts).all(1), v, 0.0)
        # spectral accuracy of the smooth test fields at these resolutions
        assert np.abs(got[q] - v).max() <= tol
    # the few-points and the grouped kernel sum the same terms in another order
    assert np.abs(got - whole).max() <= 1e-13 * max(1.0, np.abs(got).max())


@pytest.mark.parametrize("nf", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("npts", [1, 15, 16, 17, 1000])
def test_few_and_grouped_points(ctx, nf, npts):
    _check(ctx, (17, 9, 8), nf, npts, 1e-3)


def test_tables_that_do_not_fit(ctx):
    _check(ctx, (33, 7, 8), 2, 200, 1e-3)  # more than 32 radial points: the plain kernel


def test_points_in_no_domain_and_zero_fields(ctx):
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Scalar, Space_spheric, val_points
    space = Space_spheric(CHEB_TYPE, (0, 0, 0), (9, 5, 4), (1.0, 2.0), withzec=False, ctx=ctx)
    one, zero = Scalar(space, 1.0).std_base(), Scalar(space, 0.0).std_base()
    for n in (4, 70000):
        pts = np.tile([[0.5, 0, 0], [3.0, 0, 0], [0, 1.5, 0], [np.nan, 0, 0]], (n // 4, 1))
        got = val_points([one, zero], pts)
        inside = np.tile([True, False, True, False], n // 4)
        assert np.abs(got[0][inside] - 1.0).max() < 1e-14 and (got[1][inside] == 0.0).all()
        assert np.isnan(got[:, ~inside]).all()
