"""A resolution whose line passes need nearly all of an SM's shared memory, the
matrices beside two stages of the field: collected into levels or launched one by
one, the residual is the same to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [(156, 3, 2), (155, 3, 2), (157, 2, 4)])
def test_residual(ctx, res):
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Scalar, Space_spheric, System_of_eqs, profile_enable
    space = Space_spheric(CHEB_TYPE, (0, 0, 0), res, (1.0, 2.0), ctx=ctx)
    f = Scalar(space)
    for d in range(3):
        r = space.get_radius(d)
        f.set_domain(d, np.where(np.isfinite(r), 1.0 / (1.0 + np.where(np.isfinite(r), r, 0.0) ** 2), 0.0))
    f.std_base()
    syst = System_of_eqs(space, 0, 2)
    syst.add_var("f", f)
    for d in range(3):
        syst.add_eq_inside(d, "Lap(f) + f^3 = 0")
    collected = syst.sec_member()
    profile_enable(ctx, True)
    try:
        single = syst.sec_member()
    finally:
        profile_enable(ctx, False)
    assert np.array_equal(collected, single) and np.isfinite(collected).all() and np.any(collected != 0.0)
