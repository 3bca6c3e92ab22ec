"""Value passes with integral-type equations, whose numbers come back to the host
in the middle of the collected pass: the residual and J x are those of the pass
launched operation by operation, to the bit, and the equation really is there."""
import numpy as np
import pytest

from tests.test_gpu_integral import build_eigen, build_mass

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build", [lambda: build_eigen((9, 5, 4), "integral"), lambda: build_eigen((9, 5, 4), "val"),
                                   lambda: build_mass((9, 5, 4))])
def test_collected_and_single(ctx, build):
    from kadath_frontera_gb300.kadath import profile_enable
    space, syst, f = build()
    x = None

    def passes():
        nonlocal x
        F = syst.sec_member()
        if x is None:
            x = np.random.default_rng(1).standard_normal(syst.get_nbr_unknowns())
        return F, syst.do_JX(x)

    collected, again = passes(), passes()
    profile_enable(space.ctx, True)
    try:
        single = passes()
    finally:
        profile_enable(space.ctx, False)
    for c, a, s in zip(collected, again, single):
        assert np.isfinite(c).all() and np.any(c != 0.0)
        assert np.array_equal(c, a) and np.array_equal(c, s)
    # the integral's row comes first: it is not zero, or depends on the unknowns
    assert abs(collected[0][0]) > 1e-6 or abs(collected[1][0]) > 1e-6
