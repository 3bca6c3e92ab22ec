"""Value passes and J x collected into levels (one launch per level) against the
same passes launched operation by operation (profile mode times single
launches and collects nothing): equal to the bit, for scalar and index-notation
systems, EOS operators (which launch in between), integral equations and a
resolution whose fields are too large to be collected."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _perturbed(wl, seed):
    rng = np.random.default_rng(seed)
    sp = wl.space
    for name, f in wl.unknowns:
        a = rng.uniform(0.01, 0.05)
        for d in range(sp.get_nbr_domains()):
            r = sp.get_radius(d)
            q = np.where(np.isfinite(r), 1.0 / (1.0 + np.where(np.isfinite(r), r, 0.0) ** 2 / 9.0), 0.0)
            v = f.get_domain(d)
            if name == "H":
                f.set_domain(d, v * (1.0 - a * q) if np.any(v) else v)
            elif not name.startswith("b"):
                f.set_domain(d, v + a * q)


def _both(wl, fn):
    from kadath_frontera_gb300.kadath import profile_enable
    ctx = wl.space.ctx
    collected = fn()
    again = fn()
    profile_enable(ctx, True)
    try:
        single = fn()
    finally:
        profile_enable(ctx, False)
    assert np.array_equal(collected, again)
    assert np.array_equal(collected, single)
    assert np.isfinite(collected).all() and np.any(collected != 0.0)


@pytest.mark.parametrize("name,res", [("toy", (9, 5, 4)), ("star", (9, 5, 4)), ("star_vector", (9, 5, 4)),
                                      ("ns_tov", (9, 5, 4)), ("star", (11, 9, 8)), ("star", (25, 11, 14))])
def test_residual_is_the_same_to_the_bit(ctx, name, res):
    from kadath_frontera_gb300 import workloads
    wl = workloads.WORKLOADS[name](res=res, ctx=ctx)
    _perturbed(wl, 1)
    _both(wl, wl.syst.sec_member)


@pytest.mark.parametrize("name", ["toy", "star_vector", "ns_tov"])
def test_jx_is_the_same_to_the_bit(ctx, name):
    from kadath_frontera_gb300 import workloads
    wl = workloads.WORKLOADS[name](res=(9, 5, 4), ctx=ctx)
    _perturbed(wl, 2)
    wl.syst.sec_member()
    x = np.random.default_rng(3).standard_normal(wl.syst.get_nbr_unknowns())
    _both(wl, lambda: wl.syst.do_JX(x))


def test_integral_equations_and_a_failing_pass(ctx):
    """A pass that reads a number in between, then one that throws: the context
    stays usable and the next pass is right."""
    from kadath_frontera_gb300 import KadathError, workloads
    from kadath_frontera_gb300.kadath import Scalar, System_of_eqs
    wl = workloads.toy(res=(9, 5, 4), ctx=ctx)
    psi = wl.unknowns[0][1]
    syst = System_of_eqs(wl.space, 0, 2)
    syst.add_var("psi", psi)
    syst.add_eq_int_volume(0, 2, "integvolume(psi^5) = 1")
    for d in range(3):
        syst.add_eq_inside(d, "Lap(psi) = 0")
    wl.syst.sec_member()
    try:
        a, b = syst.sec_member(), syst.sec_member()
        assert np.array_equal(a, b)
    except KadathError:
        pass  # the volume of an unbounded domain may be refused; the context must survive it
    bad = System_of_eqs(wl.space, 0, 2)
    bad.add_var("psi", psi)
    bad.add_cst("z", Scalar(wl.space, 0.0).std_base())
    bad.add_eq_inside(0, "Lap(psi) + psi / z = 0")
    with pytest.raises(KadathError):
        bad.sec_member()
    _both(wl, wl.syst.sec_member)
