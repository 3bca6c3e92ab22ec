"""Points so close to the axis that the squares of their coordinates are subnormal:
phi is that of the point, to all its digits, for fields whose values there depend
on phi (nothing holds a field's coefficients to be regular)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 3000])
def test_phi_near_the_axis(ctx, copies):
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Scalar, Space_spheric, val_points
    space = Space_spheric(CHEB_TYPE, (0, 0, 0), (9, 5, 8), (1.0, 2.5), ctx=ctx)
    rng = np.random.default_rng(3)
    f = Scalar(space)
    for d in range(3):
        f.set_domain(d, rng.standard_normal((9, 5, 8)))
    f.std_base()
    phi = np.array([0.3, 1.1, 2.5, -0.7, -2.9])

    def at(s, z):
        xyz = np.stack([s * np.cos(phi), s * np.sin(phi), np.full(len(phi), z)], -1)
        return val_points([f], np.tile(xyz, (copies, 1)))[0]
    for z in (1.7, -1.7, 0.4, 8.0):
        ref = at(1e-100, z)
        assert np.ptp(ref[:5]) > 0.1  # phi matters
        for s in (1e-150, 1e-157, 1e-160, 3e-161):
            # theta differs by less than 1e-99: rounding of some 300 terms of size 1
            # and of phi itself, whose cosine and sine are formed from it here
            assert np.abs(at(s, z) - ref).max() <= 1e-11
    assert np.abs(at(0.0, 1.7) - at(0.0, 1.7)[0]).max() == 0.0


def test_near_the_origin(ctx):
    """The same with z as small: theta from the coordinates too."""
    from kadath_frontera_gb300.kadath import CHEB_TYPE, Scalar, Space_spheric, val_points
    space = Space_spheric(CHEB_TYPE, (0, 0, 0), (9, 5, 8), (1.0, 2.5), ctx=ctx)
    rng = np.random.default_rng(4)
    f = Scalar(space)
    for d in range(3):
        f.set_domain(d, rng.standard_normal((9, 5, 8)))
    f.std_base()
    u = rng.standard_normal((40, 3))
    few, ref = val_points([f], u * 1e-150)[0], val_points([f], u * 1e-100)[0]
    assert np.ptp(ref) > 0.1
    # coordinates with squares of 1e-300: 20 bits or more below the normal range's end
    assert np.abs(few - ref).max() <= 1e-11
