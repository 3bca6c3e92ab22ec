"""Infinities and NaN among coefficients reach the points they are summed at: all
but those where a sine of phi vanishes exactly (y = 0 and x >= 0), on the many-
and on the few-points path."""
import numpy as np
import pytest

from oracle import kadath as K, kadath_io as KIO

pytestmark = pytest.mark.gpu


def _field(ctx, path, column, junk):
    from kadath_frontera_gb300.kadath import KadathFile, Scalar, Space_spheric
    doms = K.space_spheric((9, 5, 8), [1.0, 2.5])
    f = K.scalar_field(doms, lambda d: np.ones(d.np))
    rng = np.random.default_rng(2)
    for d in doms:
        f[d.num].coef()
    shell = f[1]
    shell.c = None
    shell.cf = rng.standard_normal((1,) + tuple(doms[1].nc))
    shell.cf[..., 1] = shell.cf[..., doms[1].nc[2] - 1] = 0.0
    if column is not None:
        shell.cf[0, 2, 1, column] = junk
    with open(path, "wb") as fp:
        KIO.write_space(fp, doms)
        KIO.write_scalar(fp, doms, f)
    with KadathFile(path, "r") as kf:
        space = Space_spheric.from_file(kf, ctx=ctx)
        return Scalar.from_file(space, kf)


@pytest.mark.parametrize("copies", [1, 4000])
@pytest.mark.parametrize("junk", [np.nan, np.inf])
@pytest.mark.parametrize("column", [2, 3, 6, 7])
def test_shell(ctx, tmp_path, copies, junk, column):
    from kadath_frontera_gb300.kadath import val_points
    clean = _field(ctx, tmp_path / "clean.dat", None, 0.0)
    bad = _field(ctx, tmp_path / "bad.dat", column, junk)
    pts = np.array([[1.5, 0.0, 0.3], [1.2, 0.0, -0.9], [0.0, 0.0, 2.0], [0.0, 0.0, -2.0],  # sin(m phi) is zero
                    [-1.5, 0.0, 0.3], [0.0, 1.5, 0.3], [0.0, -1.5, 0.3], [0.7, 0.8, 0.9], [-1.0, 1.0, -1.0],
                    [0.5, 0.0, 0.1], [3.0, 0.0, 1.0]])
    pts = np.tile(pts, (copies, 1))
    ref, got = val_points([clean], pts)[0], val_points([bad], pts)[0]
    shell, axis = np.arange(len(pts)) % 11 < 9, np.arange(len(pts)) % 11 < 4
    spared = ~shell | axis if column % 2 else ~shell
    assert np.isfinite(ref).all()
    assert np.array_equal(got[spared], ref[spared])
    assert not np.isfinite(got[~spared]).any()
