"""Point evaluation of a field whose radial basis in a shell is even or odd, as a
save file may hold it: the sums need Chebyshev polynomials up to twice the
number of coefficients there too, not in the nucleus alone."""
import numpy as np
import pytest

from oracle import kadath as K, kadath_io as KIO, spectral as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("code", [S.CHEB, S.CHEB_EVEN, S.CHEB_ODD])
@pytest.mark.parametrize("npts", [300, 40000])
def test_shell_with_a_radial_parity(ctx, tmp_path, code, npts):
    from kadath_frontera_gb300.kadath import KadathFile, Scalar, Space_spheric, val_points
    doms = K.space_spheric((9, 5, 4), [1.0, 2.5])
    f = K.scalar_field(doms, lambda d: np.ones(d.np))
    rng = np.random.default_rng(2)
    for d in doms:
        f[d.num].coef()
    shell = f[1]
    shell.base.r[...] = code
    shell.c = None
    shell.cf = rng.standard_normal((1,) + tuple(doms[1].nc))
    shell.cf[..., 1] = shell.cf[..., doms[1].nc[2] - 1] = 0.0
    path = tmp_path / "field.dat"
    with open(path, "wb") as fp:
        KIO.write_space(fp, doms)
        KIO.write_scalar(fp, doms, f)
    with KadathFile(path, "r") as kf:
        space = Space_spheric.from_file(kf, ctx=ctx)
        s = Scalar.from_file(space, kf)
    pts = rng.standard_normal((npts, 3))
    pts *= (rng.uniform(1.01, 2.49, npts) / np.linalg.norm(pts, axis=1))[:, None]
    got = val_points([s], pts)[0]
    r = np.linalg.norm(pts, axis=1)
    xi, th = (r - doms[1].beta) / doms[1].alpha, np.arccos(pts[:, 2] / r)
    ph = np.arctan2(pts[:, 1], pts[:, 0])
    ref = np.zeros(npts)
    nr, nt, nk = doms[1].nc
    bt = np.asarray(shell.base.t)
    n = np.arange(nr) * (1 if code == S.CHEB else 2) + (1 if code == S.CHEB_ODD else 0)
    rad = np.cos(n[None] * np.arccos(np.clip(xi, -1, 1))[:, None])
    for k in range(nk):
        phi = np.cos(k // 2 * ph) if k % 2 == 0 else np.sin(k // 2 * ph)
        j = np.arange(nt)
        tt = {S.COS_EVEN: np.cos(2 * j * th[:, None]), S.COS_ODD: np.cos((2 * j + 1) * th[:, None]),
              S.SIN_EVEN: np.sin(2 * j * th[:, None]), S.SIN_ODD: np.sin((2 * j + 1) * th[:, None])}[bt[k]]
        ref += phi * ((rad @ shell.cf[0, :, :, k]) * tt).sum(1)
    # some 300 terms of size 1, recurrences of at most 18 steps
    assert np.abs(got - ref).max() <= 1e-11
