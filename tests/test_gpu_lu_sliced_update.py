"""The FP64 LU's trailing update by exact 8-bit slices on the tensor cores:
sizes around its tiles (128 x 64, panels of 96 with a remainder) and matrices
whose entries spread over many magnitudes, against LAPACK on the same matrix."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _matrix(kind, n, rng):
    a = rng.standard_normal((n, n)) / np.sqrt(n) + 2.0 * np.diag(rng.choice([-1.0, 1.0], n))
    if kind == "rows":
        a *= 10.0 ** rng.uniform(-6, 6, (n, 1))
    elif kind == "columns":
        a *= 10.0 ** rng.uniform(-6, 6, (1, n))
    elif kind == "both":
        a *= 10.0 ** rng.uniform(-4, 4, (n, 1)) * 10.0 ** rng.uniform(-4, 4, (1, n))
    elif kind == "tiny":
        a *= 1e-290
    elif kind == "huge":
        a *= 1e290
    elif kind == "sparse":
        a[rng.random((n, n)) < 0.9] = 0.0
        a += 3.0 * np.eye(n)
    return a


def _errors(a, x, b):
    """Largest componentwise backward error |r| / (|A||x| + |b|), in long double."""
    la, lx, lb = a.astype(np.longdouble), x.astype(np.longdouble), b.astype(np.longdouble)
    r = np.abs(la @ lx - lb)
    return float((r / (np.abs(la) @ np.abs(lx) + np.abs(lb))).max())


@pytest.mark.parametrize("kind", ["plain", "rows", "columns", "both", "tiny", "huge", "sparse"])
@pytest.mark.parametrize("n", [352, 353, 480, 737, 1100])
def test_fp64_solve_is_as_exact_as_lapack(ctx, kind, n):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP64
    rng = np.random.default_rng(n)
    a = _matrix(kind, n, rng)
    b = a @ rng.standard_normal(n)
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(da.data_ptr(), n, n, KD_LU_FP64)
    lu.solve(db.data_ptr())
    got, ref = _errors(a, db.cpu().numpy(), b), _errors(a, np.linalg.solve(a, b), b)
    # both are Gaussian elimination with partial pivoting in 53 bits, whose
    # backward error is a modest multiple of n u (u = 1.1e-16) that depends on
    # the order of the sums; a lost digit of a slice would show as 2^-45 or more
    assert got <= 4 * ref + n * 1.2e-16, (got, ref)


def test_non_finite_entries_stay_non_finite(ctx):
    from kadath_frontera_gb300 import KadathError
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP64
    n = 480
    a = _matrix("plain", n, np.random.default_rng(0))
    a[470, 3] = np.nan
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.ones(n, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    try:
        lu.factor(da.data_ptr(), n, n, KD_LU_FP64)
        lu.solve(db.data_ptr())
    except KadathError:
        return
    assert not np.isfinite(db.cpu().numpy()).all()
