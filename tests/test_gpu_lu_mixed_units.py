"""The FP64 LU on matrices whose unknowns are in different units: two interleaved
groups, one of whose equations hold that group's unknowns only, its columns
scaled by a power of two.  Elimination with partial pivoting in FP64 gives the
same digits whatever that power is; an update that holds its operands relative
to their row's largest entry does not."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _coupled(n, t, weight, coupling, seed):
    """Even equations hold all unknowns, odd ones (times `weight`) the odd
    unknowns and, times `coupling`, the even ones; odd columns scaled by 2^t."""
    rng = np.random.default_rng([n, seed])
    a = rng.standard_normal((n, n)) / np.sqrt(n) + 2.0 * np.diag(rng.choice([-1.0, 1.0], n))
    a[1::2, 0::2] *= coupling
    a[1::2] *= weight
    a[:, 1::2] *= 2.0 ** t
    x = rng.standard_normal(n)
    x[1::2] *= 2.0 ** -t
    return a, a @ x


def _backward(a, x, b):
    """Largest componentwise backward error |r| / (|A||x| + |b|), in long double."""
    la, lx, lb = a.astype(np.longdouble), x.astype(np.longdouble), b.astype(np.longdouble)
    return float((np.abs(la @ lx - lb) / (np.abs(la) @ np.abs(lx) + np.abs(lb))).max())


def _solve(ctx, a, b):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP64
    n = len(b)
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(da.data_ptr(), n, n, KD_LU_FP64)
    lu.solve(db.data_ptr())
    return db.cpu().numpy()


@pytest.mark.parametrize("weight,coupling", [(1.0, 0.0), (8.0, 0.0), (8.0, 2.0 ** -30)])
@pytest.mark.parametrize("t", [0, -10, -20, -30, -40, -60, -200, 40])
@pytest.mark.parametrize("n", [400, 737])
def test_backward_error_is_lapacks(ctx, n, t, weight, coupling):
    got, ref = 0.0, 0.0
    for seed in range(2):
        a, b = _coupled(n, t, weight, coupling, seed)
        got = max(got, _backward(a, _solve(ctx, a, b), b))
        ref = max(ref, _backward(a, np.linalg.solve(a, b), b))
    # both run the same elimination in 53 bits and differ in the order of their
    # sums; the errors of two such runs are of one size (a factor of a few), and
    # the group's digits lost at t = -20 already cost a factor of 25
    assert got <= 6 * ref, (got, ref)


@pytest.mark.parametrize("scale", [2.0 ** -1000, 2.0 ** -500, 2.0 ** 900])
def test_equations_near_the_ends_of_the_range(ctx, scale):
    """Every third equation scaled to near the ends of FP64's range: its
    multipliers are tiny (or the others' are), the products too."""
    a, b = _coupled(480, 0, 1.0, 1.0, 5)
    a[::3] *= scale
    b[::3] *= scale
    got = _backward(a, _solve(ctx, a, b), b)
    assert got <= 6 * _backward(a, np.linalg.solve(a, b), b)  # as above
