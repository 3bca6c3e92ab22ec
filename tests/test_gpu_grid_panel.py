"""The cooperative grid panel (FP64, and FP32 panels too tall for a cluster) and
the FP64 U12 solve where they can go wrong: fewer rows than a CTA takes, one
row more than the CTAs share evenly, ties, zero pivots in the middle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _solve(ctx, a, mode=0):
    from kadath_frontera_gb300.kadath import DenseLU
    n = a.shape[0]
    x = np.random.default_rng(n).standard_normal(n)
    b = a @ x
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(da.data_ptr(), n, n, mode)
    lu.solve(db.data_ptr())
    return db.cpu().numpy(), x, da.cpu().numpy().T


@pytest.mark.parametrize("n", [1, 2, 31, 33, 95, 96, 97, 127, 193, 289, 1000])
def test_factors_are_lapacks(ctx, n):
    """Same pivots as LAPACK (largest modulus, lowest row first), so the factors
    agree entry by entry to a growth of rounding errors."""
    from scipy.linalg import lu_factor
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + n ** 0.5 * np.diag(rng.choice([-1.0, 1.0], n))
    got, x, f = _solve(ctx, a)
    ref, _ = lu_factor(a)
    # entries of L are at most 1 and of U of the size of a: n u of the largest,
    # times a growth that stays below 1e3 for such matrices
    assert np.abs(f - ref).max() <= 1e3 * n * 1.2e-16 * np.abs(ref).max()
    assert np.linalg.norm(got - x) <= 1e-9 * np.linalg.norm(x)


def test_ties_go_to_the_lowest_row(ctx):
    """Entries of equal modulus everywhere: the factors of integers are exact,
    so one other choice of pivot would show in them."""
    from scipy.linalg import lu_factor
    n = 300
    a = np.where(np.arange(n)[:, None] >= np.arange(n)[None, :], 1.0, 0.0) * np.where(np.arange(n) % 2, -1.0, 1.0)[:, None]
    a[:, -1] = 1.0
    a[-1, -1] = 3.0
    _, _, f = _solve(ctx, a)
    ref, _ = lu_factor(a)
    assert np.array_equal(f, ref)


@pytest.mark.parametrize("col", [0, 40, 95, 96, 150])
def test_zero_column_is_reported(ctx, col):
    from kadath_frontera_gb300 import KadathError
    n = 200
    a = np.random.default_rng(1).standard_normal((n, n))
    a[:, col] = 0.0
    with pytest.raises(KadathError) as e:
        _solve(ctx, a)
    assert e.value.status == 3  # KD_ERR_SINGULAR


@pytest.mark.parametrize("n", [2, 33, 95, 97, 200, 450, 897, 1300, 3600])
def test_cluster_panel_pivots_as_lapack(ctx, n):
    """The FP32 cluster panel (clusters of 2 to 16 CTAs, one or two rows a thread,
    last panels of any width) on a matrix of small integers, whose first pivots are
    exact in FP32 as in LAPACK: the solves then need few refinements."""
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP32_IR
    rng = np.random.default_rng(n)
    a = rng.integers(-4, 5, (n, n)).astype(float) + 3.0 * n ** 0.5 * np.diag(rng.choice([-1.0, 1.0], n))
    x = rng.standard_normal(n)
    b = a @ x
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(da.data_ptr(), n, n, KD_LU_FP32_IR)
    lu.solve(db.data_ptr())
    # refined to 1e-14 relative residual; the condition number is below 1e3
    assert np.linalg.norm(db.cpu().numpy() - x) <= 1e-10 * np.linalg.norm(x)
    assert lu.stats()["refine_iters"] <= 6
