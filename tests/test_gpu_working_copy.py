"""The FP32 working copy of the mixed modes: powers of two moved and entries
rounded on the bit patterns, in the matrix's own row order and in a reused
pivot order, with entries that are zero, subnormal or below FP32's range."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _solve(lu, a, b, mode):
    n = a.shape[0]
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu.factor(da.data_ptr(), n, n, mode)
    lu.solve(db.data_ptr())
    return db.cpu().numpy(), lu.stats()["refine_iters"], lu.pivot_info()


@pytest.mark.parametrize("n", [33, 511, 513, 1100, 4099])
@pytest.mark.parametrize("mode", [1, 2])
def test_scaled_columns_and_tiny_entries_are_preconditioned_alike(ctx, mode, n):
    from kadath_frontera_gb300.kadath import DenseLU
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) / np.sqrt(n) + 2.0 * np.diag(rng.choice([-1.0, 1.0], n))
    spots = rng.integers(0, n, (5, 64))
    for value, at in zip((0.0, -0.0, 1e-300, 5e-324, 1e-42), spots):
        a[at, rng.integers(0, n, 64)] = value
    a[np.arange(n), np.arange(n)] += 1.0
    c = 2.0 ** rng.integers(-40, 41, n)  # the sweeps hold x in FP32
    b = rng.standard_normal(n)
    lu = DenseLU(ctx)
    lu.set_pivot_reuse(True)
    plain = [_solve(lu, a, b, mode) for _ in range(2)]
    lu = DenseLU(ctx)
    lu.set_pivot_reuse(True)
    scaled = [_solve(lu, a * c, b, mode) for _ in range(2)]
    for (x, it, info), (y, its, infos), reused in zip(plain, scaled, (False, True)):
        assert info == infos == (reused, False)
        # GMRES ends at the rounding level of FP64; a copy off by more than FP32
        # rounding would precondition worse, so it would take more iterations
        assert np.linalg.norm(a @ x - b) / np.linalg.norm(b) < 1e-12
        assert np.linalg.norm(a @ (c * y) - b) / np.linalg.norm(b) < 1e-12
        assert its <= it + 1


@pytest.mark.parametrize("mode", [1, 2])
def test_entries_are_rounded_to_nearest_even(ctx, mode):
    """A diagonal matrix is its own factor: with every entry a float (half-way
    cases excluded) the preconditioner is the inverse and one step is enough;
    with entries that FP32 rounds up into the next binade it still contracts by
    2^-24 a step, where a truncated or overflowing copy would not."""
    from kadath_frontera_gb300.kadath import DenseLU
    n = 640
    rng = np.random.default_rng(1)
    up = np.nextafter(2.0 ** rng.integers(-60, 60, n), 0.0)  # all mantissa bits set
    tie = (1.0 + 2.0 ** -24 + 2.0 ** -22 * rng.integers(0, 1 << 20, n)) * 2.0 ** rng.integers(-60, 60, n)
    for d in (up, tie, -up):
        b = d * rng.standard_normal(n)
        x, it, _ = _solve(DenseLU(ctx), np.diag(d), b, mode)
        assert np.abs(x - b / d).max() <= 1e-9 * np.abs(b / d).max()
        assert it <= 4
