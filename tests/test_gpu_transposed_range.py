"""Transposed solves with FP32 factors: the sweeps work in FP64, so columns or
equations in any units change neither the steps of the refinement nor the
digits of the solution."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _solve(ctx, a, b, mode=2):
    from kadath_frontera_gb300.kadath import DenseLU
    n = len(b)
    w, x = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(w.data_ptr(), n, n, mode)
    lu.solve(x.data_ptr(), 1)
    return x.cpu().numpy(), lu.stats()["refine_iters"]


def _matrix(n, seed=0):
    rng = np.random.default_rng([n, seed])
    return rng.standard_normal((n, n)) / np.sqrt(n) + 2.0 * np.diag(rng.choice([-1.0, 1.0], n)), rng


def _check(a, x, b, it):
    r = np.abs(a.T @ x - b)
    # refined to FP64's rounding, row by row: every entry of b stands for itself
    assert (r / (np.abs(a.T) @ np.abs(x) + np.abs(b))).max() <= 1e-12
    # a step of refinement with FP32 factors of a matrix of condition O(10) gains
    # a factor of 1e5 or more, and FP64 has 16 digits
    assert it <= 4


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("n", [1, 64, 65, 193, 600, 1001])
def test_steps(ctx, n, mode):
    a, rng = _matrix(n)
    b = rng.standard_normal(n)
    x, it = _solve(ctx, a, b, mode)
    _check(a, x, b, it)


@pytest.mark.parametrize("bits", [40, 140, 200])
def test_columns_in_any_units(ctx, bits):
    n = 600
    a, rng = _matrix(n)
    c = 2.0 ** rng.integers(-bits, bits + 1, n)
    b = c * rng.standard_normal(n)
    x, it = _solve(ctx, a * c, b)
    _check(a * c, x, b, it)


@pytest.mark.parametrize("bits", [40, 140, 200])
def test_equations_in_any_units(ctx, bits):
    n = 600
    a, rng = _matrix(n)
    c = 2.0 ** rng.integers(-bits, bits + 1, n)[:, None]
    b = rng.standard_normal(n)
    x, it = _solve(ctx, a * c, b)
    _check(a * c, x, b, it)
