"""An infinite entry in the FP64 LU: as the pivot of its column it gives zero
multipliers, so its unknown is zero and the others solve the system without its
row and column."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("n,row,col", [(90, 7, 3), (300, 250, 5), (520, 40, 130)])
def test_infinite_pivot(ctx, n, row, col, sign):
    from kadath_frontera_gb300 import KadathError
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP64
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) / np.sqrt(n) + 2.0 * np.diag(rng.choice([-1.0, 1.0], n))
    a[row, col] = sign * np.inf
    b = rng.standard_normal(n)
    da, db = torch.tensor(a.T.copy(), device="cuda"), torch.tensor(b, device="cuda")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    try:
        lu.factor(da.data_ptr(), n, n, KD_LU_FP64)
        lu.solve(db.data_ptr())
    except KadathError:
        # an infinity right of its first panel spreads as NaN, which no pivot is
        assert col >= 96
        return
    x = db.cpu().numpy()
    keep_r, keep_c = np.arange(n) != row, np.arange(n) != col
    ref = np.zeros(n)
    ref[keep_c] = np.linalg.solve(a[np.ix_(keep_r, keep_c)], b[keep_r])
    assert np.abs(x - ref).max() <= 1e-9 * np.abs(ref).max()
