"""Triangular sweeps over FP32 factors in groups of two 64-row blocks with the
inverse of each group: sizes around a block and a group, both directions, and a
right-hand side that is not a number."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    a.diagonal().add_(3.0)  # condition O(10)
    return a, torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n", [2, 62, 66, 126, 127, 128, 129, 130, 192, 255, 257, 385, 1029])
def test_sizes_around_blocks_and_groups(ctx, n, trans):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP32_IR
    a, b = _matrix(n, n)
    x = b.clone()
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    # row-major a is the column-major transpose: solve a x = b with trans
    lu.factor(a.data_ptr(), n, n, KD_LU_FP32_IR)
    lu.solve(x.data_ptr(), trans)
    r = (a @ x if trans else a.t() @ x) - b
    assert float(r.norm() / b.norm()) < 1e-12  # the refinement's own test is 1e-14
    # FP32 factors of a matrix of condition O(10) gain about six digits a step
    assert lu.stats()["refine_iters"] <= 5


@pytest.mark.parametrize("trans", [0, 1])
def test_nan_travels_through_the_sweeps(ctx, trans):
    from kadath_frontera_gb300 import KadathError
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP32_IR
    n = 700
    a, b = _matrix(n, 3)
    b[5] = float("nan")
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(a.data_ptr(), n, n, KD_LU_FP32_IR)
    with pytest.raises(KadathError, match="did not converge"):  # and no wait runs out
        lu.solve(b.data_ptr(), trans)
