"""Static-pivot panels: row counts around a CTA's share of L21 (128 rows and
multiples of 32 on up to 38 CTAs), odd last rows, and more rows than one round."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# panel heights below the first diagonal block of n - 96: 0, 1, 127 .. 129, an
# odd number of rows; 38 * 128 and one more; 38 * 384 and one more (a second round)
@pytest.mark.parametrize("n", [96, 97, 223, 224, 225, 291, 1003, 4960, 4961, 14688, 14689])
def test_reused_order_is_as_good_as_pivoting(ctx, n):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_TF32_IR
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    a.diagonal().add_(3.0)  # condition O(10)
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    lu = DenseLU(ctx)
    lu.set_pivot_reuse(True)
    iters = []
    for reused in (False, True):
        x = b.clone()
        torch.cuda.synchronize()
        lu.factor(a.data_ptr(), n, n, KD_LU_TF32_IR)  # the column-major transpose of a
        lu.solve(x.data_ptr())
        assert lu.pivot_info() == (reused, False)
        assert float((a.t() @ x - b).norm() / b.norm()) < 1e-12  # the refinement's own test is 1e-14
        iters.append(lu.stats()["refine_iters"])
    assert iters[1] <= iters[0] + 1  # the same matrix in the same order
