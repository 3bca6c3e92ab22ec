"""Partial pivoting with panels taller than a cluster: 192 columns as two halves
on the cooperative grid, then the change to cluster panels.  The pivot order that
the wide panels leave behind is checked by factoring again in that order."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# 12,768 rows are the most a cluster panel holds: one row more, so that a cluster
# panel follows the first wide one; two wide ones; several and a ragged end
@pytest.mark.parametrize("n", [12769, 12961, 14209])
def test_factors_and_pivot_order(ctx, n):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_TF32_IR
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    a += 2.0 * torch.eye(n, device="cuda", dtype=torch.float64)[torch.randperm(n, generator=g, device="cuda")]
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
    # condition O(100) and FP32 factors: a wrong exchange would not converge, or
    # only with many more iterations than the other order of the same products
    assert iters[0] <= 12 and iters[1] <= iters[0] + 2
