"""GMRES refinement with more basis vectors than one combination launch takes
(32), and sizes around the CTAs of its vector kernels."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 1023, 4097])
def test_many_steps_of_one_cycle(ctx, n):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_FP32_IR
    g = torch.Generator(device="cuda").manual_seed(n)
    a = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    a.diagonal().add_(3.0)
    b = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    lu = DenseLU(ctx)
    lu.set_refinement(1e-13, 50, 4)
    torch.cuda.synchronize()
    lu.factor(a.data_ptr(), n, n, KD_LU_FP32_IR)
    # the refinement reads the matrix where it lies: a change of rank 40 takes
    # the factors' product to one with 41 distinct eigenvalues, so 41 steps
    u = torch.linalg.qr(torch.randn((n, 40), generator=g, device="cuda", dtype=torch.float64))[0]
    a += (u * torch.linspace(2.0, 40.0, 40, device="cuda", dtype=torch.float64)) @ u.t()
    x = b.clone()
    torch.cuda.synchronize()
    lu.solve(x.data_ptr())
    r = a.t() @ x - b  # a's memory is the column-major transpose
    assert float(r.norm() / b.norm()) < 1e-11
    assert 33 <= lu.stats()["refine_iters"] <= 90
