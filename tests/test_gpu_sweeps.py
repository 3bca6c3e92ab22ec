"""The chained triangular sweeps where they can go wrong: transposed sweeps
around the 64-row block and the three-block group, and matrices of more
groups than SMs (a CTA then works on several groups in turn)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    # diagonally weighted random matrix: condition number O(10)
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64) / n ** 0.5
    a.diagonal().add_(3.0)
    return a, torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 191, 192, 193, 577, 1001])
def test_transposed_solve_matches_numpy(ctx, n, mode):
    from kadath_frontera_gb300.kadath import DenseLU
    a, b = _matrix(n, n)
    x = b.clone()
    work = a.t().contiguous()  # column-major storage of a
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    lu.factor(work.data_ptr(), n, n, mode)
    lu.solve(x.data_ptr(), 1)
    ref = np.linalg.solve(a.cpu().numpy().T, b.cpu().numpy())
    # backward stable solve: error <= c n eps cond with cond = O(10), c n eps
    # below 1e-11 for n <= 1001; the refinement stops at 1e-14 relative residual
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("trans", [0, 1])
def test_more_groups_than_sms(ctx, trans):
    from kadath_frontera_gb300.kadath import DenseLU, KD_LU_TF32_IR
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 192 * sms + 71  # one group more than the SMs, with a ragged last block
    a, b = _matrix(n, 5)
    x = b.clone()
    torch.cuda.synchronize()
    lu = DenseLU(ctx)
    # row-major a is the column-major transpose: solve a x = b with trans
    lu.factor(a.data_ptr(), n, n, KD_LU_TF32_IR)
    lu.solve(x.data_ptr(), trans)
    r = (a @ x if trans else a.t() @ x) - b
    assert float(r.norm() / b.norm()) < 1e-12  # the refinement's own test is 1e-14
    assert lu.stats()["refine_iters"] <= 8  # FP32 factors of a matrix of condition O(10)
