"""The 3xTF32 update in 128 x 256 tiles: at least two tiles an SM, k above 128,
with ragged last tiles in both directions and a last tile that is half empty."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(4096, 2560, 192), (4100, 2561, 192), (2004, 6100, 161), (38916, 1025, 130)])
def test_update_is_fp32_accurate(ctx, m, n, k):
    lib = ctx.lib
    lib.kd_tf32x3_gemm_update.restype = C.c_int
    lib.kd_tf32x3_gemm_update.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_longlong,
                                          C.c_void_p, C.c_longlong, C.c_void_p, C.c_longlong]
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    ldc = m + 4  # the entry point takes whole 16-byte rows only
    # column-major operands: column c at [c]
    a = torch.randn((k, m + 3), generator=g, device="cuda")
    b = torch.randn((n, k + 1), generator=g, device="cuda")
    c = torch.randn((n, ldc), generator=g, device="cuda")
    before = c.clone()
    torch.cuda.synchronize()
    st = lib.kd_tf32x3_gemm_update(ctx.h, m, n, k, a.data_ptr(), m + 3, b.data_ptr(), k + 1, c.data_ptr(), ldc)
    assert st == 0, lib.kd_last_error(ctx.h)
    ctx.synchronize()
    ref = before[:, :m].double() - b[:, :k].double() @ a[:, :m].double()
    # hi/lo split of both operands: the bound of the narrower tile's test
    scale = float(a.abs().max() * b.abs().max()) * k
    assert float((c[:, :m].double() - ref).abs().max()) <= 2.0 ** -17 * scale
    assert torch.equal(c[:, m:], before[:, m:])  # padding rows untouched
