"""A value pass that fails while its rows are exported leaves no recorded node
values behind: a Jacobian that may reuse the values of the preceding pass
evaluates them again.  (A C++ client: the C entry points evaluate a residual
before every such Jacobian themselves.)"""
import shutil
import subprocess

import pytest

from kadath_frontera_gb300 import _lib

pytestmark = pytest.mark.gpu

CLIENT = r"""
#include <cmath>
#include <cstdio>
#include "kd_system.hpp"
using namespace kd;

static void values(Field& f, double a) {
  for (int d = 0; d < f.sp->ndom(); d++) {
    const Domain& dm = f.sp->dom(d);
    std::vector<double> v(dm.npts());
    for (int i = 0; i < dm.np[0]; i++)
      for (int e = 0; e < dm.np[1] * dm.np[2]; e++)
        v[i * dm.np[1] * dm.np[2] + e] = 1.0 + a / (1.0 + d + 0.1 * i * i);
    f.set_conf_host(d, v.data());
  }
}

int main() {
  Context ctx(0);
  const double center[3] = {0, 0, 0};
  const int n[3] = {9, 5, 4};
  Space sp(center, n, {1.0, 2.0}, true);
  Field f(&ctx, &sp);
  f.std_base();
  values(f, 0.1);
  System sys(&ctx, &sp, 0, 2);
  sys.add_var("f", &f);
  for (int d = 0; d < 3; d++) sys.add_eq_inside(d, "Lap(f) - f^3 = 0");
  for (int d = 0; d < 2; d++) {
    sys.add_eq_matching(d, 0, "f");
    sys.add_eq_matching(d, 0, "dn(f)");
  }
  sys.add_eq_bc(2, 0, "f = 1");
  sys.residual(nullptr, true);
  const int N = sys.nbr_unknowns();
  if (sys.nbr_conditions() != N) return std::printf("%d conditions, %d unknowns\n", sys.nbr_conditions(), N), 1;
  double *J, *F;
  cudaMalloc(&J, sizeof(double) * N * N);
  cudaMalloc(&F, sizeof(double) * N);
  std::vector<double> first(size_t(N) * N), reused(first), fresh(first);
  auto get = [&](std::vector<double>& to) {
    cudaStreamSynchronize(ctx.stream());
    cudaMemcpy(to.data(), J, sizeof(double) * to.size(), cudaMemcpyDeviceToHost);
  };
  sys.jacobian(J, N, true);
  get(first);
  // other values, and a basis with another number of conditions: the pass
  // evaluates every node, then its export throws
  values(f, 0.7);
  const Base base = f.d[1].base;
  f.d[1].base = sp.dom(1).cart_base(2);
  try {
    sys.residual(F, true);
    return std::printf("the export did not throw\n"), 1;
  } catch (const KdError&) {
  }
  f.d[1].base = base;
  sys.jacobian(J, N, true);
  get(reused);
  sys.jacobian(J, N, false);
  get(fresh);
  double worst = 0, change = 0;
  for (size_t i = 0; i < fresh.size(); i++) {
    worst = std::fmax(worst, std::fabs(reused[i] - fresh[i]));
    change = std::fmax(change, std::fabs(first[i] - fresh[i]));
    if (!std::isfinite(reused[i]) || !std::isfinite(fresh[i])) return std::printf("not finite\n"), 1;
  }
  std::printf("%g %g\n", worst, change);
  return 0;
}
"""


def test_reuse_after_a_failed_pass(tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not available")
    _lib.load()
    lib = _lib.LIB_PATH
    src, exe = tmp_path / "client.cpp", tmp_path / "client"
    src.write_text(CLIENT)
    csrc = lib.parent / "csrc"
    cmd = ["nvcc", "-std=c++17", "-I", str(csrc), "-I", str(lib.parent.parent / "include"), str(src), "-o", str(exe),
           "-L", str(lib.parent), "-lkadath_gb300", "-Xlinker", "-rpath=" + str(lib.parent)]
    out = subprocess.run(cmd, capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr
    worst, change = map(float, run.stdout.split())
    assert worst == 0.0 and change > 1e-3
