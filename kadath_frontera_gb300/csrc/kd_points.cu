// Spectral summation at arbitrary points (Scalar::val_point,
// include/scalar.hpp:221; Base_spectral::summation, src/Ope_1d/summation_1d.cpp)
// for many points and several fields at once: the step the reference's
// exporters (src/Utilities/Exporters) run point by point on the host.
//
// Bound: the FP64 pipe (one warp instruction in 16 cycles of an SM), so the
// kernels keep close to one multiply-add per coefficient: the Chebyshev values
// and the theta factors of a point are tabulated once for all fields, fields
// with the same bases are summed together (one table load for up to five
// multiply-adds), phi columns whose coefficients are all zero (sin 0, the sine
// at the highest frequency) are left out, and the angles enter through
// cos(theta) = z / r and so on, without trigonometric functions.
// One million points of five (13,9,4) fields: 10.2 -> 4.8 ms (2.8 k FP64
// instructions a point, 0.97 TFLOP/s of the 2,340 useful multiply-adds of each).
//   Many points: grouped by domain (two counting passes), a CTA takes runs of
//   128-point chunks of one domain with that domain's coefficients in shared
//   memory, one thread a point.
//   Few points (fewer than fill the GPU that way): one launch, eight lanes a
//   point, each lane a share of the (theta, phi) lines.
// Fields too large for the tables take the plain kernel: one thread a point,
// Clenshaw sums of coefficients read through the read-only cache.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "kd_points.hpp"

namespace kd {

namespace {

struct PtDom {
  int type;
  double alpha, beta, rin, rout;
  int nc0, nc1, nc2;
  int ncheb;  // Chebyshev values its fields need: nc0, twice that with even or odd radial bases
};

struct PtArgs {
  int ndom, nfields;
  double cx, cy, cz;
  PtDom d[PT_MAX_DOM];
  const double* cf[PT_MAX_FIELDS][PT_MAX_DOM];  // coefficients (null: a zero field)
  int tab_off[PT_MAX_FIELDS][PT_MAX_DOM];       // basis tables in `tab` (r: nc1*nc2 codes, then t: nc2 codes)
  // fields with equal bases, in runs of 1, 2, 4 or 5: field[first[g] .. + size[g])
  int ngroups, first[PT_MAX_FIELDS], size[PT_MAX_FIELDS], field[PT_MAX_FIELDS];
  int slot[4];  // table of each theta kind (-1: no field has it)
};

constexpr int B_CHEB = 1, B_CHEB_EVEN = 2, B_CHEB_ODD = 3;
constexpr int B_COS_EVEN = 6, B_COS_ODD = 7, B_SIN_EVEN = 9, B_SIN_ODD = 10;

// sum_{i < n} c[i * stride] T_i(y)
__device__ __forceinline__ double clenshaw(const double* __restrict__ c, int stride, int n, double y) {
  double b1 = 0.0, b2 = 0.0;
  for (int i = n - 1; i >= 1; i--) {
    const double b0 = fma(2.0 * y, b1, __ldg(c + static_cast<long long>(i) * stride) - b2);
    b2 = b1;
    b1 = b0;
  }
  return fma(y, b1, __ldg(c) - b2);
}

// sum_{i < n} c[i * stride] T_{2i+1}(x), as the full series with zero even terms
__device__ __forceinline__ double clenshaw_odd(const double* __restrict__ c, int stride, int n, double x) {
  double b1 = 0.0, b2 = 0.0;
  for (int m = 2 * n - 1; m >= 1; m--) {
    const double a = (m & 1) ? __ldg(c + static_cast<long long>(m >> 1) * stride) : 0.0;
    const double b0 = fma(2.0 * x, b1, a - b2);
    b2 = b1;
    b1 = b0;
  }
  return x * b1 - b2;  // a_0 = 0
}

__global__ void __launch_bounds__(256) val_points_kernel(const __grid_constant__ PtArgs a, const int* __restrict__ tab, long long npts,
                                                         const double* __restrict__ xyz, double* __restrict__ out) {
  for (long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; p < npts;
       p += static_cast<long long>(gridDim.x) * blockDim.x) {
    const double x = xyz[3 * p] - a.cx, y = xyz[3 * p + 1] - a.cy, z = xyz[3 * p + 2] - a.cz;
    const double r = sqrt(x * x + y * y + z * z);
    int dd = -1;
    for (int d = 0; d < a.ndom; d++)
      if (a.d[d].rin - 1e-12 <= r && r <= a.d[d].rout + 1e-12) {
        dd = d;
        break;
      }
    if (dd < 0) {
      for (int f = 0; f < a.nfields; f++) out[f * npts + p] = nan("");
      continue;
    }
    const PtDom& D = a.d[dd];
    double xi;
    if (D.type == 1) xi = r / D.alpha;
    else if (D.type == 2) xi = (r - D.beta) / D.alpha;
    else xi = 1.0 + 1.0 / r / D.alpha;
    const double rho = sqrt(x * x + y * y);
    double th, ph;
    if (rho == 0.0) {
      th = (z >= 0) ? 0.0 : M_PI;
      ph = 0.0;
    } else {
      th = (z != 0.0) ? atan(rho / z) : M_PI / 2;
      ph = atan2(y, x);
    }
    if (th < 0) th += M_PI;
    double st1, ct1, st2, ct2, sp1, cp1;
    sincos(th, &st1, &ct1);
    sincos(2.0 * th, &st2, &ct2);
    sincos(ph, &sp1, &cp1);
    const double y2 = fma(2.0 * xi, xi, -1.0);
    const int lstride = D.nc1 * D.nc2;
    for (int f = 0; f < a.nfields; f++) {
      const double* c = a.cf[f][dd];
      if (!c) {
        out[f * npts + p] = 0.0;
        continue;
      }
      const int* rb = tab + a.tab_off[f][dd];
      const int* tb = rb + lstride;
      double val = 0.0;
      double cm = 1.0, sm = 0.0;  // cos(m phi), sin(m phi), m = k / 2 (COSSIN)
      for (int k = 0; k < D.nc2; k++) {
        const double phik = (k & 1) ? sm : cm;
        if (k & 1) {  // advance m
          const double cn = cm * cp1 - sm * sp1;
          sm = sm * cp1 + cm * sp1;
          cm = cn;
        }
        if (phik == 0.0) continue;
        const int bt = __ldg(tb + k);
        // first angle of the theta series and its step (2 theta)
        double ct, st;
        if (bt == B_COS_EVEN || bt == B_SIN_EVEN) {
          ct = 1.0;
          st = 0.0;
        } else {
          ct = ct1;
          st = st1;
        }
        const bool use_cos = (bt == B_COS_EVEN || bt == B_COS_ODD);
        double acc = 0.0;
        for (int j = 0; j < D.nc1; j++) {
          const double thj = use_cos ? ct : st;
          const int br = __ldg(rb + j * D.nc2 + k);
          const double* line = c + j * D.nc2 + k;
          double rad;
          if (br == B_CHEB) rad = clenshaw(line, lstride, D.nc0, xi);
          else if (br == B_CHEB_EVEN) rad = clenshaw(line, lstride, D.nc0, y2);
          else rad = clenshaw_odd(line, lstride, D.nc0, xi);
          acc = fma(thj, rad, acc);
          const double cn = ct * ct2 - st * st2;
          st = st * ct2 + ct * st2;
          ct = cn;
        }
        val = fma(phik, acc, val);
      }
      out[f * npts + p] = val;
    }
  }
}

// ---- evaluation from per-point tables --------------------------------------
constexpr int PT_THREADS = 128;
constexpr int PT_SUB = 8;                              // lanes a point of the few-points kernel
// Fewer points than give every SM a chunk: eight lanes a point.  (1,000 points
// of one (13,9,4) field from the host: 80 us, 224 with the grouped kernels and
// a device allocation per call; 57,000 points of one (9,5,4) field: 215 with
// eight lanes each against about 145 grouped.)
constexpr long long PT_FEW = 152LL * PT_THREADS;
constexpr int PT_MAX_NR = 32;                          // tables of T_0 .. T_63

// A point in its domain: numerical radius, cosine and sine of its angles.
struct PtPos {
  double xi, ct, st, cp, sp;
};

// Whether every sine of phi is left out: at phi = 0, where all are exactly zero.
// (Elsewhere Inf and NaN among the coefficients of a column reach the point even
// where its factor happens to be zero.)
__device__ __forceinline__ bool pt_no_sines(const PtPos& q) { return q.sp == 0.0 && q.cp > 0.0; }

__device__ __forceinline__ int pt_locate(const PtArgs& a, const double* __restrict__ xyz, long long p, double& x,
                                         double& y, double& z, double& r) {
  x = xyz[3 * p] - a.cx;
  y = xyz[3 * p + 1] - a.cy;
  z = xyz[3 * p + 2] - a.cz;
  r = sqrt(x * x + y * y + z * z);
  for (int d = 0; d < a.ndom; d++)
    if (a.d[d].rin - 1e-12 <= r && r <= a.d[d].rout + 1e-12) return d;
  return -1;
}

__device__ __forceinline__ PtPos pt_position(const PtDom& D, double x, double y, double z, double r) {
  PtPos q;
  if (D.type == 1) q.xi = r / D.alpha;
  else if (D.type == 2) q.xi = (r - D.beta) / D.alpha;
  else q.xi = 1.0 + 1.0 / r / D.alpha;
  const double rho = sqrt(x * x + y * y);
  if (rho == 0.0) {  // the axis: theta 0 or pi, phi 0
    q.ct = z >= 0 ? 1.0 : -1.0;
    q.st = 0.0;
    q.cp = 1.0;
    q.sp = 0.0;
  } else if (isinf(r) || rho < 1e-140) {  // a point at infinity, or squares among the subnormals: angles first
    double th = (z != 0.0) ? atan(rho / z) : M_PI / 2;
    if (th < 0) th += M_PI;
    sincos(th, &q.st, &q.ct);
    sincos(atan2(y, x), &q.sp, &q.cp);
  } else {
    q.ct = z / r;
    q.st = rho / r;
    q.cp = x / rho;
    q.sp = y / rho;
  }
  return q;
}

// T_0 .. T_(n-1) of xi at t[i * stride].
__device__ __forceinline__ void pt_chebyshev(double xi, int n, double* t, int stride) {
  double tm2 = 1.0, tm1 = xi;
  t[0] = 1.0;
  if (n > 1) t[stride] = xi;
  for (int i = 2; i < n; i++) {
    const double v = fma(2.0 * xi, tm1, -tm2);
    t[i * stride] = v;
    tm2 = tm1;
    tm1 = v;
  }
}

// Index of a theta basis's table: cos 2j, cos 2j+1, sin 2j, sin 2j+1.
__device__ __forceinline__ int pt_theta_kind(int bt) {
  return bt == B_COS_EVEN ? 0 : bt == B_COS_ODD ? 1 : bt == B_SIN_EVEN ? 2 : 3;
}

// cos and sin of (2j + odd) theta, j < n, at c[j * stride] and s[j * stride]
// (null: not kept).
__device__ __forceinline__ void pt_theta(const PtPos& q, int odd, int n, double* c, double* s, int stride) {
  const double c2 = fma(2.0 * q.ct, q.ct, -1.0), s2 = 2.0 * q.st * q.ct;
  double cj = odd ? q.ct : 1.0, sj = odd ? q.st : 0.0;
  for (int j = 0; j < n; j++) {
    if (c) c[j * stride] = cj;
    if (s) s[j * stride] = sj;
    const double cn = cj * c2 - sj * s2;
    sj = sj * c2 + cj * s2;
    cj = cn;
  }
}

// acc[f] += th * sum_i c[(i * NF) + f] T, T at t[(ts i) * stride].
template <int NF>
__device__ __forceinline__ void pt_line(const double* __restrict__ c, int nr, const double* t, int step, double th,
                                        double (&acc)[NF]) {
  double rad[NF];
#pragma unroll
  for (int f = 0; f < NF; f++) rad[f] = 0.0;
#pragma unroll 2
  for (int i = 0; i < nr; i++) {
    const double ti = *t;
    t += step;
#pragma unroll
    for (int f = 0; f < NF; f++) rad[f] = fma(c[f], ti, rad[f]);
    c += NF;
  }
#pragma unroll
  for (int f = 0; f < NF; f++) acc[f] = fma(th, rad[f], acc[f]);
}

// Points per domain (bucket ndom: in none), counted per block first.
constexpr int PT_BLOCK_POINTS = 2048;
__global__ void pt_count(const __grid_constant__ PtArgs a, long long npts, const double* __restrict__ xyz,
                         int* __restrict__ count) {
  __shared__ int c[PT_MAX_DOM + 1];
  if (threadIdx.x <= PT_MAX_DOM) c[threadIdx.x] = 0;
  __syncthreads();
  const long long p0 = static_cast<long long>(blockIdx.x) * PT_BLOCK_POINTS;
  for (int e = threadIdx.x; e < PT_BLOCK_POINTS && p0 + e < npts; e += blockDim.x) {
    double x, y, z, r;
    const int d = pt_locate(a, xyz, p0 + e, x, y, z, r);
    atomicAdd(&c[d < 0 ? a.ndom : d], 1);
  }
  __syncthreads();
  if (threadIdx.x <= a.ndom && c[threadIdx.x]) atomicAdd(count + threadIdx.x, c[threadIdx.x]);
}

// First slot of each domain's points in `perm`, a multiple of the chunk.
__device__ __forceinline__ int pt_first_slot(const int* __restrict__ count, int d) {
  int s = 0;
  for (int q = 0; q < d; q++) s += (count[q] + PT_THREADS - 1) / PT_THREADS * PT_THREADS;
  return s;
}

// perm[slot] = point, grouped by domain (slots between the groups keep -1);
// points in no domain get their NaN here.
__global__ void pt_scatter(const __grid_constant__ PtArgs a, long long npts, const double* __restrict__ xyz,
                           const int* __restrict__ count, int* __restrict__ cursor, int* __restrict__ perm,
                           double* __restrict__ out) {
  __shared__ int c[PT_MAX_DOM + 1], base[PT_MAX_DOM + 1], at[PT_MAX_DOM + 1];
  if (threadIdx.x <= PT_MAX_DOM) c[threadIdx.x] = at[threadIdx.x] = 0;
  __syncthreads();
  const long long p0 = static_cast<long long>(blockIdx.x) * PT_BLOCK_POINTS;
  int mine[PT_BLOCK_POINTS / 256];
#pragma unroll
  for (int q = 0; q < PT_BLOCK_POINTS / 256; q++) {
    const long long p = p0 + threadIdx.x + q * 256;
    mine[q] = -1;
    if (p >= npts) continue;
    double x, y, z, r;
    mine[q] = pt_locate(a, xyz, p, x, y, z, r);
    if (mine[q] >= 0) atomicAdd(&c[mine[q]], 1);
    else
      for (int f = 0; f < a.nfields; f++) out[f * npts + p] = nan("");
  }
  __syncthreads();
  if (threadIdx.x < a.ndom && c[threadIdx.x])
    base[threadIdx.x] = pt_first_slot(count, threadIdx.x) + atomicAdd(cursor + threadIdx.x, c[threadIdx.x]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PT_BLOCK_POINTS / 256; q++)
    if (mine[q] >= 0) perm[base[mine[q]] + atomicAdd(&at[mine[q]], 1)] = static_cast<int>(p0 + threadIdx.x + q * 256);
}

// One group of NF fields at one point per thread; cs: the domain's
// coefficients of the group, [k][j][i][field].
template <int NF>
__device__ __forceinline__ void pt_group(const PtArgs& a, int g, int dd, const PtDom& D, const PtPos& q,
                                         const double* cs, const int* __restrict__ tab, const int* live,
                                         const double* T, const double* TH, long long npts, int p,
                                         double* __restrict__ out) {
  const int* rb = tab + a.tab_off[a.field[a.first[g]]][dd];
  const int* tb = rb + D.nc1 * D.nc2;
  double val[NF];
#pragma unroll
  for (int f = 0; f < NF; f++) val[f] = 0.0;
  const bool no_sines = pt_no_sines(q);
  double cm = 1.0, sm = 0.0;  // cos(m phi), sin(m phi), m = k / 2 (COSSIN)
  for (int k = 0; k < D.nc2; k++) {
    const double phik = (k & 1) ? sm : cm;
    if (k & 1) {
      const double cn = cm * q.cp - sm * q.sp;
      sm = sm * q.cp + cm * q.sp;
      cm = cn;
    }
    if (k == 1 || !live[k] || (no_sines && (k & 1))) continue;  // sin(0), or no coefficient
    const double* th = TH + a.slot[pt_theta_kind(__ldg(tb + k))] * D.nc1 * PT_THREADS;
    double acc[NF];
#pragma unroll
    for (int f = 0; f < NF; f++) acc[f] = 0.0;
    for (int j = 0; j < D.nc1; j++) {
      const int br = __ldg(rb + j * D.nc2 + k);
      pt_line<NF>(cs + static_cast<size_t>(k * D.nc1 + j) * D.nc0 * NF, D.nc0, T + (br == B_CHEB_ODD ? PT_THREADS : 0),
                  (br == B_CHEB ? 1 : 2) * PT_THREADS, th[j * PT_THREADS], acc);
    }
#pragma unroll
    for (int f = 0; f < NF; f++) val[f] = fma(phik, acc[f], val[f]);
  }
#pragma unroll
  for (int f = 0; f < NF; f++) out[a.field[a.first[g] + f] * npts + p] = val[f];
}

// Many points: CTA b works on its run of 128-slot chunks of `perm`, group of
// fields by group, restaging coefficients when the domain changes.
__global__ void __launch_bounds__(PT_THREADS) val_points_sorted_kernel(
    const __grid_constant__ PtArgs a, const int* __restrict__ tab, long long npts, const double* __restrict__ xyz,
    const int* __restrict__ count, const int* __restrict__ perm, int coef_doubles, int theta_rows,
    double* __restrict__ out) {
  extern __shared__ __align__(16) double pt_sm[];
  __shared__ int first_chunk[PT_MAX_DOM + 1], live[2048 / PT_MAX_NR];
  double* cs = pt_sm;
  const int tid = threadIdx.x;
  double* TH = pt_sm + coef_doubles + tid;                    // [kind][j] of this thread's point
  double* T = TH + static_cast<size_t>(theta_rows) * PT_THREADS;  // [n]
  if (tid <= a.ndom) first_chunk[tid] = pt_first_slot(count, tid) / PT_THREADS;
  __syncthreads();
  const int chunks = first_chunk[a.ndom];
  const int per = (chunks + gridDim.x - 1) / gridDim.x;
  const int c0 = blockIdx.x * per, c1 = min(chunks, c0 + per);
  for (int g = 0; g < a.ngroups; g++) {
    int staged = -1;
    const int nf = a.size[g];
    for (int c = c0; c < c1; c++) {
      int dd = 0;
      while (first_chunk[dd + 1] <= c) dd++;
      const PtDom& D = a.d[dd];
      if (dd != staged) {
        __syncthreads();
        for (int k = tid; k < D.nc2; k += PT_THREADS) live[k] = 0;
        __syncthreads();
        const int n = D.nc0 * D.nc1 * D.nc2;
        for (int f = 0; f < nf; f++) {
          const double* src = a.cf[a.field[a.first[g] + f]][dd];
          for (int e = tid; e < n; e += PT_THREADS) {
            const int k = e % D.nc2, ij = e / D.nc2, j = ij % D.nc1, i = ij / D.nc1;
            const double v = src ? __ldg(src + e) : 0.0;
            cs[(static_cast<size_t>(k * D.nc1 + j) * D.nc0 + i) * nf + f] = v;
            if (v != 0.0) live[k] = 1;  // NaN counts
          }
        }
        __syncthreads();
        staged = dd;
      }
      const int p = perm[static_cast<long long>(c) * PT_THREADS + tid];
      if (p < 0) continue;
      double x, y, z, r;
      pt_locate(a, xyz, p, x, y, z, r);
      const PtPos q = pt_position(D, x, y, z, r);
      pt_chebyshev(q.xi, D.ncheb, T, PT_THREADS);
      const int row = D.nc1 * PT_THREADS;
#pragma unroll
      for (int odd = 0; odd < 2; odd++) {
        const int sc = a.slot[odd], ss = a.slot[2 + odd];
        if (sc >= 0 || ss >= 0)
          pt_theta(q, odd, D.nc1, sc >= 0 ? TH + sc * row : nullptr, ss >= 0 ? TH + ss * row : nullptr, PT_THREADS);
      }
      switch (nf) {
        case 1: pt_group<1>(a, g, dd, D, q, cs, tab, live, T, TH, npts, p, out); break;
        case 2: pt_group<2>(a, g, dd, D, q, cs, tab, live, T, TH, npts, p, out); break;
        case 4: pt_group<4>(a, g, dd, D, q, cs, tab, live, T, TH, npts, p, out); break;
        default: pt_group<5>(a, g, dd, D, q, cs, tab, live, T, TH, npts, p, out); break;
      }
    }
  }
}

// Few points: PT_SUB lanes a point.  The lanes tabulate the point's Chebyshev,
// theta and phi factors, then each sums its share of the (j, k) lines from
// global memory; a fixed shuffle tree adds the shares.
__global__ void __launch_bounds__(PT_THREADS) val_points_few_kernel(const __grid_constant__ PtArgs a,
                                                                    const int* __restrict__ tab, long long npts,
                                                                    const double* __restrict__ xyz, int nr_max,
                                                                    int nt_max, double* __restrict__ out) {
  extern __shared__ __align__(16) double pt_sm[];
  constexpr int PPB = PT_THREADS / PT_SUB;  // points a CTA
  const int pt = threadIdx.x / PT_SUB, sub = threadIdx.x % PT_SUB;
  double* T = pt_sm + pt;                      // [n] at stride PPB
  double* TH = T + 2 * nr_max * PPB;           // [kind][j]
  double* PH = TH + 4 * nt_max * PPB;          // [k]
  const long long p = static_cast<long long>(blockIdx.x) * PPB + pt;
  double x, y, z, r;
  const int dd = p < npts ? pt_locate(a, xyz, p, x, y, z, r) : -1;
  const PtDom& D = a.d[dd < 0 ? 0 : dd];
  bool no_sines = false;
  if (dd >= 0) {
    const PtPos q = pt_position(D, x, y, z, r);
    no_sines = pt_no_sines(q);
    const int row = nt_max * PPB;
    if (sub == 0) pt_chebyshev(q.xi, D.ncheb, T, PPB);
    if (sub == 1) pt_theta(q, 0, D.nc1, TH, TH + 2 * row, PPB);
    if (sub == 2) pt_theta(q, 1, D.nc1, TH + row, TH + 3 * row, PPB);
    if (sub == 3) {
      double cm = 1.0, sm = 0.0;
      for (int k = 0; k < D.nc2; k++) {
        PH[k * PPB] = (k & 1) ? sm : cm;
        if (k & 1) {
          const double cn = cm * q.cp - sm * q.sp;
          sm = sm * q.cp + cm * q.sp;
          cm = cn;
        }
      }
    }
  }
  __syncwarp();
  const int lines = dd >= 0 ? D.nc1 * D.nc2 : 0;
  for (int f = 0; f < a.nfields; f++) {
    double val = 0.0;
    const double* c = dd >= 0 ? a.cf[f][dd] : nullptr;
    if (c) {
      const int* rb = tab + a.tab_off[f][dd];
      const int* tb = rb + lines;
      for (int l = sub; l < lines; l += PT_SUB) {
        const int k = l % D.nc2, j = l / D.nc2;
        if (k == 1 || (no_sines && (k & 1))) continue;
        const double phik = PH[k * PPB];
        const int br = __ldg(rb + l);
        const double* t = T + (br == B_CHEB_ODD ? PPB : 0);
        const int ts = (br == B_CHEB ? 1 : 2) * PPB;
        const double* ci = c + l;
        double rad = 0.0;
#pragma unroll 4
        for (int i = 0; i < D.nc0; i++) rad = fma(__ldg(ci + static_cast<size_t>(i) * lines), t[i * ts], rad);
        val = fma(phik * TH[(pt_theta_kind(__ldg(tb + k)) * nt_max + j) * PPB], rad, val);
      }
    }
#pragma unroll
    for (int o = PT_SUB / 2; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
    if (sub == 0 && p < npts) out[f * npts + p] = dd >= 0 ? val : nan("");
  }
}

}  // namespace

void fields_val_points(Context* ctx, const std::vector<const Field*>& fields, long long npts, const double* d_xyz,
                       double* d_out) {
  if (fields.empty() || npts <= 0) return;
  if (static_cast<int>(fields.size()) > PT_MAX_FIELDS)
    throw KdError(KD_ERR_ARG, "val_points: too many fields in one call");
  const Space* sp = fields[0]->sp;
  if (sp->ndom() > PT_MAX_DOM) throw KdError(KD_ERR_UNSUPPORTED, "val_points: too many domains");
  PtArgs a{};
  a.ndom = sp->ndom();
  a.nfields = static_cast<int>(fields.size());
  a.cx = sp->dom(0).center[0];
  a.cy = sp->dom(0).center[1];
  a.cz = sp->dom(0).center[2];
  for (int d = 0; d < a.ndom; d++) {
    const Domain& dm = sp->dom(d);
    a.d[d].type = dm.type;
    a.d[d].alpha = dm.alpha;
    a.d[d].beta = dm.beta;
    a.d[d].rin = dm.inner_radius();
    a.d[d].rout = dm.outer_radius();
    a.d[d].nc0 = dm.nc[0];
    a.d[d].nc1 = dm.nc[1];
    a.d[d].nc2 = dm.nc[2];
    a.d[d].ncheb = dm.nc[0];
  }
  // basis tables, and fields grouped by them
  std::vector<int> tab;
  std::vector<std::vector<int>> bases(a.nfields);
  for (int f = 0; f < a.nfields; f++) {
    if (fields[f]->sp != sp) throw KdError(KD_ERR_ARG, "val_points: fields on different spaces");
    for (int d = 0; d < a.ndom; d++) {
      const Domain& dm = sp->dom(d);
      const Field::PerDom& pd = fields[f]->d[d];
      a.tab_off[f][d] = static_cast<int>(tab.size());
      const Base b = (pd.zero || !pd.base.def) ? dm.std_base() : pd.base;
      if (b.p != KD_COSSIN) throw KdError(KD_ERR_UNSUPPORTED, "val_points: phi basis other than COSSIN");
      for (int code : b.r) {
        if (code != KD_CHEB && code != KD_CHEB_EVEN && code != KD_CHEB_ODD)
          throw KdError(KD_ERR_UNSUPPORTED, "val_points: radial basis not handled");
        // (a file may hold any of them in any domain)
        if (code != KD_CHEB) a.d[d].ncheb = 2 * dm.nc[0];
      }
      for (int code : b.t)
        if (code != KD_COS_EVEN && code != KD_COS_ODD && code != KD_SIN_EVEN && code != KD_SIN_ODD)
          throw KdError(KD_ERR_UNSUPPORTED, "val_points: theta basis not handled");
      tab.insert(tab.end(), b.r.begin(), b.r.end());
      tab.insert(tab.end(), b.t.begin(), b.t.end());
      bases[f].insert(bases[f].end(), b.r.begin(), b.r.end());
      bases[f].insert(bases[f].end(), b.t.begin(), b.t.end());
    }
  }
  int nr_max = 0, nt_max = 0, np_max = 0;
  long long nc_max = 0;
  for (int d = 0; d < a.ndom; d++) {
    nr_max = std::max(nr_max, a.d[d].nc0);
    nt_max = std::max(nt_max, a.d[d].nc1);
    np_max = std::max(np_max, a.d[d].nc2);
    nc_max = std::max(nc_max, static_cast<long long>(a.d[d].nc0) * a.d[d].nc1 * a.d[d].nc2);
  }
  cudaStream_t s = ctx->stream();
  DeviceArena& ar = ctx->scratch();
  const size_t mark = ar.mark();
  // coefficients: the field's own, or transformed here in packed launches
  {
    std::vector<KdItem> items;
    std::vector<int> ones;
    for (int f = 0; f < a.nfields; f++)
      for (int d = 0; d < a.ndom; d++) {
        const Domain& dm = sp->dom(d);
        const Field::PerDom& pd = fields[f]->d[d];
        a.cf[f][d] = nullptr;
        if (pd.zero) continue;
        DVal v = fields[f]->val(d);
        if (v.in_coef) {
          a.cf[f][d] = v.cf;
          continue;
        }
        double* dst = ar.alloc_doubles(static_cast<size_t>(dm.ncoefs()));
        items.push_back(make_item(coef_plan(*ctx, v.base, dm.np, dm.nc, false, 1), v.c, dst, dm.np, dm.npts(),
                                  dm.ncoefs(), 1.0));
        ones.push_back(1);
        a.cf[f][d] = dst;
      }
    if (!items.empty()) ctx->run_items(items, ones);
  }
  const int* d_tab = ctx->table(tab);
  // shared memory of the sorted kernel: coefficients of the widest group that
  // leaves room, theta tables, Chebyshev table
  int kinds = 0;
  {
    bool has[4] = {};
    for (int f = 0; f < a.nfields; f++)
      for (int d = 0; d < a.ndom; d++)
        for (int k = 0; k < a.d[d].nc2; k++) {
          const int bt = tab[a.tab_off[f][d] + a.d[d].nc1 * a.d[d].nc2 + k];
          has[bt == B_COS_EVEN ? 0 : bt == B_COS_ODD ? 1 : bt == B_SIN_EVEN ? 2 : 3] = true;
        }
    for (int q = 0; q < 4; q++) a.slot[q] = has[q] ? kinds++ : -1;
  }
  const long long tables = static_cast<long long>(PT_THREADS) * (kinds * nt_max + 2 * nr_max);
  const long long room = 226 * 1024 / 8 - tables;
  // (the even rounding below takes one more)
  const int widest = static_cast<int>(std::min<long long>(5, (room - 1) / nc_max));
  const bool fits = nr_max <= PT_MAX_NR && np_max <= 2048 / PT_MAX_NR && npts <= (1LL << 31) - 4096;
  const size_t few_smem = sizeof(double) * (PT_THREADS / PT_SUB) * (2 * static_cast<size_t>(nr_max) + 4 * nt_max + np_max);
  if (fits && npts < PT_FEW && few_smem <= 48 * 1024) {
    ProfScope ps(ctx, Context::PROF_LINE_PASS, 0.0);
    const int ppb = PT_THREADS / PT_SUB;
    val_points_few_kernel<<<static_cast<int>((npts + ppb - 1) / ppb), PT_THREADS, few_smem, s>>>(
        a, d_tab, npts, d_xyz, nr_max, nt_max, d_out);
    ctx->launches++;
  } else if (fits && widest >= 1) {
    int used = 0;
    std::vector<char> done(a.nfields, 0);
    for (int f = 0; f < a.nfields; f++) {
      if (done[f]) continue;
      std::vector<int> same;
      for (int h = f; h < a.nfields; h++)
        if (!done[h] && bases[h] == bases[f]) {
          same.push_back(h);
          done[h] = 1;
        }
      for (size_t at = 0; at < same.size();) {
        const int left = std::min<int>(widest, static_cast<int>(same.size() - at));
        const int n = left >= 4 ? left : left >= 2 ? 2 : 1;  // 1, 2, 4 or 5
        a.first[a.ngroups] = used;
        a.size[a.ngroups++] = n;
        for (int q = 0; q < n; q++) a.field[used++] = same[at++];
      }
    }
    int nf_max = 1;
    for (int g = 0; g < a.ngroups; g++) nf_max = std::max(nf_max, a.size[g]);
    const int coef_doubles = static_cast<int>((nc_max * nf_max + 1) & ~1LL);
    const size_t smem = sizeof(double) * (static_cast<size_t>(coef_doubles) + static_cast<size_t>(tables));
    static std::once_flag attr;
    std::call_once(attr, [] {
      cuda_check(cudaFuncSetAttribute(val_points_sorted_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024),
                 "cudaFuncSetAttribute(val_points)");
    });
    const long long slots = npts + static_cast<long long>(a.ndom) * PT_THREADS;
    int* perm = static_cast<int*>(ar.alloc_bytes(sizeof(int) * static_cast<size_t>(slots)));
    int* cnt = static_cast<int*>(ar.alloc_bytes(sizeof(int) * 2 * (PT_MAX_DOM + 1)));
    cuda_check(cudaMemsetAsync(cnt, 0, sizeof(int) * 2 * (PT_MAX_DOM + 1), s), "memset counts");
    cuda_check(cudaMemsetAsync(perm, 0xff, sizeof(int) * static_cast<size_t>(slots), s), "memset slots");
    const int nb = static_cast<int>((npts + PT_BLOCK_POINTS - 1) / PT_BLOCK_POINTS);
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, val_points_sorted_kernel, PT_THREADS, smem),
               "occupancy (val_points)");
    ProfScope ps(ctx, Context::PROF_LINE_PASS, 0.0);
    pt_count<<<nb, 256, 0, s>>>(a, npts, d_xyz, cnt);
    pt_scatter<<<nb, 256, 0, s>>>(a, npts, d_xyz, cnt, cnt + PT_MAX_DOM + 1, perm, d_out);
    val_points_sorted_kernel<<<152 * std::max(per_sm, 1), PT_THREADS, smem, s>>>(a, d_tab, npts, d_xyz, cnt, perm,
                                                                                  coef_doubles, kinds * nt_max, d_out);
    ctx->launches += 3;
  } else {
    long long nb = (npts + 255) / 256;
    if (nb > 152LL * 16) nb = 152LL * 16;
    ProfScope ps(ctx, Context::PROF_LINE_PASS, 0.0);
    val_points_kernel<<<static_cast<int>(nb), 256, 0, s>>>(a, d_tab, npts, d_xyz, d_out);
    ctx->launches++;
  }
  cuda_check(cudaGetLastError(), "val_points kernels");
  // the coefficients are read by the kernel: keep them until it ran
  cuda_check(cudaStreamSynchronize(s), "sync val_points");
  ar.release_to(mark);
}

}  // namespace kd
