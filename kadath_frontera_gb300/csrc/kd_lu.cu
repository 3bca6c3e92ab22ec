// Dense LU with partial pivoting (column-major) and triangular solves.
// Blocked right-looking factorisation, per panel of jb <= 96 columns (192 as two
// halves where the update is better off with k = 192):
//   panel    the rows of the panel held in shared memory, by one 16-CTA cluster
//            (FP32), by a cooperative kernel over the whole GPU with one exchange
//            a column, or, in a kept pivot order, without any search;
//   swaps    the panel's row exchanges as one list of row moves, applied
//            to the other columns by one warp per column;
//   TRSM     U12 = L11^{-1} A12 with L11 staged in shared memory;
//   update   A22 -= L21 U12 on the tensor cores: 3xTF32 (kd_gemm_tc.cu) for the
//            mixed modes, exact slices (kd_gemm_f64.cu) for FP64; the library's
//            GEMM for small FP64 updates and the FP32 mode.
// Solves are one launch a sweep, with inverses of the 64 x 64 diagonal blocks.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "kd_gemm_tc.hpp"
#include "kd_lu.hpp"

namespace kd {

namespace {

// A CTA's candidate for one column of a grid panel.
struct PanelRecord {
  unsigned long long key;  // of its modulus
  unsigned long long row;
};

// U12 = L11^-1 A12 (L11 unit lower, jb <= 96) for FP64 factors, 16 columns a
// CTA.  By 32-row chunks: the chunk's own triangle with 8 lanes a column (rows
// l, l + 8, l + 16, l + 24; each finished entry broadcast by a shuffle), then
// its products with the rows below as a register-tiled product, every entry
// summed in column order as by plain substitution.
// Bound: the FP64 pipe (4,560 multiply-adds a column); three CTAs an SM.  One
// thread a column on 64-column CTAs, as before, was bound by its chain of
// dependent multiply-adds instead (0.23 ms at any width).
constexpr int TD_COLS = 16, TD_THREADS = 128, TD_LD = 97;
constexpr size_t TD_SMEM = sizeof(double) * (6 * 32 * 32 + TD_COLS * TD_LD);
__global__ void __launch_bounds__(TD_THREADS) trsm_chunk_f64(double* __restrict__ A, long long ld, int j0, int jb,
                                                             int c0, int c1) {
  extern __shared__ __align__(16) double td_sm[];
  double* LT = td_sm;                // block (rb, kb) of L11, transposed: [k][r]
  double* X = td_sm + 6 * 32 * 32;   // X[c * TD_LD + row]
  const int tid = threadIdx.x, cb = c0 + blockIdx.x * TD_COLS;
  for (int blk = 0; blk < 6; blk++) {
    const int rb = blk < 1 ? 0 : blk < 3 ? 1 : 2, kb = blk - rb * (rb + 1) / 2;
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int e = tid + u * TD_THREADS, r = rb * 32 + (e & 31), k = kb * 32 + (e >> 5);
      v[u] = (r < jb && k < jb) ? A[static_cast<long long>(j0 + k) * ld + j0 + r] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; u++) LT[blk * 1024 + tid + u * TD_THREADS] = v[u];
  }
  for (int e = tid; e < TD_COLS * 96; e += TD_THREADS) {
    const int c = e / 96, i = e - c * 96;
    X[c * TD_LD + i] = (i < jb && cb + c < c1) ? A[static_cast<long long>(cb + c) * ld + j0 + i] : 0.0;
  }
  __syncthreads();
  const int l = tid & 7, col = tid >> 3, lane = tid & 31;
  for (int c = 0; c < 3; c++) {
    if (c * 32 >= jb) break;
    {
      const double* L = LT + (c * (c + 1) / 2 + c) * 1024;
      double* xc = X + col * TD_LD + c * 32;
      double x[4];
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = xc[l + 8 * q];
#pragma unroll
      for (int k = 0; k < 31; k++) {
        const double xk = __shfl_sync(0xffffffffu, x[k >> 3], (lane & 24) | (k & 7));
#pragma unroll
        for (int q = k >> 3; q < 4; q++)
          if (q > (k >> 3) || l > (k & 7)) x[q] = fma(-L[k * 32 + l + 8 * q], xk, x[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) xc[l + 8 * q] = x[q];
    }
    __syncthreads();
    const double* xk = X + c * 32;
    if (c == 0) {  // rows 32..95: 4 rows x 2 columns a thread
      const int r = (tid & 15) * 4, cc = (tid >> 4) * 2, rb = 1 + (r >> 5);
      const double* L = LT + (rb * (rb + 1) / 2) * 1024 + (r & 31);
      double acc[2][4];
#pragma unroll
      for (int u = 0; u < 2; u++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[u][q] = X[(cc + u) * TD_LD + 32 + r + q];
#pragma unroll 4
      for (int k = 0; k < 32; k++) {
        const double2 a = *reinterpret_cast<const double2*>(L + k * 32), b = *reinterpret_cast<const double2*>(L + k * 32 + 2);
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const double x = xk[(cc + u) * TD_LD + k];
          acc[u][0] = fma(-a.x, x, acc[u][0]);
          acc[u][1] = fma(-a.y, x, acc[u][1]);
          acc[u][2] = fma(-b.x, x, acc[u][2]);
          acc[u][3] = fma(-b.y, x, acc[u][3]);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; u++)
#pragma unroll
        for (int q = 0; q < 4; q++) X[(cc + u) * TD_LD + 32 + r + q] = acc[u][q];
    } else if (c == 1) {  // rows 64..95: 4 rows x 1 column a thread
      const int r = (tid & 7) * 4, cc = tid >> 3;
      const double* L = LT + (2 * 3 / 2 + 1) * 1024 + r;
      double acc[4];
#pragma unroll
      for (int q = 0; q < 4; q++) acc[q] = X[cc * TD_LD + 64 + r + q];
#pragma unroll 4
      for (int k = 0; k < 32; k++) {
        const double2 a = *reinterpret_cast<const double2*>(L + k * 32), b = *reinterpret_cast<const double2*>(L + k * 32 + 2);
        const double x = xk[cc * TD_LD + k];
        acc[0] = fma(-a.x, x, acc[0]);
        acc[1] = fma(-a.y, x, acc[1]);
        acc[2] = fma(-b.x, x, acc[2]);
        acc[3] = fma(-b.y, x, acc[3]);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) X[cc * TD_LD + 64 + r + q] = acc[q];
    }
    __syncthreads();
  }
  for (int e = tid; e < TD_COLS * 96; e += TD_THREADS) {
    const int c = e / 96, i = e - c * 96;
    if (i < jb && cb + c < c1) A[static_cast<long long>(cb + c) * ld + j0 + i] = X[c * TD_LD + i];
  }
}

// U12 = L11^-1 A12 (L11 unit lower, jb <= 96) for FP32 factors, 128 columns
// per CTA of 512 threads.  L11, transposed (LT[k][i] = l_ik), and the CTA's
// 96 x 128 column tile X go through shared memory.  The solve runs by 32-row
// chunks: a chunk's own triangle by columns (one thread per column, threads
// 0..127), and its products with the finished chunks as a register-tiled
// product (8 rows x 4 columns per thread, 128 threads).  Those products are
// split by k: right after chunk 0's triangle, chunks 1 and 2 take off their
// products with chunk 0 at the same time (threads 0..127 and 128..255).
// Every element still receives its multiply-adds in increasing k: the
// operations of a column-by-column forward substitution, in its order.  All
// 512 threads stage the tile (every load of a thread in flight before its
// stores) and write it back.
constexpr int TS_THREADS = 512;
constexpr int TS_COLS = 128;
constexpr int TS_LDL = 100;  // row stride of LT: 16-byte aligned rows
constexpr int TS_LDX = 132;  // row stride of X: 16-byte aligned rows
constexpr size_t TS_SMEM = sizeof(float) * (96 * TS_LDL + 96 * TS_LDX);

// X[r][c] -= sum_{k0 <= k < k1} l_rk X[k][c] (k in order) for the rows
// r = R0 + 8 tr + a and columns c = 4 tc + b of thread t = 32 tr + tc < 128.
__device__ __forceinline__ void ts_cross(const float* __restrict__ LT, float* __restrict__ X, int R0, int k0, int k1,
                                         int t) {
  const int tr = t >> 5, tc = t & 31;
  const int r0 = R0 + 8 * tr;
  float acc[8][4];
#pragma unroll
  for (int a = 0; a < 8; a++) {
    const float4 q = *reinterpret_cast<const float4*>(X + (r0 + a) * TS_LDX + 4 * tc);
    acc[a][0] = q.x;
    acc[a][1] = q.y;
    acc[a][2] = q.z;
    acc[a][3] = q.w;
  }
#pragma unroll 4
  for (int k = k0; k < k1; k++) {
    const float4 la = *reinterpret_cast<const float4*>(LT + k * TS_LDL + r0);  // the same for the whole warp
    const float4 lb = *reinterpret_cast<const float4*>(LT + k * TS_LDL + r0 + 4);
    const float4 y = *reinterpret_cast<const float4*>(X + k * TS_LDX + 4 * tc);
    const float l[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
    const float yy[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b] = fmaf(-l[a], yy[b], acc[a][b]);
  }
#pragma unroll
  for (int a = 0; a < 8; a++)
    *reinterpret_cast<float4*>(X + (r0 + a) * TS_LDX + 4 * tc) = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
}

// The 32 x 32 unit lower triangle of chunk R0 for column t (< 128).
__device__ __forceinline__ void ts_diag(const float* __restrict__ LT, float* __restrict__ X, int R0, int t) {
  float x[32];
#pragma unroll
  for (int j = 0; j < 32; j++) x[j] = X[(R0 + j) * TS_LDX + t];
#pragma unroll
  for (int kk = 0; kk < 32; kk++) {
    const float y = x[kk];
    const float* lrow = LT + (R0 + kk) * TS_LDL + R0;
#pragma unroll
    for (int j = 0; j < 32; j++)
      if (j > kk) x[j] = fmaf(-lrow[j], y, x[j]);
  }
#pragma unroll
  for (int j = 0; j < 32; j++) X[(R0 + j) * TS_LDX + t] = x[j];
}

__global__ void __launch_bounds__(TS_THREADS) trsm_chunk_f32(float* __restrict__ A, long long ld, int j0, int jb,
                                                             int c0, int c1) {
  extern __shared__ __align__(16) float ts_sm[];
  float* LT = ts_sm;                // LT[k * TS_LDL + i] = l_ik (i > k, i < jb), zero elsewhere
  float* X = ts_sm + 96 * TS_LDL;  // X[i * TS_LDX + c]
  const int tid = threadIdx.x;
  const int cb = c0 + blockIdx.x * TS_COLS;
  {
    constexpr int NL = (96 * 96 + TS_THREADS - 1) / TS_THREADS, NX = 96 * TS_COLS / TS_THREADS;
    float v[NL], w[NX];
#pragma unroll
    for (int u = 0; u < NL; u++) {
      const int e = u * TS_THREADS + tid;
      const int i = e % 96, k = e / 96;  // down the columns: coalesced reads
      v[u] = (e < 96 * 96 && i < jb && k < i) ? A[static_cast<long long>(j0 + k) * ld + j0 + i] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < NX; u++) {
      const int e = u * TS_THREADS + tid;
      const int i = e % 96, col = cb + e / 96;
      w[u] = (i < jb && col < c1) ? A[static_cast<long long>(col) * ld + j0 + i] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < NL; u++) {
      const int e = u * TS_THREADS + tid;
      if (e < 96 * 96) LT[(e / 96) * TS_LDL + e % 96] = v[u];
    }
#pragma unroll
    for (int u = 0; u < NX; u++) {
      const int e = u * TS_THREADS + tid;
      X[(e % 96) * TS_LDX + e / 96] = w[u];
    }
  }
  __syncthreads();
  const int nch = (jb + 31) / 32;
  // chunk by chunk: its own triangle, then its products with every later chunk,
  // 128 threads each; one copy of the unrolled code for all chunks, so less to
  // fetch (12,331 rows in a reused order 15.75 -> 15.64 ms)
#pragma unroll 1
  for (int c = 0; c < nch; c++) {
    if (tid < 128) ts_diag(LT, X, 32 * c, tid);
    __syncthreads();
    const int r = c + 1 + (tid >> 7);
    if (r < nch) ts_cross(LT, X, 32 * r, 32 * c, 32 * c + 32, tid & 127);
    __syncthreads();
  }
  // write-back: four consecutive rows of one column per thread and step, as
  // one 16-byte store where the rows start 16-byte aligned
  const bool vec = (reinterpret_cast<unsigned long long>(A) & 15) == 0 && (ld & 3) == 0 && (j0 & 3) == 0;
#pragma unroll
  for (int q = 0; q < 96 * TS_COLS / 4 / TS_THREADS; q++) {
    const int e = tid + q * TS_THREADS;
    const int i = 4 * (e % 24), c = e / 24;
    const int col = cb + c;
    if (col < c1 && i < jb) {
      float* dst = A + static_cast<long long>(col) * ld + j0 + i;
      const float4 r = make_float4(X[i * TS_LDX + c], X[(i + 1) * TS_LDX + c], X[(i + 2) * TS_LDX + c],
                                   X[(i + 3) * TS_LDX + c]);
      if (vec && i + 3 < jb) {
        *reinterpret_cast<float4*>(dst) = r;
      } else {
        dst[0] = r.x;
        if (i + 1 < jb) dst[1] = r.y;
        if (i + 2 < jb) dst[2] = r.z;
        if (i + 3 < jb) dst[3] = r.w;
      }
    }
  }
}

// ---- equilibration of the FP32 working copy (mixed modes) --------------
// Row scales r_i = 2^-round(log2 max_j |A_ij|), then column scales
// c_j = 2^-round(log2 max_i |r_i A_ij|): powers of two, so scaling is exact
// and only the FP32 rounding remains.  The factors are those of
// D_r A D_c; the preconditioner is M^-1 b = D_c (LU)^-1 (D_r b).
__device__ __forceinline__ double pow2_inverse(double m) {
  if (!(m > 0.0) || !isfinite(m)) return 1.0;
  int e;
  frexp(m, &e);  // m = f 2^e, f in [0.5, 1)
  return ldexp(1.0, 1 - e);  // 2^-(e-1): scaled max in [1, 2)
}

// The equilibration and the FP32 working copy move powers of two about: on
// integers, because an FP64 multiply, compare or maximum takes 16 cycles of an
// SM per warp (the copy of a 12,331 x 12,331 matrix took 1.5 ms with five FP64
// instructions an entry, 0.3 ms of which are its bytes).
// |v| as bits (ordered like it), 0 for NaN.
__device__ __forceinline__ unsigned long long modulus_bits(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffull;
  return b > 0x7ff0000000000000ull ? 0ull : b;
}
// v * 2^k, exact like the product.  The rare case is a call, not inlined: the
// loops below hold sixteen of them.
__device__ __noinline__ double times_pow2_rare(double v, int k) { return scalbn(v, k); }  // subnormal, Inf, NaN, out of range
__device__ __forceinline__ double times_pow2(double v, int k) {
  const int hi = __double2hiint(v), lo = __double2loint(v);
  const int e = (hi >> 20) & 0x7ff;
  if (static_cast<unsigned>(e - 1) < 0x7feu && static_cast<unsigned>(e + k - 1) < 0x7feu)
    return __hiloint2double(hi + (k << 20), lo);
  if (((hi & 0x7fffffff) | lo) == 0) return v;
  return times_pow2_rare(v, k);
}
// v * 2^k rounded to FP32: where the result is a normal float, the top 23
// mantissa bits rounded to nearest even by hand, since the conversion also
// runs at the FP64 rate (it bounded the copy: 0.65 ms, its bytes 0.28 ms).
__device__ __noinline__ float pow2_to_float_rare(double v, int k) { return static_cast<float>(scalbn(v, k)); }
__device__ __forceinline__ float pow2_to_float(double v, int k) {
  const unsigned hi = static_cast<unsigned>(__double2hiint(v)), lo = static_cast<unsigned>(__double2loint(v));
  const int e = static_cast<int>((hi >> 20) & 0x7ffu), ef = e + k - 1023 + 127;  // the float's exponent field
  if (static_cast<unsigned>(e - 1) < 0x7feu && static_cast<unsigned>(ef - 1) < 0xfeu) {
    const unsigned f = (hi & 0x80000000u) | (static_cast<unsigned>(ef) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
    // the 29 bits cut off, against half a unit: up if above, or equal and f odd
    return __uint_as_float(f + (((lo & 0x1fffffffu) + (f & 1u) > 0x10000000u) ? 1u : 0u));
  }
  if (((hi & 0x7fffffffu) | lo) == 0u) return __uint_as_float(hi);
  return pow2_to_float_rare(v, k);
}
// k of a scale 2^k
__device__ __forceinline__ int pow2_exponent(double s) {
  return ((__double2hiint(s) >> 20) & 0x7ff) - 1023;
}

// Maxima of |A_ij| over column chunks, merged with atomicMax on the bit
// patterns of non-negative doubles (order-independent, deterministic).
__global__ void row_absmax_kernel(const double* __restrict__ A, long long ld, int N, int chunk,
                                  unsigned long long* __restrict__ rmax) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int c0 = blockIdx.y * chunk;
  const int c1 = (c0 + chunk < N) ? c0 + chunk : N;
  unsigned long long m = 0;
  int j = c0;
  for (; j + 8 <= c1; j += 8) {
    unsigned long long v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = modulus_bits(A[static_cast<long long>(j + u) * ld + i]);
#pragma unroll
    for (int u = 0; u < 8; u++) m = max(m, v[u]);
  }
  for (; j < c1; j++) m = max(m, modulus_bits(A[static_cast<long long>(j) * ld + i]));
  atomicMax(rmax + i, m);
}

__global__ void row_scale_kernel(const unsigned long long* __restrict__ rmax, int N, double* __restrict__ rs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) rs[i] = pow2_inverse(__longlong_as_double(static_cast<long long>(rmax[i])));
}

// One CTA per column: c_j from max_i |r_i A_ij|, then the scaled FP32 column,
// its rows in the order perm when one is given.  rs null: no scales.  The
// converted column is put in order in shared memory where it fits (KEEP): rows
// gathered from global memory cost a 32-byte sector each.  Memory's share of
// 12,331 rows is 0.28 ms; measured 0.51 ms in order and 0.78 ms permuted (the
// column kept as doubles, half as many CTAs an SM: 1.9 ms; FP64 products and
// comparisons and a global gather: 1.5 ms each).
constexpr int SC_THREADS = 512;
constexpr size_t SC_MAX_SMEM = 220 * 1024;
template <bool KEEP>
__global__ void __launch_bounds__(SC_THREADS) scale_convert_kernel(const double* __restrict__ A, long long lda,
                                                                   const double* __restrict__ rs, int N,
                                                                   double* __restrict__ cs, float* __restrict__ B,
                                                                   long long ldb, const int* __restrict__ perm) {
  extern __shared__ float kept[];  // the converted column, rows in A's order
  __shared__ unsigned long long red[SC_THREADS / 32];
  constexpr int U = 8;
  const int j = blockIdx.x;
  const double* col = A + static_cast<long long>(j) * lda;
  int kc = 0;
  if (rs) {
    unsigned long long m = 0;
    for (int i0 = threadIdx.x; i0 < N; i0 += U * SC_THREADS) {
      double v[U], r[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u * SC_THREADS;
        v[u] = i < N ? col[i] : 0.0;
        r[u] = i < N ? rs[i] : 1.0;
      }
#pragma unroll
      for (int u = 0; u < U; u++) m = max(m, modulus_bits(times_pow2(v[u], pow2_exponent(r[u]))));
    }
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < SC_THREADS / 32; w++) m = max(m, red[w]);
    const double c = pow2_inverse(__longlong_as_double(static_cast<long long>(m)));
    if (threadIdx.x == 0) cs[j] = c;
    kc = pow2_exponent(c);
  }
  float* out = B + static_cast<long long>(j) * ldb;
  for (int i0 = threadIdx.x; i0 < N; i0 += U * SC_THREADS) {
    double v[U], r[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * SC_THREADS;
      const int p = (!KEEP && perm && i < N) ? perm[i] : i;
      v[u] = i < N ? col[p] : 0.0;
      r[u] = (rs && i < N) ? rs[p] : 1.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * SC_THREADS;
      const float f = pow2_to_float(v[u], pow2_exponent(r[u]) + kc);
      if (i < N) {
        if (KEEP)
          kept[i] = f;
        else
          out[i] = f;
      }
    }
  }
  if (KEEP) {
    __syncthreads();
    for (int i0 = threadIdx.x; i0 < N; i0 += U * SC_THREADS) {
      int p[U];
#pragma unroll
      for (int u = 0; u < U; u++) p[u] = i0 + u * SC_THREADS < N ? perm[i0 + u * SC_THREADS] : 0;
#pragma unroll
      for (int u = 0; u < U; u++)
        if (i0 + u * SC_THREADS < N) out[i0 + u * SC_THREADS] = kept[p[u]];
    }
  }
}

// ---- panel of a static-pivot factorisation (FP32, rows in pivot order) ----
// The rows of the working copy were gathered in the pivot order of an
// earlier partial-pivoting factorisation, so this panel does no row search:
// A11 = L11 U11 without exchanges, then L21 = A21 U11^-1.  Every CTA factors
// the (at most 96 x 96) diagonal block itself in shared memory -- redundant,
// but it removes every grid-wide synchronisation -- and then solves
// x U11 = a for its share of A21's rows, two rows a thread.  The last CTA to
// read the diagonal block writes L11 \ U11 back.  A zero or non-finite pivot sets
// *info (the caller then factors with partial pivoting instead).
constexpr int NP_NB = 96;
constexpr int NP_LD = NP_NB + 4;  // row stride: 16-byte aligned rows, read four elements at a time by L21
constexpr int NP_THREADS = 256;
// L21: two rows a thread.  The 16-byte reads of U11 take the shared memory four
// cycles each whatever they feed: with one row a thread they were the bound
// (35,000 cycles for 256 rows); with four a warp is alone on its scheduler and
// waits for them (36,000 for 128).  A thread's rows of the panel wait in its own
// column of dynamic shared memory, copied there while the diagonal block is
// factored.
// Measured, N = 12,331, beside the trailing update: a panel 82,000 -> 60,000
// cycles below 5,000 rows (L21 35,000 -> 23,000, diagonal block 25,000 -> 19,600,
// write-back 8,000 -> 0) and 110,000 - 180,000 -> 84,000 above 10,000; the whole
// factorisation in a reused order 17.1 -> 15.9 ms.
constexpr int NP_L21_THREADS = 192;
constexpr int NP_L21_ROWS = 2 * NP_L21_THREADS;  // rows of A21 a round
constexpr int NP_XS_BYTES = NP_NB * NP_L21_THREADS * 8;
constexpr int NP_MIN_ROWS = 128;  // of a CTA: fewer would not be faster
constexpr int NP_MAX_CTAS = 38;  // SMs outside the seven 16-CTA clusters of a GB300's trailing update: 152 - 112 = 40
static_assert(NP_THREADS == 256 && NP_NB == 96, "three 32-column blocks; 16 x 16 threads tile the trailing blocks");

// Rank-32 update of the trailing block of the diagonal block after its
// 32-column block o: a_ij -= l_ik u_kj for k = o .. o+31 in order, rows and
// columns o+32 .. 95; thread (ty, tx) holds rows ty + 16 a and columns
// tx + 16 c (a, c < R) in registers.
template <int R>
__device__ __forceinline__ void np_trailing(float* __restrict__ U, int o, int tid) {
  const int ty = tid >> 4, tx = tid & 15, b = o + 32;
  float acc[R][R];
#pragma unroll
  for (int a = 0; a < R; a++)
#pragma unroll
    for (int c = 0; c < R; c++) acc[a][c] = U[(b + ty + 16 * a) * NP_LD + b + tx + 16 * c];
#pragma unroll 4
  for (int k = 0; k < 32; k++) {
    float l[R], u[R];
#pragma unroll
    for (int a = 0; a < R; a++) l[a] = U[(b + ty + 16 * a) * NP_LD + o + k];
#pragma unroll
    for (int c = 0; c < R; c++) u[c] = U[(o + k) * NP_LD + b + tx + 16 * c];
#pragma unroll
    for (int a = 0; a < R; a++)
#pragma unroll
      for (int c = 0; c < R; c++) acc[a][c] = fmaf(-l[a], u[c], acc[a][c]);
  }
#pragma unroll
  for (int a = 0; a < R; a++)
#pragma unroll
    for (int c = 0; c < R; c++) U[(b + ty + 16 * a) * NP_LD + b + tx + 16 * c] = acc[a][c];
}

// Eight elimination steps k0 .. k0+7 of a 32 x 32 diagonal block held by
// one warp, lane l holding row l with its values shifted so that d[0] is
// column k (see panel_nopiv_kernel).  From step k0 on at most W = 32 - k0
// columns are live.  The pivot row goes to the other lanes through shared
// memory (prow, one of two in turn), 16 bytes at a time.  A multiplier is the
// quotient q = d r corrected by q (1 - p r), r about 1 / p: as accurate as the
// product with a rounded reciprocal, and without the branch of __frcp_rn, behind
// which a lone warp waits (28,000 cycles for the 96 steps).  (r, 1 - p r) enter
// for step k0 and leave for the next one; every lane works them out with the
// pivot's owner's operations from three shuffles.  Each step stores the element
// of column k that became final.
__device__ __forceinline__ float2 np_reciprocal(float p) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(p));
  return make_float2(r, fmaf(-p, r, 1.0f));
}
__device__ __forceinline__ float np_quotient(float d, float2 rp) {
  const float q = d * rp.x;
  return fmaf(q, rp.y, q);
}
template <int W>
__device__ __forceinline__ void np_diag_steps(float (&d)[32], float2& rp, float* __restrict__ urow, float* prow,
                                              int lane, int k0) {
#pragma unroll 1
  for (int k = k0; k < k0 + 8; k++) {
    float* row = prow + (k & 1) * 32;
    if (lane == k) {
#pragma unroll
      for (int j = 0; j < W; j += 4) *reinterpret_cast<float4*>(row + j) = make_float4(d[j], d[j + 1], d[j + 2], d[j + 3]);
    }
    __syncwarp();
    const float p1 = __shfl_sync(0xffffffffu, d[1], k);
    const float a0 = __shfl_sync(0xffffffffu, d[0], (k + 1) & 31), a1 = __shfl_sync(0xffffffffu, d[1], (k + 1) & 31);
    // rows up to k (the finished ones and the pivot row) take a zero
    // multiplier: their multiply-adds leave them as they are
    const float q = np_quotient(d[0], rp);
    const float lm = (lane > k) ? q : 0.0f;
    urow[k] = (lane > k) ? lm : d[0];
    rp = np_reciprocal(fmaf(-np_quotient(a0, rp), p1, a1));
    float pr[W];
#pragma unroll
    for (int j = 0; j < W; j += 4) {
      const float4 v = *reinterpret_cast<const float4*>(row + j);
      pr[j] = v.x;
      pr[j + 1] = v.y;
      pr[j + 2] = v.z;
      pr[j + 3] = v.w;
    }
#pragma unroll
    for (int j = 1; j < W; j++) d[j - 1] = fmaf(-lm, pr[j], d[j]);
    d[W - 1] = 0.0f;
  }
}

// two FP32 multiply-adds in one instruction
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__global__ void __launch_bounds__(NP_THREADS) panel_nopiv_kernel(float* __restrict__ A, long long ld, int N, int j0,
                                                                 int jb, int rows, int* __restrict__ info,
                                                                 unsigned* __restrict__ done) {
  __shared__ __align__(16) float U[NP_NB * NP_LD];
  __shared__ float rdiag[NP_NB];
  __shared__ float rpv[NP_NB];  // __frcp_rn of the pivots
  __shared__ __align__(16) float prow[2 * 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // rows first .. end of A21 are this CTA's; A's columns are 128-byte aligned
  // and padded to a multiple of 32 rows, first is a multiple of 4
  const int first = j0 + jb + blockIdx.x * rows, end = min(first + rows, N);
  const int lt = tid - (NP_THREADS - NP_L21_THREADS);  // L21's threads: all warps but the first two
  extern __shared__ __align__(16) float2 np_xs[];  // [column][thread]: two rows
  auto fetch = [&](int row) {
    if (lt >= 0 && row < end) {
      const float* src = A + static_cast<long long>(j0) * ld + row;
      for (int k = 0; k < jb; k++, src += ld)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<unsigned>(
                         __cvta_generic_to_shared(np_xs + k * NP_L21_THREADS + lt))),
                     "l"(src)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  {
    // all 36 loads of the thread in flight before the shared stores
    constexpr int NV = NP_NB * NP_NB / NP_THREADS;
    static_assert(NV * NP_THREADS == NP_NB * NP_NB, "the diagonal block splits evenly over the threads");
    float v[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
      const int e = tid + q * NP_THREADS;
      const int i = e % NP_NB, k = e / NP_NB;  // down the columns: coalesced reads
      v[q] = (i < jb && k < jb) ? A[static_cast<long long>(j0 + k) * ld + j0 + i]
                                : ((i == k) ? 1.0f : 0.0f);  // identity padding past jb
    }
#pragma unroll
    for (int q = 0; q < NV; q++) {
      const int e = tid + q * NP_THREADS;
      U[(e % NP_NB) * NP_LD + e / NP_NB] = v[q];
    }
  }
  fetch(first + 2 * lt);
  // L11 \ U11 goes back to A only when every CTA has read the diagonal block:
  // the last CTA to have read it writes it (each holds the same factors), with
  // the two warps that have no rows of L21, and resets the counter for the next
  // panel.  CTAs need not be resident together, as they are beside the trailing
  // update on a side stream.
  __shared__ int np_last;
  __syncthreads();
  if (tid == NP_THREADS - 1) {  // not of the warp that factors the diagonal block
    __threadfence();
    np_last = (atomicAdd(done, 1u) == gridDim.x - 1) ? 1 : 0;
    __threadfence();
    if (np_last) *done = 0u;
  }
  // Blocked right-looking elimination in shared memory, by 32-column
  // blocks o = 0, 32, 64 (identity padding past jb stays identity):
  //  (a) warp 0 factors the diagonal block in registers, lane l holding row
  //      o + l, no barrier;
  //  (b) threads 0..rest-1 solve the block row U12 by columns and threads
  //      128..128+rest-1 the block column L21 by rows;
  //  (c) all threads apply the rank-32 update to the trailing block, a
  //      register tile each.
  // Every element receives its multiply-adds in increasing k, like in the
  // unblocked right-looking elimination.
  // The loop over k of (a) stays rolled: one warp running unrolled
  // straight-line code once per launch waits on instruction fetch most of
  // the time.  So that registers are never indexed by k, each step shifts
  // the lane's values down by one (column o + k is always d[0]) and stores
  // the element that became final.
#pragma unroll 1
  for (int o = 0; o < NP_NB; o += 32) {
    if (warp == 0) {
      float d[32];  // row o + lane, columns o + k + j
#pragma unroll
      for (int j = 0; j < 32; j++) d[j] = U[(o + lane) * NP_LD + o + j];
      float* urow = U + (o + lane) * NP_LD + o;
      float2 rp = np_reciprocal(__shfl_sync(0xffffffffu, d[0], 0));
      np_diag_steps<32>(d, rp, urow, prow, lane, 0);
      np_diag_steps<24>(d, rp, urow, prow, lane, 8);
      np_diag_steps<16>(d, rp, urow, prow, lane, 16);
      np_diag_steps<8>(d, rp, urow, prow, lane, 24);
      __syncwarp();
      rpv[o + lane] = __frcp_rn(urow[lane]);  // the correctly rounded 1 / pivot
    }
    __syncthreads();
    const int rest = NP_NB - o - 32;
    if (rest == 0) break;
    if (tid < rest) {  // column j of U12: u_tj -= l_tk u_kj, k < t
      const int j = o + 32 + tid;
      float c[32];
#pragma unroll
      for (int t = 0; t < 32; t++) c[t] = U[(o + t) * NP_LD + j];
#pragma unroll
      for (int k = 0; k < 31; k++)
#pragma unroll
        for (int t = k + 1; t < 32; t++) c[t] = fmaf(-U[(o + t) * NP_LD + o + k], c[k], c[t]);
#pragma unroll
      for (int t = 1; t < 32; t++) U[(o + t) * NP_LD + j] = c[t];
    } else if (tid >= 128 && tid < 128 + rest) {  // row i of L21: l_ik = (a_ik - l_it u_tk, t < k) / u_kk
      const int i = o + 32 + tid - 128;
      float r[32];
#pragma unroll
      for (int k = 0; k < 32; k++) r[k] = U[i * NP_LD + o + k];
#pragma unroll
      for (int k = 0; k < 32; k++) {
        r[k] *= rpv[o + k];
#pragma unroll
        for (int t = k + 1; t < 32; t++) r[t] = fmaf(-r[k], U[(o + k) * NP_LD + o + t], r[t]);
      }
#pragma unroll
      for (int k = 0; k < 32; k++) U[i * NP_LD + o + k] = r[k];
    }
    __syncthreads();
    if (rest == 64)
      np_trailing<4>(U, o, tid);
    else
      np_trailing<2>(U, o, tid);
    __syncthreads();
  }
  if (tid < NP_NB) {
    const float d = U[tid * NP_LD + tid];
    if (tid < jb && !(fabsf(d) > 0.0f && isfinite(d)) && blockIdx.x == 0) atomicExch(info, j0 + tid + 1);
    rdiag[tid] = 1.0f / d;
  }
  __syncthreads();
  if (np_last && lt < 0) {
#pragma unroll 8
    for (int e = tid; e < NP_NB * NP_NB; e += NP_THREADS - NP_L21_THREADS) {
      const int i = e % NP_NB, k = e / NP_NB;
      if (i < jb && k < jb) A[static_cast<long long>(j0 + k) * ld + j0 + i] = U[i * NP_LD + k];
    }
  }
  // L21: x U11 = a for two rows a thread, by 32-column chunks with the chunk in
  // registers (pairs of columns): a chunk first takes off the products with the
  // finished chunks, then is solved against its 32 x 32 diagonal block of U11,
  // then written back.  The loop over the chunks stays rolled, for the
  // instruction cache's sake.
  for (int r0 = first; r0 < end; r0 += NP_L21_ROWS) {
    const int row = r0 + 2 * lt;
    if (r0 != first) fetch(row);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (lt < 0 || row >= end) continue;
    float2* xs = np_xs + lt;
#pragma unroll 1
    for (int c = 0; c < jb; c += 32) {
      unsigned long long x[2][16];
#pragma unroll
      for (int p = 0; p < 16; p++) {
        float2 lo = make_float2(0.f, 0.f), hi = lo;
        if (c + 2 * p < jb) lo = xs[(c + 2 * p) * NP_L21_THREADS];
        if (c + 2 * p + 1 < jb) hi = xs[(c + 2 * p + 1) * NP_L21_THREADS];
        x[0][p] = pack2(lo.x, hi.x);
        x[1][p] = pack2(lo.y, hi.y);
      }
#pragma unroll 4
      for (int k = 0; k < c; k++) {
        const float2 y = xs[k * NP_L21_THREADS];
        const unsigned long long n0 = pack2(-y.x, -y.x), n1 = pack2(-y.y, -y.y);
        const ulonglong2* u = reinterpret_cast<const ulonglong2*>(U + k * NP_LD + c);
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const ulonglong2 v = u[q];
          x[0][2 * q] = fma2(n0, v.x, x[0][2 * q]);
          x[0][2 * q + 1] = fma2(n0, v.y, x[0][2 * q + 1]);
          x[1][2 * q] = fma2(n1, v.x, x[1][2 * q]);
          x[1][2 * q + 1] = fma2(n1, v.y, x[1][2 * q + 1]);
        }
      }
#pragma unroll
      for (int k = 0; k < 32; k++) {
        const float rd = rdiag[c + k];
        const ulonglong2* u = reinterpret_cast<const ulonglong2*>(U + (c + k) * NP_LD + c);
        unsigned long long n[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const float2 f = unpack2(x[r][k / 2]);
          const float xk = ((k & 1) ? f.y : f.x) * rd;
          n[r] = pack2(-xk, -xk);
          if (k & 1)
            x[r][k / 2] = pack2(f.x, xk);
          else
            x[r][k / 2] = pack2(xk, fmaf(-xk, U[(c + k) * NP_LD + c + k + 1], f.y));
        }
#pragma unroll
        for (int q = (k / 2 + 1) / 2; q < 8; q++) {
          const ulonglong2 v = u[q];
#pragma unroll
          for (int r = 0; r < 2; r++) {
            if (2 * q > k / 2) x[r][2 * q] = fma2(n[r], v.x, x[r][2 * q]);
            x[r][2 * q + 1] = fma2(n[r], v.y, x[r][2 * q + 1]);
          }
        }
      }
      float* dst = A + static_cast<long long>(j0 + c) * ld + row;
#pragma unroll
      for (int p = 0; p < 16; p++) {
        const float2 f0 = unpack2(x[0][p]), f1 = unpack2(x[1][p]);
        const float2 lo = make_float2(f0.x, f1.x), hi = make_float2(f0.y, f1.y);
        if (c + 2 * p < jb) {
          *reinterpret_cast<float2*>(dst) = lo;
          xs[(c + 2 * p) * NP_L21_THREADS] = lo;
        }
        if (c + 2 * p + 1 < jb) {
          *reinterpret_cast<float2*>(dst + ld) = hi;
          xs[(c + 2 * p + 1) * NP_L21_THREADS] = hi;
        }
        dst += 2 * ld;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---- triangular solves on one right-hand side (blocked by TB rows) --------
constexpr int TB = 64;

// ipiv[j] = j: every pivot entry holds a valid row before the panels write
// theirs, so that a panel which gave up (a grid barrier wait ran out) leaves
// only in-range rows behind for the row exchanges that follow it.
__global__ void iota_kernel(int* __restrict__ v, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v[i] = i;
}

// out = P (scale b), and out = scale (P^T z); scale null: 1
__global__ void gather_perm(const double* __restrict__ b, const int* __restrict__ perm,
                            const double* __restrict__ scale, int N, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int p = perm[i];
  out[i] = scale ? b[p] * scale[p] : b[p];
}

__global__ void scatter_perm(const double* __restrict__ z, const int* __restrict__ perm,
                             const double* __restrict__ scale, int N, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int p = perm[i];
  out[p] = scale ? z[i] * scale[p] : z[i];
}

// Inverse of the unit-lower (blockIdx.y 0) or upper part (1) of one TB x TB
// diagonal block, row-major, zero padded to TB x TB: in FP64, or as (hi, lo) float
// pairs (the one or the other is null).  Eight lanes a column, rows l + 8 q each; a finished
// entry is broadcast by a shuffle and a warp starts at the first row of its four
// columns.  Bound: the FP64 pipe.  (One thread a column took 140 us, a chain of
// 2,000 dependent multiply-adds.)
constexpr int ID_THREADS = TB * 8;
template <class T>
__global__ void __launch_bounds__(ID_THREADS) invert_diag_blocks(const T* __restrict__ A, long long ld, int N,
                                                                 double* __restrict__ Linv, double* __restrict__ Uinv,
                                                                 float2* __restrict__ Linv2,
                                                                 float2* __restrict__ Uinv2) {
  extern __shared__ double sm[];
  double* D = sm;              // D[k * TB + i]: entry (i, k), rows reversed in both directions for U
  double* X = sm + TB * TB;    // X[c * (TB + 1) + i]
  __shared__ double rd[TB];
  const int blk = blockIdx.x, upper = blockIdx.y;
  const int r0 = blk * TB;
  const int n = (N - r0 < TB) ? N - r0 : TB;
  // the upper part read from its last row and column on is a lower one
  for (int e = threadIdx.x; e < TB * TB; e += ID_THREADS) {
    const int i = e % TB, k = e / TB, si = upper ? n - 1 - i : i, sk = upper ? n - 1 - k : k;
    const double v = (i < n && k < n && i >= k) ? static_cast<double>(A[static_cast<long long>(r0 + sk) * ld + r0 + si]) : 0.0;
    D[e] = v;
    if (i == k) rd[i] = (upper && i < n) ? 1.0 / v : 1.0;
  }
  __syncthreads();
  const int l = threadIdx.x & 7, c = threadIdx.x >> 3, lane = threadIdx.x & 31;
  double x[8];
#pragma unroll
  for (int q = 0; q < 8; q++) x[q] = (l + 8 * q == c) ? 1.0 : 0.0;
  const int k0 = c & ~3;  // first column of the warp
#pragma unroll
  for (int kq = 0; kq < 8; kq++) {
    if (8 * kq + 7 < k0) continue;
    for (int kr = 0; kr < 8; kr++) {
      const int k = 8 * kq + kr;
      if (k < k0) continue;
      const double xk = __shfl_sync(0xffffffffu, x[kq], (lane & 24) | kr) * rd[k];
      if (l == kr) x[kq] = xk;
#pragma unroll
      for (int q = kq; q < 8; q++)
        if (q > kq || l > kr) x[q] = fma(-D[k * TB + l + 8 * q], xk, x[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 8; q++) X[c * (TB + 1) + l + 8 * q] = x[q];
  __syncthreads();
  double* out = (upper ? Uinv : Linv) + static_cast<size_t>(blk) * TB * TB;
  float2* out2 = upper ? Uinv2 : Linv2;
  for (int e = threadIdx.x; e < TB * TB; e += ID_THREADS) {
    const int i = e / TB, k = e % TB;  // row, column of the block
    const double v = (i < n && k < n) ? (upper ? X[(n - 1 - k) * (TB + 1) + n - 1 - i] : X[k * (TB + 1) + i]) : 0.0;
    if (Linv) {
      out[e] = v;
    } else {
      const float h = static_cast<float>(v);
      out2[static_cast<size_t>(blk) * TB * TB + e] = make_float2(h, static_cast<float>(v - static_cast<double>(h)));
    }
  }
}

// y = alpha A x + beta b (FP64, column-major).  The columns are split into
// chunks: gemv_partial writes one partial sum per (chunk, row), gemv_finish
// adds them in chunk order (deterministic).  Bound: the FP64 pipe (an FP64
// multiply-add takes a warp 16 cycles of its SM: 0.26 ms for N = 12,331, the
// matrix's bytes 0.18 ms), so every SM needs the same share: 16 CTAs an SM
// while the chunks allow it (four an SM left some SMs with five: 0.31 ms).
constexpr int GEMV_ROWS = 256;
constexpr int GEMV_MAX_CHUNKS = 64;
__global__ void __launch_bounds__(GEMV_ROWS) gemv_partial(const double* __restrict__ A, long long ld, int N,
                                                          const double* __restrict__ x, int chunk,
                                                          double* __restrict__ part) {
  const int row = blockIdx.x * GEMV_ROWS + threadIdx.x;
  if (row >= N) return;
  const int c0 = blockIdx.y * chunk;
  const int c1 = (c0 + chunk < N) ? c0 + chunk : N;
  const double* a = A + static_cast<long long>(c0) * ld + row;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int k = c0;
  // eight column loads in flight per thread, then the multiply-adds
  for (; k + 7 < c1; k += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = __ldcs(a + u * ld);
    s0 = fma(v[0], x[k], s0);
    s1 = fma(v[1], x[k + 1], s1);
    s2 = fma(v[2], x[k + 2], s2);
    s3 = fma(v[3], x[k + 3], s3);
    s0 = fma(v[4], x[k + 4], s0);
    s1 = fma(v[5], x[k + 5], s1);
    s2 = fma(v[6], x[k + 6], s2);
    s3 = fma(v[7], x[k + 7], s3);
    a += 8 * ld;
  }
  for (; k + 3 < c1; k += 4) {
    s0 = fma(a[0], x[k], s0);
    s1 = fma(a[ld], x[k + 1], s1);
    s2 = fma(a[2 * ld], x[k + 2], s2);
    s3 = fma(a[3 * ld], x[k + 3], s3);
    a += 4 * ld;
  }
  for (; k < c1; k++) {
    s0 = fma(a[0], x[k], s0);
    a += ld;
  }
  part[static_cast<size_t>(blockIdx.y) * N + row] = (s0 + s1) + (s2 + s3);
}

// Eight threads a row, a share of the chunks each (50 chunks one after the
// other took 10 us, as much as the rest of a GMRES step's vector work).
constexpr int GEMV_SHARES = 8;
__global__ void __launch_bounds__(32 * GEMV_SHARES) gemv_finish(const double* __restrict__ part, int nchunk, int N,
                                                                double alpha, double beta,
                                                                const double* __restrict__ b, double* __restrict__ y) {
  __shared__ double sums[GEMV_SHARES][32];
  const int lane = threadIdx.x & 31, share = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (row < N) {
#pragma unroll 8
    for (int c = share; c < nchunk; c += GEMV_SHARES) s += part[static_cast<size_t>(c) * N + row];
  }
  sums[share][lane] = s;
  __syncthreads();
  if (share == 0 && row < N) {
#pragma unroll
    for (int k = 1; k < GEMV_SHARES; k++) s += sums[k][lane];
    y[row] = alpha * s + (b ? beta * b[row] : 0.0);
  }
}

// y = alpha A^T x + beta b: one warp per column of A (a row of A^T), the
// column read coalesced, lane partial sums reduced by xor shuffles (fixed
// order).
constexpr int GEMVT_WARPS = 2;  // small CTAs: the SMs' shares differ by a column or two
__global__ void __launch_bounds__(GEMVT_WARPS * 32) gemv_t_kernel(const double* __restrict__ A, long long ld, int N,
                                                                 const double* __restrict__ x, double alpha,
                                                                 double beta, const double* __restrict__ b,
                                                                 double* __restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int col = blockIdx.x * GEMVT_WARPS + (threadIdx.x >> 5);
  if (col >= N) return;
  const double* a = A + static_cast<long long>(col) * ld;
  double s0 = 0.0, s1 = 0.0;
  int k = lane;
  for (; k + 7 * 32 < N; k += 8 * 32) {  // eight loads in flight
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = __ldcs(a + k + 32 * u);
#pragma unroll
    for (int u = 0; u < 8; u += 2) {
      s0 = fma(v[u], x[k + 32 * u], s0);
      s1 = fma(v[u + 1], x[k + 32 * u + 32], s1);
    }
  }
  for (; k + 32 < N; k += 64) {
    s0 = fma(a[k], x[k], s0);
    s1 = fma(a[k + 32], x[k + 32], s1);
  }
  if (k < N) s0 = fma(a[k], x[k], s0);
  double sum = s0 + s1;
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) y[col] = alpha * sum + (b ? beta * b[col] : 0.0);
}

// ---- vector algebra of GMRES (fixed reduction order: bitwise reproducible) --
// Bound by latency and launches: few, and each with enough loads in flight.
constexpr int VA_THREADS = 256;
constexpr int VD_THREADS = 1024;

// The sum over a CTA of THREADS threads, in thread 0.
template <int THREADS>
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double part[THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x >= 32) return 0.0;
  v = threadIdx.x < THREADS / 32 ? part[threadIdx.x] : 0.0;
  for (int o = THREADS / 64; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// h[i] = V_i . w for the k basis vectors V_i = V + i N: one CTA per i (N =
// 12,331: 4 us; 256 threads and one load at a time 14).
__global__ void __launch_bounds__(VD_THREADS) basis_dots(const double* __restrict__ V, int N,
                                                         const double* __restrict__ w, double* __restrict__ h) {
  const double* v = V + static_cast<size_t>(blockIdx.x) * N;
  double acc = 0.0;
  int t = threadIdx.x;
  for (; t + 3 * VD_THREADS < N; t += 4 * VD_THREADS) {
    double a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      a[u] = v[t + u * VD_THREADS];
      b[u] = w[t + u * VD_THREADS];
    }
#pragma unroll
    for (int u = 0; u < 4; u++) acc = fma(a[u], b[u], acc);
  }
  for (; t < N; t += VD_THREADS) acc = fma(v[t], w[t], acc);
  acc = block_sum<VD_THREADS>(acc);
  if (threadIdx.x == 0) h[blockIdx.x] = acc;
}

// w -= sum_i h[i] V_i over the k basis vectors; with norms, also each CTA's
// sum of w^2 (added on the host, in their order).
__global__ void __launch_bounds__(VA_THREADS) basis_subtract(const double* __restrict__ V, int N, int k,
                                                             const double* __restrict__ h, double* __restrict__ w,
                                                             double* __restrict__ norms) {
  const int t = blockIdx.x * VA_THREADS + threadIdx.x;
  double v = 0.0;
  if (t < N) {
    double acc = 0.0;
#pragma unroll 4
    for (int i = 0; i < k; i++) acc = fma(h[i], V[static_cast<size_t>(i) * N + t], acc);
    v = w[t] - acc;
    w[t] = v;
  }
  if (norms) {
    v = block_sum<VA_THREADS>(v * v);
    if (threadIdx.x == 0) norms[blockIdx.x] = v;
  }
}

// Each CTA's sum of x^2.
__global__ void __launch_bounds__(VA_THREADS) sum_squares(const double* __restrict__ x, int N,
                                                          double* __restrict__ norms) {
  const int t = blockIdx.x * VA_THREADS + threadIdx.x;
  const double v = t < N ? x[t] : 0.0;
  const double sum = block_sum<VA_THREADS>(v * v);
  if (threadIdx.x == 0) norms[blockIdx.x] = sum;
}

// y = sum_i c_i V_i over k vectors, added to y when accumulate is set.
constexpr int COMBINE_MAX = 32;
struct CombineCoefs {
  double c[COMBINE_MAX];
};
__global__ void basis_combine(const double* __restrict__ V, int N, int k, const __grid_constant__ CombineCoefs c,
                              double* __restrict__ y, int accumulate) {
  const int t = blockIdx.x * VA_THREADS + threadIdx.x;
  if (t >= N) return;
  double acc = accumulate ? y[t] : 0.0;
  for (int i = 0; i < k; i++) acc = fma(c.c[i], V[static_cast<size_t>(i) * N + t], acc);
  y[t] = acc;
}

// y = alpha x, or y += alpha x when accumulate is set.
__global__ void scaled_copy(int N, double alpha, const double* __restrict__ x, double* __restrict__ y,
                            int accumulate) {
  const int t = blockIdx.x * VA_THREADS + threadIdx.x;
  if (t >= N) return;
  y[t] = accumulate ? fma(alpha, x[t], y[t]) : alpha * x[t];
}

int blocks(long long n, int t) { return static_cast<int>((n + t - 1) / t); }

double now_ms() {
  using namespace std::chrono;
  return duration<double, std::milli>(steady_clock::now().time_since_epoch()).count();
}

}  // namespace

DenseLU::DenseLU(Context* ctx) : ctx_(ctx) {
  if (cublasCreate(&blas_) != CUBLAS_STATUS_SUCCESS) throw KdError(KD_ERR_CUDA, "cublasCreate failed");
  cublasSetStream(blas_, ctx_->stream());
  cuda_check(cudaMalloc(&d_info_, sizeof(int)), "cudaMalloc(info)");
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  cuda_check(cudaDeviceGetAttribute(&nsm_, cudaDevAttrMultiProcessorCount, dev), "SM count");
  // panel exchange slots (sized for FP64 rows), barrier counter, error flag,
  // then the row-move list of one panel
  const size_t slot_bytes = sizeof(double) * (2 * 128 * static_cast<size_t>(nsm_) + 2 * 128) +
                            sizeof(PanelRecord) * 2 * static_cast<size_t>(nsm_) + 32;
  const size_t map_bytes = sizeof(int) * (1 + 4 * 128) + 60;  // + padding to 16 bytes
  cuda_check(cudaMalloc(&slot_mem_, slot_bytes + map_bytes + 32), "cudaMalloc(panel slots)");
  cuda_check(cudaMemsetAsync(slot_mem_, 0, slot_bytes + map_bytes + 32, ctx_->stream()), "memset panel slots");
  swap_map_ = reinterpret_cast<int*>(static_cast<char*>(slot_mem_) + slot_bytes);
  tri_bar_ = reinterpret_cast<unsigned*>(static_cast<char*>(slot_mem_) + slot_bytes + map_bytes);
  panel_err_ = reinterpret_cast<int*>(static_cast<char*>(slot_mem_) + slot_bytes - 16);
  np_done_ = tri_bar_ + 4;
}

DenseLU::~DenseLU() {
  cudaStreamSynchronize(ctx_->stream());
  if (blas_) cublasDestroy(blas_);
  cudaFree(A32_);
  cudaFree(ipiv_);
  cudaFree(d_info_);
  cudaFree(slot_mem_);
  cudaFree(eq_buf_);
  cudaFree(part_);
  cudaFree(work_);
  if (hproj_) cudaFreeHost(hproj_);
  cudaFree(work32_);
  cudaFree(dinv_l_);
  cudaFree(dinv_u_);
  cudaFree(dinv2_l_);
  cudaFree(dinv2_u_);
  cudaFree(group_x_l_);
  cudaFree(group_x_u_);
  cudaFree(perm_);
  cudaFree(tri_work_);
  cudaFree(bsave_);
}

void DenseLU::ensure_work(size_t n) {
  if (n > work_cap_) {
    cudaFree(work_);
    cuda_check(cudaMalloc(&work_, n * sizeof(double)), "cudaMalloc(lu work)");
    work_cap_ = n;
  }
}

// Panel of jb columns factored by one thread-block cluster: CTA r owns a
// contiguous slice of the rows [j0, N).  Per column: local arg-max, cluster
// barrier, every CTA reads the CL candidates from distributed shared memory
// and agrees on the pivot, CTA 0 swaps the two rows of the panel, cluster
// barrier, then each CTA scales and rank-1-updates its own rows.  Panel data
// stays in global memory (it fits in L2).
constexpr int PANEL_CL = 8;
constexpr int PANEL_THREADS = 1024;

template <class T>
__global__ void panel_cluster_kernel(T* __restrict__ A, long long ld, int N, int j0, int jb, int* __restrict__ ipiv,
                                     int* __restrict__ info) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double cand_v[1];
  __shared__ int cand_i[1];
  __shared__ double red_v[32];
  __shared__ int red_i[32];
  __shared__ double prow[128];  // pivot row segment (jb <= 128)
  __shared__ int s_piv;
  const int rank = static_cast<int>(cluster.block_rank());
  const int nrows = N - j0;
  const int per = (nrows + PANEL_CL - 1) / PANEL_CL;
  const int my0 = j0 + rank * per;
  const int my1 = (my0 + per < N) ? my0 + per : N;
  const int c1 = j0 + jb;
  for (int j = j0; j < c1; j++) {
    // 1. local arg-max of |A[i, j]| over my rows i >= j
    const T* col = A + static_cast<long long>(j) * ld;
    double best = -1.0;
    int bi = N;  // "no row" sentinel, larger than any row index
    int start = my0 > j ? my0 : j;
    for (int i = start + threadIdx.x; i < my1; i += blockDim.x) {
      double v = fabs(static_cast<double>(col[i]));
      if (v > best || (v == best && i < bi)) {
        best = v;
        bi = i;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      double ov = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      red_v[threadIdx.x >> 5] = best;
      red_i[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      int nw = blockDim.x >> 5;
      best = (threadIdx.x < nw) ? red_v[threadIdx.x] : -1.0;
      bi = (threadIdx.x < nw) ? red_i[threadIdx.x] : N;
      for (int o = 16; o > 0; o >>= 1) {
        double ov = __shfl_xor_sync(0xffffffffu, best, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
          best = ov;
          bi = oi;
        }
      }
      if (threadIdx.x == 0) {
        cand_v[0] = best;
        cand_i[0] = bi;
      }
    }
    __threadfence();
    cluster.sync();
    // 2. every CTA combines the CL candidates (same order, same result)
    if (threadIdx.x == 0) {
      double gb = -1.0;
      int gi = N;
      for (int r = 0; r < PANEL_CL; r++) {
        double v = *cluster.map_shared_rank(&cand_v[0], r);
        int ii = *cluster.map_shared_rank(&cand_i[0], r);
        if (v > gb || (v == gb && ii < gi)) {
          gb = v;
          gi = ii;
        }
      }
      if (gi >= N) gi = j;  // empty column below the diagonal
      s_piv = gi;
      if (rank == 0) {
        ipiv[j] = gi;
        if (!(gb > 0.0) && *info == 0) *info = j + 1;  // zero or NaN pivot
      }
    }
    __syncthreads();
    const int p = s_piv;
    // 3. CTA 0 swaps rows j and p inside the panel
    if (rank == 0 && p != j)
      for (int c = j0 + threadIdx.x; c < c1; c += blockDim.x) {
        T* cc = A + static_cast<long long>(c) * ld;
        T t = cc[j];
        cc[j] = cc[p];
        cc[p] = t;
      }
    __threadfence();
    cluster.sync();
    // 4. scale and rank-1 update of my rows below j
    for (int k = threadIdx.x; k < c1 - j; k += blockDim.x)
      prow[k] = static_cast<double>(A[static_cast<long long>(j + k) * ld + j]);
    __syncthreads();
    const double piv = prow[0];
    if (piv != 0.0) {
      // the update runs in the storage precision (FP32 for the mixed modes)
      const T inv = static_cast<T>(1.0 / piv);
      int rs = my0 > j + 1 ? my0 : j + 1;
      for (int i = rs + threadIdx.x; i < my1; i += blockDim.x) {
        T* ci = A + static_cast<long long>(j) * ld + i;
        T l = *ci * inv;
        *ci = l;
        for (int k = 1; k < c1 - j; k++) {
          T* ck = A + static_cast<long long>(j + k) * ld + i;
          *ck = fma(-l, static_cast<T>(prow[k]), *ck);
        }
      }
    }
    __syncthreads();
  }
}

// ---- panel over the whole GPU (cooperative launch) ------------------------
// CTA b owns rows [j0 + b*per, j0 + (b+1)*per) of the panel and keeps them in
// shared memory, column-major (tile[k*per + r]), for the whole panel.  Per
// column j one exchange:
//   warp 0 finds the CTA's arg-max |a(i, j)|, stores that candidate's full
//   panel row (the CTA owning row j also row j; double-buffered slots, indexed
//   by the column's parity) and its record {modulus, row}, and arrives at a
//   counter;
//   when all have arrived, one lane per CTA reads the records, every CTA
//   reduces them to the same winner (largest modulus, ties to the lowest row,
//   as idamax) and reads the winning row as the pivot row; the owner of the
//   pivot row takes row j in its place, the owner of row j takes the pivot row,
//   and each CTA scales and rank-1-updates its own rows.
// Slot reuse is safe: a CTA writes slot (jj & 1) at column jj only after all
// have arrived at column jj-1, by which every CTA has finished reading that
// slot (column jj-2).  Cross-CTA data is read with L1-bypassing loads.
// Bound: latency.  Of about 9,000 cycles a column (FP64, 40 rows a CTA) the
// update takes 2,700 (1,500 of the FP64 pipe), storing and arriving 1,350, the
// counter 1,400, records 700, the pivot row 1,100.  Moduli are compared as
// integers and reduced by redux (FP64 compares made the two arg-max 1,300
// cycles each), the reciprocal is formed once beside the row's load and not by
// every warp, and the row moves are listed here: 692 -> 405 us per FP64 panel at
// N = 8,000, FP32 panels of up to 40,081 rows 412 -> 327 us on average.  Polling
// all records instead of one counter was slower (560 us): 152 CTAs reading
// 152 records each keep the L2 slices busy that hold them.
constexpr int GP_THREADS = 512;
constexpr int GP_POLL_WARPS = 6;  // one lane a CTA: at most 192 CTAs
constexpr int GP_MIN_ROWS = 32;
constexpr size_t GP_MAX_SMEM = 200 * 1024;
constexpr size_t GP_MIN_SMEM = 8 * 1024;

template <class T>
struct PanelSlots {
  T* cand_rows;      // [2][nblk][jb]
  PanelRecord* rec;  // [2][nblk]
  T* jrow;           // [2][jb]
  int* err;          // set when a wait runs out
  unsigned long long wait_ns;  // limit of one wait (Context::grid_wait_ns)
  unsigned* count;   // arrivals, zeroed before the launch
  unsigned stall;    // added to every arrival target (Context::stall_waits)
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The modulus of v as an integer that orders the same way: 0 for NaN (never a
// pivot), else its bits + 1.  Integer compares, because an FP64 compare costs
// an FP64 instruction.
__device__ __forceinline__ unsigned long long modulus_key(double v) {
  const unsigned long long k = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffull;
  return k > 0x7ff0000000000000ull ? 0ull : k + 1;
}
__device__ __forceinline__ unsigned long long modulus_key(float v) {
  const unsigned k = __float_as_uint(v) & 0x7fffffffu;
  return k > 0x7f800000u ? 0ull : static_cast<unsigned long long>(k) + 1;
}
constexpr unsigned long long KEY_OF_ZERO = 1;

// Largest key, ties to the lowest row.
struct Candidate {
  unsigned long long key;
  int row;
};
__device__ __forceinline__ Candidate better_of(const Candidate& a, const Candidate& b) {
  return (b.key > a.key || (b.key == a.key && b.row < a.row)) ? b : a;
}
// The best of a warp, in every lane: three integer reductions in hardware.
__device__ __forceinline__ Candidate warp_best(const Candidate& c) {
  const unsigned hi = static_cast<unsigned>(c.key >> 32), lo = static_cast<unsigned>(c.key);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const int row = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? c.row : 0x7fffffff);
  return Candidate{static_cast<unsigned long long>(mh) << 32 | ml, row};
}
__device__ __forceinline__ void modulus_of(unsigned long long key, double& v) {
  v = __longlong_as_double(static_cast<long long>(key - 1));
}
__device__ __forceinline__ void modulus_of(unsigned long long key, float& v) {
  v = __uint_as_float(static_cast<unsigned>(key - 1));
}

// Double-float arithmetic (a value is an unevaluated sum hi + lo of two
// floats): Knuth's two-sum, about 48 significant bits on the FP32 pipe.
struct DF {
  float h, l;
};
__device__ __forceinline__ DF df_add(DF a, DF b) {
  const float s = a.h + b.h;
  const float v = s - a.h;
  float e = (a.h - (s - v)) + (b.h - v);
  e += a.l + b.l;
  const float r = s + e;
  return {r, e - (r - s)};
}

// ---- triangular sweeps -----------------------------------------------------
// Block k of the solution, x_k = Dinv_k (b_k - sum_i T_ki x_i) over the
// 64-row blocks i before k in sweep order.  With FP64 factors finished blocks
// are announced through one progress counter (release max by the producer,
// acquire loads by the consumers), the number of sweep positions whose x is in
// y; with FP32 factors x is its own signal.  Every wait is bounded by wait_ns:
// on timeout the CTA sets *err and leaves.
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until *progress >= target; returns the value seen, or 0 on timeout.
__device__ __forceinline__ unsigned wait_progress(const unsigned* progress, unsigned target,
                                                  unsigned long long wait_ns) {
  unsigned v = ld_acquire_u32(progress);
  if (v >= target) return v;
  const unsigned long long t0 = globaltimer_ns();
  for (unsigned it = 0;; it++) {
    __nanosleep(32);
    v = ld_acquire_u32(progress);
    if (v >= target) return v;
    if ((it & 15) == 15 && globaltimer_ns() - t0 > wait_ns) return 0;
  }
}

// ---- sweeps over FP32 factors ----
// Groups of TG consecutive 64-row blocks (from row 0 on), whose triangle is
// inverted as a whole after the factorisation: with G its inverse,
// x_g = G (b_g - sum of the products with earlier groups).
constexpr int TG = 2;
constexpr int TG_ROWS = TG * TB;
constexpr int TG_LD = TB + 1;  // row stride of the staged blocks: conflict-free reads down a column

// Off-diagonal 64 x 64 block of the inverse of every group's triangle, as
// (hi, lo) float pairs, row-major: X = -D1 T10 D0 of L (blockIdx.y 0), of U the
// same with the order of the blocks reversed, from the diagonal blocks'
// inverses D.  Two products of 64^3, four rows and columns a thread, in
// double-float like the D.  Bound: FP32 instructions, about 12 a term.
constexpr int GI_LD = TB + 4;  // 16-byte aligned rows
constexpr int GI_PLANE = TB * GI_LD;
constexpr size_t GI_SMEM = 7 * static_cast<size_t>(GI_PLANE) * sizeof(float);
// acc (sum, lost) += L R, L of hi and (LOW) lo planes, R of both
template <bool LOW>
__device__ __forceinline__ void gi_product(float2 (&acc)[4][4], const float* __restrict__ L,
                                           const float* __restrict__ R, int ty, int tx) {
#pragma unroll 4
  for (int k = 0; k < TB; k++) {
    const float4 h4 = *reinterpret_cast<const float4*>(R + k * GI_LD + 4 * tx);
    const float4 l4 = *reinterpret_cast<const float4*>(R + GI_PLANE + k * GI_LD + 4 * tx);
    const float rh[4] = {h4.x, h4.y, h4.z, h4.w}, rl[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float lh = L[(4 * ty + i) * GI_LD + k];
      const float ll = LOW ? L[GI_PLANE + (4 * ty + i) * GI_LD + k] : 0.0f;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float p = lh * rh[j];
        float low = fmaf(lh, rl[j], fmaf(lh, rh[j], -p));
        if (LOW) low = fmaf(ll, rh[j], low);
        const float s = acc[i][j].x, n = s + p, z = n - s;
        acc[i][j].y += ((s - (n - z)) + (p - z)) + low;
        acc[i][j].x = n;
      }
    }
  }
}
__global__ void __launch_bounds__(256) invert_groups(const float* __restrict__ A, long long ld, int N,
                                                     const float2* __restrict__ Linv2,
                                                     const float2* __restrict__ Uinv2, float2* __restrict__ Lx,
                                                     float2* __restrict__ Ux) {
  extern __shared__ __align__(16) float gi[];  // planes of 64 x GI_LD
  float* D[TG] = {gi, gi + 2 * GI_PLANE};       // hi, lo; in the order of elimination
  float* S = gi + 4 * GI_PLANE;                 // T D0: hi, lo
  float* T = gi + 6 * GI_PLANE;
  const int g = blockIdx.x, upper = blockIdx.y, tid = threadIdx.x;
  const int nblk = (N + TB - 1) / TB;
  const int ty = tid >> 4, tx = tid & 15;
  const float2* Dinv2 = upper ? Uinv2 : Linv2;
  float2* out = (upper ? Ux : Lx) + static_cast<size_t>(g) * TB * TB;
  auto natural = [&](int o) { return TG * g + (upper ? TG - 1 - o : o); };  // block of elimination step o
#pragma unroll
  for (int o = 0; o < TG; o++) {
    const int b = natural(o);
#pragma unroll 8
    for (int e = tid; e < TB * TB; e += 256) {
      const float2 d = b < nblk ? Dinv2[static_cast<size_t>(b) * TB * TB + e] : make_float2(0.f, 0.f);
      float* at = D[o] + (e / TB) * GI_LD + e % TB;
      at[0] = d.x;
      at[GI_PLANE] = d.y;
    }
  }
  const int r0 = natural(1) * TB, k0 = natural(0) * TB;
#pragma unroll 8
  for (int e = tid; e < TB * TB; e += 256) {
    const int i = e % TB, k = e / TB;
    T[i * GI_LD + k] = (r0 + i < N && k0 + k < N) ? A[static_cast<long long>(k0 + k) * ld + r0 + i] : 0.0f;
  }
  __syncthreads();
  float2 s[4][4] = {};
  gi_product<false>(s, T, D[0], ty, tx);
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float n = s[i][j].x + s[i][j].y;
      float* at = S + (4 * ty + i) * GI_LD + 4 * tx + j;
      at[0] = n;
      at[GI_PLANE] = s[i][j].y - (n - s[i][j].x);
    }
  __syncthreads();
  float2 v[4][4] = {};
  gi_product<true>(v, D[1], S, ty, tx);
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float n = v[i][j].x + v[i][j].y;
      out[(4 * ty + i) * TB + 4 * tx + j] = make_float2(-n, -(v[i][j].y - (n - v[i][j].x)));
    }
}

// A whole sweep in one cooperative launch; CTA c owns the groups c, c + grid,
// ... in sweep order.  Bound: the chain from group to group, whose links are the
// way of the last x through L2, its products and G's product; the tiles over
// earlier groups are loaded a group ahead.  The FP32 copy of x is its own
// signal: yf enters as all ones (a NaN that no x is stored as) and a thread
// waits for its entries to change, which saves the release, the acquire and one
// more way to L2; only the CTA whose turn is next polls without a pause.  Sums
// are double-float (G and the right-hand side as float pairs, about 48 bits) of
// FP32 products with x in sums of 8 terms: FP64 adds and conversions would run
// at the FP64 rate.  Inside the group the rows run in sweep order (reversed when
// descending): G is lower triangular in both sweeps.  b enters times bscale, y
// leaves times yscale (null: 1).  Every CTA is resident and a group waits for
// earlier ones only.
// N = 12,331: 0.177 ms a sweep (97 groups, about 3,700 cycles a link: 2,000 in
// the order of the arithmetic, 1,250 of them G's product, and the way through
// L2); 192-row groups chained block by block with a released counter 0.351 ms.
// Tried: G's product formed ahead for all but the last x, whose share then went
// through G in FP32: faster still, but matrices with ill-conditioned diagonal
// blocks took more refinement.  4-byte loads of the tiles: 6,000 cycles a link.
constexpr int TG_PART = 161;
// place of a row's partial sums: without bank conflicts for 16 lanes of rows
// 4 s + a each, for 16 lanes of one row, and for 8 consecutive rows read in pairs
__device__ __forceinline__ int tg_place(int row) { return (row >> 6) * 80 + (row & 3) * 20 + ((row & 63) >> 2); }
constexpr unsigned TG_EMPTY = 0xffffffffu;
__device__ __forceinline__ uint4 ld_relaxed_v4(const float* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
struct TgShared {
  float2 D[TG][TB * TG_LD];   // diagonal blocks of G, (hi, lo)
  float2 X[TB * TG_LD];       // block (1, 0)
  float2 part[16][TG_PART];   // sums of 16 threads a row, then of 8 warps
  float2 b[TG_ROWS];          // right-hand side, natural row order
  float2 v[TG_ROWS];          // in sweep order
  int abort;
};
__global__ void __launch_bounds__(256, 1) trsv_group(const float* __restrict__ A, long long ld, int N,
                                                     const double* __restrict__ b,
                                                     const double* __restrict__ bscale, double* __restrict__ y,
                                                     const double* __restrict__ yscale, float* yf,
                                                     const float2* __restrict__ Dinv2,
                                                     const float2* __restrict__ Xinv, int ascending, int* err,
                                                     unsigned long long wait_ns, unsigned stall) {
  static_assert(TG == 2 && TG_ROWS == 128, "two threads a row");
  extern __shared__ __align__(16) unsigned char tg_raw[];
  TgShared& sh = *reinterpret_cast<TgShared*>(tg_raw);
  const int nblk = (N + TB - 1) / TB, ng = (nblk + TG - 1) / TG;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // This thread's 16 entries of a 64 x 64 tile: four columns from 4 slot on and
  // four rows; four 16-byte loads, 256 contiguous bytes a half-warp.
  const int slot = 2 * warp + (lane >> 4), c0 = 4 * slot;
  auto tile_row = [&](int a) { return 4 * (lane & 15) + a; };
  const int i0 = lane, i1 = TB - 1 - lane;  // G: two rows of each block, columns warp + 8 i
  const int rown = tid >> 1, half = tid & 1;
  auto group = [&](int pos) { return ascending ? pos : ng - 1 - pos; };
  auto order = [&](int i) { return ascending ? i : TG_ROWS - 1 - i; };  // natural row of a group <-> sweep order
  auto df = [](float2 f) { return DF{f.x, f.y}; };
  auto both = [](DF a) {  // the sum of a pair of threads
    return df_add(a, {__shfl_xor_sync(0xffffffffu, a.h, 1), __shfl_xor_sync(0xffffffffu, a.l, 1)});
  };
  if (tid == 0) sh.abort = 0;
  __syncthreads();
  for (int pos = blockIdx.x; pos < ng; pos += gridDim.x) {
    const int R0 = group(pos) * TG_ROWS;
    bool inside = true;  // no row of this thread past the matrix
#pragma unroll
    for (int a = 0; a < 4; a++) inside = inside && R0 + TB + tile_row(a) < N;
    float t[TG][TG][16];  // [block of columns][block of rows][4 row + column]
    auto load_tile = [&](int p) {
      const int p0 = group(p) * TG_ROWS;
#pragma unroll
      for (int cb = 0; cb < TG; cb++) {
        const int k0 = p0 + cb * TB + c0;
        // the working copy's columns are 128-byte aligned, k0 and the first row multiples of 4
        if (inside && k0 + 4 <= N) {
          const float* src = A + static_cast<long long>(k0) * ld + R0 + tile_row(0);
#pragma unroll
          for (int rb = 0; rb < TG; rb++) {
            const float* q = src + rb * TB;
#pragma unroll
            for (int u = 0; u < 4; u++) {  // the thread's columns
              const float4 v = __ldg(reinterpret_cast<const float4*>(q));
              t[cb][rb][u] = v.x;
              t[cb][rb][4 + u] = v.y;
              t[cb][rb][8 + u] = v.z;
              t[cb][rb][12 + u] = v.w;
              q += ld;
            }
          }
        } else {
#pragma unroll
          for (int rb = 0; rb < TG; rb++)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
              for (int j = 0; j < 4; j++) {
                const int row = R0 + rb * TB + tile_row(a), k = k0 + j;
                t[cb][rb][4 * a + j] = (row < N && k < N) ? A[static_cast<long long>(k) * ld + row] : 0.f;
              }
        }
      }
    };
    if (pos > 0) load_tile(0);
    for (int nb = 0; nb < TG; nb++) {  // natural block nb of the group
      const int blk = group(pos) * TG + nb, ob = ascending ? nb : TG - 1 - nb;
#pragma unroll 8
      for (int e = tid; e < TB * TB; e += 256) {
        const float2 d = blk < nblk ? Dinv2[static_cast<size_t>(blk) * TB * TB + e] : make_float2(0.f, 0.f);
        int r = e / TB, c = e % TB;
        if (!ascending) r = TB - 1 - r, c = TB - 1 - c;
        sh.D[ob][r * TG_LD + c] = d;
      }
    }
#pragma unroll 8
    for (int e = tid; e < TB * TB; e += 256) {
      int r = e / TB, c = e % TB;
      if (!ascending) r = TB - 1 - r, c = TB - 1 - c;
      sh.X[r * TG_LD + c] = Xinv[static_cast<size_t>(group(pos)) * TB * TB + e];
    }
    if (tid < TG_ROWS) {
      double bv = R0 + tid < N ? b[R0 + tid] : 0.0;
      if (bscale && R0 + tid < N) bv *= bscale[R0 + tid];
      const float h = static_cast<float>(bv);
      sh.b[tid] = make_float2(h, static_cast<float>(bv - static_cast<double>(h)));
    }
    DF acc[TG][4];
#pragma unroll
    for (int r = 0; r < TG; r++)
#pragma unroll
      for (int a = 0; a < 4; a++) acc[r][a] = {0.f, 0.f};
    __syncthreads();
    float2 g0[2][4], g1[2][8], gx[2][8];  // this thread's entries of G
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int c = warp + 8 * i;
#pragma unroll
      for (int ob = 0; ob < TG; ob++) {
        if (i < 4) g0[ob][i] = sh.D[ob][i0 * TG_LD + c];  // row i0 < 32 ends before column 32
        g1[ob][i] = sh.D[ob][i1 * TG_LD + c];
      }
      gx[0][i] = sh.X[i0 * TG_LD + c];
      gx[1][i] = sh.X[i1 * TG_LD + c];
    }
    // products with the x of position p, then the tile over the next one
    auto step = [&](int p) {
      float x[TG][4];
      unsigned long long t_first = 0;
      for (unsigned it = 0;; it++) {
        bool here = stall == 0;
#pragma unroll
        for (int cb = 0; cb < TG; cb++) {
          const int k0 = group(p) * TG_ROWS + cb * TB + c0;
          // yf is 128-byte aligned and as long as N rounded up to 32, k0 a multiple of 4
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (k0 < N) v = ld_relaxed_v4(yf + k0);
          if (k0 + 1 >= N) v.y = 0u;
          if (k0 + 2 >= N) v.z = 0u;
          if (k0 + 3 >= N) v.w = 0u;
          here = here && v.x != TG_EMPTY && v.y != TG_EMPTY && v.z != TG_EMPTY && v.w != TG_EMPTY;
          x[cb][0] = __uint_as_float(v.x);
          x[cb][1] = __uint_as_float(v.y);
          x[cb][2] = __uint_as_float(v.z);
          x[cb][3] = __uint_as_float(v.w);
        }
        if (__all_sync(0xffffffffu, here)) break;
        if (p + 1 < pos) __nanosleep(400);
        if ((it & 15) == 15) {
          const unsigned long long now = globaltimer_ns();
          if (t_first == 0) t_first = now;
          if (__any_sync(0xffffffffu, now - t_first > wait_ns)) return false;
        }
      }
#pragma unroll
      for (int r = 0; r < TG; r++)
#pragma unroll
        for (int a = 0; a < 4; a++) {
          float sum = 0.f;
#pragma unroll
          for (int cb = 0; cb < TG; cb++)
#pragma unroll
            for (int j = 0; j < 4; j++) sum = fmaf(t[cb][r][4 * a + j], x[cb][j], sum);
          acc[r][a] = df_add(acc[r][a], {sum, 0.f});
        }
      if (p + 1 < pos) load_tile(p + 1);
      return true;
    };
    bool ok = true;
    for (int p = 0; p < pos && ok; p++) ok = step(p);
    if (!ok) sh.abort = 1;
#pragma unroll
    for (int r = 0; r < TG; r++)
#pragma unroll
      for (int a = 0; a < 4; a++) sh.part[slot][tg_place(r * TB + tile_row(a))] = make_float2(acc[r][a].h, acc[r][a].l);
    __syncthreads();
    if (sh.abort) {
      if (tid == 0) atomicExch(err, 1);
      return;
    }
    {  // v = b - sums: two threads a row
      DF h[8];
#pragma unroll
      for (int k = 0; k < 8; k++) h[k] = df(sh.part[8 * half + k][tg_place(rown)]);
#pragma unroll
      for (int w = 4; w > 0; w >>= 1)
#pragma unroll
        for (int k = 0; k < w; k++) h[k] = df_add(h[k], h[k + w]);
      const DF sum = both(h[0]);
      const DF v = df_add(df(sh.b[rown]), {-sum.h, -sum.l});
      if (half == 0) sh.v[order(rown)] = make_float2(v.h, v.l);
    }
    __syncthreads();
    // x = G v: rows i0 and i1 of each block over the columns warp + 8 i
#pragma unroll
    for (int ob = 0; ob < TG; ob++) {
      float s[2] = {0.f, 0.f}, e[2] = {0.f, 0.f};  // sums, and what their roundings lost
      auto term = [&](int k, float2 d, float2 v) {
        const float p = d.x * v.x;
        const float low = fmaf(d.y, v.x, fmaf(d.x, v.y, fmaf(d.x, v.x, -p)));
        const float n = s[k] + p, z = n - s[k];
        e[k] += ((s[k] - (n - z)) + (p - z)) + low;
        s[k] = n;
      };
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int c = warp + 8 * i;
        const float2 v = sh.v[ob * TB + c];
        if (i < 4) term(0, g0[ob][i], v);
        term(1, g1[ob][i], v);
      }
      if (ob == 1) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int c = warp + 8 * i;
          const float2 v = sh.v[c];
          term(0, gx[0][i], v);
          term(1, gx[1][i], v);
        }
      }
      sh.part[warp][ob * TB + i0] = make_float2(s[0], e[0]);
      sh.part[warp][ob * TB + i1] = make_float2(s[1], e[1]);
    }
    __syncthreads();
    const DF x = both(df_add(df_add(df(sh.part[4 * half][rown]), df(sh.part[4 * half + 1][rown])),
                             df_add(df(sh.part[4 * half + 2][rown]), df(sh.part[4 * half + 3][rown]))));
    const int row = R0 + order(rown);
    if (half == 0 && row < N) {
      const unsigned bits = __float_as_uint(x.h);
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(yf + row), "r"(bits == TG_EMPTY ? 0x7fffffffu : bits)
                   : "memory");
      const double sum = static_cast<double>(x.h) + static_cast<double>(x.l);
      y[row] = yscale ? sum * yscale[row] : sum;
    }
    __syncthreads();  // the staged blocks and part are read no more
  }
}

// ---- sweeps over FP64 factors, and transposed ones over FP32 factors ----
// The latter in FP64 too: b enters times the column scales, which may span any
// range, and x rounded to FP32 costs the refinement two or three steps (3 against
// 5 or 6 on well-conditioned matrices; no convergence at all with column scales
// of 2^-140 to 2^140).  Bound: the FP64 pipe of one SM, 2,048 cycles a tile of 64
// x 64, so a group is one block, conversions are made on the bits, and x is its own
// signal (y enters as all ones, a NaN that no x is stored as): 6,200 cycles a link.
// N = 7,819: 0.39 ms a sweep; blocks by threes with the counter 1.1, by ones 0.49;
// a launch a block, as before sweeps were chained, 2.5.
// A whole sweep in one cooperative launch, R consecutive blocks per group and one
// group at a time per CTA: CTA c owns the groups c, c + grid, ..., group g the sweep
// positions g R .. g R + R - 1.  While earlier groups are worked on it
// accumulates, for all the group's blocks at once, the products with every
// finished x (phase A, one progress wait per finished block).  The group's
// own blocks then chain inside the CTA (phase B): x_p from the accumulated
// rows and Dinv, published, and its products with the group's later blocks
// from the internal L blocks, which were staged in shared memory before
// phase A.  Thread (warp w, lane) works on row h*32 + lane of each block
// (h = w >> 2) and columns 16 q .. 16 q + 15 (q = w & 3).  Only
// ceil(nblk / R) hand-offs between CTAs remain on the
// critical path.  A group waits for lower groups only, and every CTA is
// resident, so the lowest unfinished group can always go on.
//
// Bound: the chain of dependent blocks, not the factor's bytes.
// TRANS sweeps solve with the transposed factor: the tile of output block p
// and finished block pi is the stored block (pi, p), whose columns are the
// output rows, so a thread reads 16 consecutive entries of one column.
constexpr int CH_R = 3;   // FP64 factors
constexpr int CH_RF = 1;  // FP32 factors: no more rows than the FP64 pipe of an SM keeps up with
constexpr int CH_DST = TB + 1;  // row stride of the staged Dinv blocks (conflict-free row reads)
constexpr int CH_LST = TB + 1;  // column stride of the staged internal blocks (transposed staging without conflicts)
// dynamic shared memory: the internal L blocks, then Dinv of the own blocks
template <int R>
constexpr size_t CH_SMEM = (static_cast<size_t>(R * (R - 1) / 2) * TB * CH_LST + static_cast<size_t>(R) * TB * CH_DST) *
                           sizeof(double);
// A factor's entry in FP64; of an FP32 one on its bits, since the conversion costs
// as much as a multiply-add.  Subnormals count as zero: the working copy is scaled
// to entries of size 1, so they lie 2^-73 below the rounding of an FP64 sum.
__device__ __forceinline__ double ch_entry(double v) { return v; }
__device__ __forceinline__ double ch_entry(float v) {
  const unsigned u = __float_as_uint(v), m = u & 0x7fffffffu;
  const bool normal = m >= 0x00800000u;
  const unsigned rebias = m >= 0x7f800000u ? 1792u << 20 : 896u << 20;  // Inf and NaN stay so
  const unsigned hi = (u & 0x80000000u) | (normal ? (m >> 3) + rebias : 0u);
  return __hiloint2double(static_cast<int>(hi), normal ? static_cast<int>(u << 29) : 0);
}

constexpr unsigned long long CH_EMPTY = ~0ull;
__device__ __forceinline__ ulonglong2 ld_relaxed_v2(const double* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
// b enters times bscale (null: 1).
template <class T, bool TRANS, int R>
__global__ void __launch_bounds__(256) trsv_chain(const T* __restrict__ A, long long ld, int N,
                                                  const double* __restrict__ b, const double* __restrict__ bscale,
                                                  double* y, const double* __restrict__ Dinv, int lower, unsigned* progress,
                                                  int* err, unsigned long long wait_ns, unsigned stall) {
  extern __shared__ __align__(16) unsigned char ch_raw[];
  double* Lin = reinterpret_cast<double*>(ch_raw);  // internal blocks (r2, r1), r1 < r2: column-major, stride CH_LST
  // Dinv of the own blocks, row-major 64 x 64 each with row stride CH_DST
  double* Dds = Lin + static_cast<size_t>(R * (R - 1) / 2) * TB * CH_LST;
  __shared__ double bsm[R][TB];
  __shared__ double part[4][TB];
  __shared__ double vd[TB];
  __shared__ double xs[TB];
  __shared__ int s_abort;
  const int nblk = (N + TB - 1) / TB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = warp & 3, h = warp >> 2;
  const int rr = h * 32 + lane;
  const int c0 = q * 16;
  auto blk = [&](int pos) { return lower ? pos : nblk - 1 - pos; };
  auto tri = [](int r2, int r1) { return r2 * (r2 - 1) / 2 + r1; };  // index of block (r2, r1), r1 < r2
  if (tid == 0) s_abort = 0;
  unsigned avail = 0;
  // 16-byte vector loads of x only from an aligned y (callers pass offset
  // vectors, e.g. a work vector at an odd offset N)
  const bool y_aligned = (reinterpret_cast<unsigned long long>(y) & 15ull) == 0;
  for (int p0 = blockIdx.x * R; p0 < nblk; p0 += gridDim.x * R) {
  const int np = (nblk - p0 < R) ? nblk - p0 : R;
  // Stage what the own blocks need besides the x of earlier blocks: the
  // internal L blocks (rows of position p0 + r2, columns of p0 + r1), the
  // Dinv blocks and the right-hand side, 16 independent loads in flight
  // per thread.
  for (int r2 = 1; r2 < np; r2++)
    for (int r1 = 0; r1 < r2; r1++) {
      const int kr = blk(p0 + r2), kc = blk(p0 + r1);
      double* dst = Lin + static_cast<size_t>(tri(r2, r1)) * TB * CH_LST;
      for (int e0 = 0; e0 < TB * TB; e0 += 16 * 256) {
        double v[16];
#pragma unroll
        for (int u = 0; u < 16; u++) {
          const int e = e0 + u * 256 + tid;
          const int row = (TRANS ? kc : kr) * TB + e % TB, col = (TRANS ? kr : kc) * TB + e / TB;
          v[u] = (row < N && col < N) ? static_cast<double>(A[static_cast<long long>(col) * ld + row]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 16; u++) {  // entry (i, j) of the block at dst[j * CH_LST + i]
          const int e = e0 + u * 256 + tid;
          dst[TRANS ? (e % TB) * CH_LST + e / TB : (e / TB) * CH_LST + e % TB] = v[u];
        }
      }
    }
  for (int r = 0; r < np; r++) {
    const size_t src = static_cast<size_t>(blk(p0 + r)) * TB * TB;
    for (int e0 = 0; e0 < TB * TB; e0 += 16 * 256) {
      // entry e = row * TB + col of the block goes to row * CH_DST + col
      // (TRANS: the transposed inverse, to col * CH_DST + row)
      double v[16];
#pragma unroll
      for (int u = 0; u < 16; u++) v[u] = Dinv[src + e0 + u * 256 + tid];
#pragma unroll
      for (int u = 0; u < 16; u++) {
        const int e = e0 + u * 256 + tid;
        Dds[static_cast<size_t>(r) * TB * CH_DST + (TRANS ? (e % TB) * CH_DST + e / TB : (e / TB) * CH_DST + e % TB)] =
            v[u];
      }
    }
    if (tid < TB) {
      const int row = blk(p0 + r) * TB + tid;
      double v = (row < N) ? b[row] : 0.0;
      if (bscale && row < N) v *= bscale[row];
      bsm[r][tid] = v;
    }
  }
  __syncthreads();
  double acc[R];
#pragma unroll
  for (int r = 0; r < R; r++) acc[r] = 0.0;
  // phase A: the finished blocks of earlier CTAs
  bool ok = true;
  // FP32 tiles are loaded a block ahead (FP64 ones would not fit twice in registers)
  constexpr bool kAhead = std::is_same<T, float>::value;
  T a[R][16], next[kAhead ? R : 1][16];
  // rows of this thread in its CTA's blocks (N when past the matrix)
  int rowof[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int row = blk(p0 + r) * TB + rr;
    rowof[r] = (r < np && row < N) ? row : N;
  }
  auto load_tile = [&](int pi, T(&to)[R][16]) {
    const int cb = blk(pi) * TB + c0;
    if constexpr (TRANS) {
      // entries cb .. cb + 15 of column rowof[r]
#pragma unroll
      for (int r = 0; r < R; r++) {
        const T* src = A + static_cast<long long>(rowof[r] < N ? rowof[r] : 0) * ld + cb;
        if (std::is_same<T, float>::value && rowof[r] < N && cb + 16 <= N) {
          // the working copy's columns are 128-byte aligned, cb a multiple of 16
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(src + j);
            to[r][j] = static_cast<T>(v.x);
            to[r][j + 1] = static_cast<T>(v.y);
            to[r][j + 2] = static_cast<T>(v.z);
            to[r][j + 3] = static_cast<T>(v.w);
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 16; j++) to[r][j] = (rowof[r] < N && cb + j < N) ? src[j] : T(0);
      }
      return;
    }
    const T* colp = A + static_cast<long long>(cb) * ld;
    if (cb + 16 <= N) {  // whole column quarter inside the matrix: no column predicates
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (rowof[r] < N) {
          const T* src = colp + rowof[r];
#pragma unroll
          for (int j = 0; j < 16; j++) {
            to[r][j] = *src;
            src += ld;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++) to[r][j] = T(0);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < 16; j++)
          to[r][j] = (rowof[r] < N && cb + j < N) ? colp[static_cast<long long>(j) * ld + rowof[r]] : T(0);
    }
  };
  if constexpr (kAhead)
    if (p0 > 0) load_tile(0, next);
  for (int pi = 0; pi < p0; pi++) {
    const int cb = blk(pi) * TB + c0;
    if constexpr (kAhead) {
#pragma unroll
      for (int r = 0; r < R; r++)
#pragma unroll
        for (int j = 0; j < 16; j++) a[r][j] = next[r][j];
      if (pi + 1 < p0) load_tile(pi + 1, next);
    } else {
      load_tile(pi, a);
    }
    double xq[16];
    if constexpr (kAhead) {
      // x is its own signal: y enters as all ones, and is 16-byte aligned and as
      // long as N rounded up to 32
      unsigned long long t_first = 0;
      for (unsigned it = 0; ok; it++) {
        bool here = stall == 0;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          ulonglong2 v = make_ulonglong2(0ull, 0ull);
          if (cb + j < N) v = ld_relaxed_v2(y + cb + j);
          if (cb + j + 1 >= N) v.y = 0ull;
          here = here && v.x != CH_EMPTY && v.y != CH_EMPTY;
          xq[j] = __longlong_as_double(static_cast<long long>(v.x));
          xq[j + 1] = __longlong_as_double(static_cast<long long>(v.y));
        }
        if (__all_sync(0xffffffffu, here)) break;
        if (pi + 1 < p0) __nanosleep(400);
        if ((it & 15) == 15) {
          const unsigned long long now = globaltimer_ns();
          if (t_first == 0) t_first = now;
          if (__any_sync(0xffffffffu, now - t_first > wait_ns)) ok = false;
        }
      }
      if (!ok) break;
    } else {
      if (static_cast<unsigned>(pi) >= avail) {
        const unsigned v = wait_progress(progress, static_cast<unsigned>(pi) + 1 + stall, wait_ns);
        if (v == 0) {
          ok = false;
          break;
        }
        avail = v - stall;  // positions known finished
      }
      if (y_aligned && cb + 16 <= N) {  // y + cb is then 16-byte aligned (cb is a multiple of 16)
        const double2* y2 = reinterpret_cast<const double2*>(y + cb);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const double2 v = __ldcg(y2 + j);
          xq[2 * j] = v.x;
          xq[2 * j + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; j++) xq[j] = (cb + j < N) ? __ldcg(y + cb + j) : 0.0;
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      double sum = 0.0;
#pragma unroll
      for (int j = 0; j < 16; j++) sum = fma(ch_entry(a[r][j]), xq[j], sum);
      acc[r] += sum;
    }
  }
  if (!ok) s_abort = 1;
  // phase B: this CTA's own blocks, chained in shared memory
#pragma unroll
  for (int r = 0; r < R; r++) {
    if (r >= np) break;
    const int k = blk(p0 + r);
    const int r0 = k * TB;
    const int n = (N - r0 < TB) ? N - r0 : TB;
    part[q][rr] = acc[r];
    __syncthreads();
    if (s_abort) {
      if (tid == 0) atomicExch(err, 1);
      return;
    }
    if (tid < TB) {
      const double sacc = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
      vd[tid] = (tid < n) ? bsm[r][tid] - sacc : 0.0;
    }
    __syncthreads();
    // x = Dinv v: thread (h, q, lane) forms row rr over columns c0 .. c0 + 15
    // (two accumulators), the four column quarters are added in shared
    // memory in a fixed order
    const size_t drow = static_cast<size_t>(r) * TB * CH_DST + static_cast<size_t>(rr) * CH_DST + c0;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      s0 = fma(Dds[drow + j], vd[c0 + j], s0);
      s1 = fma(Dds[drow + j + 1], vd[c0 + j + 1], s1);
    }
    part[q][rr] = s0 + s1;
    __syncthreads();
    if (tid < TB) {
      double x = (part[0][tid] + part[1][tid]) + (part[2][tid] + part[3][tid]);
      if (tid >= n) x = 0.0;
      xs[tid] = x;
      if constexpr (kAhead) {
        unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(x));
        if (bits == CH_EMPTY) bits >>= 1;  // still a NaN
        if (tid < n)
          asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(y + r0 + tid), "l"(bits) : "memory");
      } else {
        if (tid < n) y[r0 + tid] = x;
      }
    }
    if (kAhead && R == 1) break;  // no later own block
    __syncthreads();
    // release after the block barrier: the barrier orders every thread's
    // store of x before thread 0's release (no separate fence)
    if (!kAhead && tid == 0)
      asm volatile("red.release.gpu.global.max.u32 [%0], %1;" ::"l"(progress), "r"(static_cast<unsigned>(p0 + r) + 1)
                   : "memory");
    // products of the later own blocks with x_p
#pragma unroll
    for (int r2 = r + 1; r2 < R; r2++) {
      if (r2 >= np) break;
      const double* L = Lin + static_cast<size_t>(tri(r2, r)) * TB * CH_LST;
      double sum = 0.0;
#pragma unroll
      for (int j = 0; j < 16; j++) sum = fma(L[(c0 + j) * CH_LST + rr], xs[c0 + j], sum);
      acc[r2] += sum;
    }
  }
  __syncthreads();  // the staged blocks are read no more: the next group's may overwrite them
  }
}

// The row exchanges of one panel (pivots piv[0 .. jb), rows j0 .. ) as a
// list of moves row dst[t] <- row src[t] over the rows they touch (at most
// 2 jb): rows j0 .. j0+jb-1 first, then the pivot rows below the panel in
// order of first appearance.  One warp: lane 0 replays the exchanges with
// the rows below the panel found through a small hash table.  piv, rows
// (2 jb), content (2 jb), hkey and hidx (256 each) and cnt in shared memory.
// map[0] = count, map[1 .. 1+2jb) = dst, map[1+2jb .. 1+4jb) = src.
constexpr int SWAP_HASH = 256;
__device__ void swap_map_warp(const int* piv, int j0, int jb, int* __restrict__ map, int* rows, int* content,
                              int* hkey, int* hidx, int* cnt_s) {
  const int lane = threadIdx.x & 31;
  for (int t = lane; t < jb; t += 32) {
    rows[t] = j0 + t;
    content[t] = j0 + t;
  }
  for (int t = lane; t < SWAP_HASH; t += 32) hkey[t] = -1;
  __syncwarp();
  if (lane == 0) {
    int cnt = jb;
    for (int jj = 0; jj < jb; jj++) {
      const int p = piv[jj];
      int idx;
      if (p < j0 + jb) {
        idx = p - j0;
      } else {
        unsigned h = (static_cast<unsigned>(p) * 2654435761u) >> 24;  // 8 bits
        while (hkey[h] != -1 && hkey[h] != p) h = (h + 1) & (SWAP_HASH - 1);
        if (hkey[h] == p) {
          idx = hidx[h];
        } else {
          idx = cnt++;
          hkey[h] = p;
          hidx[h] = idx;
          rows[idx] = p;
          content[idx] = p;
        }
      }
      const int t = content[jj];
      content[jj] = content[idx];
      content[idx] = t;
    }
    *cnt_s = cnt;
  }
  __syncwarp();
  const int n = *cnt_s;
  for (int t = lane; t < n; t += 32) {
    map[1 + t] = rows[t];
    map[1 + 2 * jb + t] = content[t];
  }
  if (lane == 0) map[0] = n;
}

__global__ void build_swap_map(const int* __restrict__ ipiv, int j0, int jb, int* __restrict__ map) {
  __shared__ int rows[256], content[256], piv[128], hkey[SWAP_HASH], hidx[SWAP_HASH];
  __shared__ int cnt;
  for (int t = threadIdx.x; t < jb; t += 32) piv[t] = ipiv[j0 + t];
  __syncwarp();
  swap_map_warp(piv, j0, jb, map, rows, content, hkey, hidx, &cnt);
}

template <class T>
__global__ void __launch_bounds__(GP_THREADS) panel_grid_kernel(T* __restrict__ A, long long ld, int N, int j0, int jb,
                                                                int per, int* __restrict__ ipiv,
                                                                int* __restrict__ info, int* __restrict__ map,
                                                                PanelSlots<T> ps) {
  extern __shared__ __align__(16) unsigned char gp_raw[];
  T* tile = reinterpret_cast<T*>(gp_raw);
  __shared__ T prow[128];  // the pivot row
  __shared__ T s_inv;
  __shared__ Candidate s_best[GP_POLL_WARPS];
  __shared__ int s_fail, s_piv[128];
  const int nblk = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = j0 + b * per;
  const int r1 = (r0 + per < N) ? r0 + per : N;
  const int nr = r1 - r0;
  if (tid == 0) s_fail = 0;
  for (int k = warp; k < jb; k += GP_THREADS / 32)
    for (int r = lane; r < nr; r += 32) tile[k * per + r] = A[static_cast<long long>(j0 + k) * ld + r0 + r];
  __syncthreads();
  for (int jj = 0; jj < jb; jj++) {
    const int j = j0 + jj, slot = jj & 1;
    if (warp == 0) {
      // 1. local candidate
      Candidate c{0, N};
      for (int i = (r0 > j ? r0 : j) + lane; i < r1; i += 32)
        c = better_of(c, Candidate{modulus_key(tile[jj * per + i - r0]), i});
      c = warp_best(c);
      if (c.key == 0) c.row = N;
      // 2. publish its row (and row j when this CTA owns it), then the record
      T* mine = ps.cand_rows + (static_cast<size_t>(slot) * nblk + b) * jb;
      if (c.row < N)
        for (int k = lane; k < jb; k += 32) mine[k] = tile[k * per + c.row - r0];
      if (j >= r0 && j < r1)
        for (int k = lane; k < jb; k += 32) ps.jrow[slot * jb + k] = tile[k * per + j - r0];
      __syncwarp();
      if (lane == 0) {
        ps.rec[slot * nblk + b] = PanelRecord{c.key, static_cast<unsigned long long>(c.row)};
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(ps.count), "r"(1u) : "memory");
      }
    }
    // 3. all arrivals seen: every CTA's record, one a lane
    if (warp == 0 && lane == 0) {
      const unsigned want = static_cast<unsigned>(nblk) * (jj + 1) + ps.stall;
      unsigned long long t0 = 0;
      for (unsigned it = 0;; it++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ps.count) : "memory");
        if (v >= want) break;
        if (it == 0) t0 = globaltimer_ns();
        else if ((it & 31) == 31 && globaltimer_ns() - t0 > ps.wait_ns) {
          s_fail = 1;
          break;
        }
      }
    }
    __syncthreads();
    if (s_fail) {
      if (tid == 0) {
        atomicExch(ps.err, 1);
        if (b == 0) map[0] = 0;  // no row moves
      }
      return;
    }
    if (warp < GP_POLL_WARPS) {
      Candidate c{0, N};
      const int t = warp * 32 + lane;
      if (t < nblk) {
        const ulonglong2 r = __ldcg(reinterpret_cast<const ulonglong2*>(ps.rec + slot * nblk + t));
        c = Candidate{r.x, static_cast<int>(r.y)};
      }
      c = warp_best(c);
      if (lane == 0) s_best[warp] = c;
    }
    __syncthreads();
    Candidate best = s_best[0];
#pragma unroll
    for (int w = 1; w < GP_POLL_WARPS; w++) best = better_of(best, s_best[w]);
    // nothing usable below the diagonal: no swap
    const int gi = best.key != 0 ? best.row : j;
    // 4. the pivot row into prow (the part left of the diagonal only where
    // the row goes) and the row exchange: nobody reads rows j and gi of the
    // tile between these barriers
    const int from = best.key != 0 ? (gi - j0) / per : 0;
    const T* src = best.key != 0 ? ps.cand_rows + (static_cast<size_t>(slot) * nblk + from) * jb : ps.jrow + slot * jb;
    const bool own_j = j >= r0 && j < r1;
    if (tid < jb) {
      if (tid >= jj || own_j) {
        const T pk = __ldcg(src + tid);
        prow[tid] = pk;
        if (own_j) tile[tid * per + j - r0] = pk;
      }
    } else if (tid >= 128 && tid < 128 + jb) {
      if (gi != j && gi >= r0 && gi < r1) tile[(tid - 128) * per + gi - r0] = __ldcg(ps.jrow + slot * jb + tid - 128);
    } else if (tid == 256) {  // the reciprocal, from the key, beside the row's load
      T v = T(1);  // (not used below a zero pivot)
      if (best.key > KEY_OF_ZERO) modulus_of(best.key, v);
      else if (best.key == 0) v = static_cast<T>(nan(""));  // every candidate is
      s_inv = T(1) / v;  // zero for an infinite pivot: so are its multipliers
      s_piv[jj] = gi;
      if (b == 0) {
        ipiv[j] = gi;
        if (best.key <= KEY_OF_ZERO && *info == 0) *info = j + 1;  // zero (or NaN) pivot
      }
    }
    __syncthreads();
    // 5. scale the column below the pivot, rank-1 update of the rest
    const T inv = prow[jj] < T(0) ? -s_inv : s_inv;
    const int rs = (r0 > j + 1) ? r0 : j + 1;
    if (prow[jj] != T(0) && rs < r1) {
      for (int i = rs + tid; i < r1; i += GP_THREADS) tile[jj * per + i - r0] *= inv;
      __syncthreads();
      // warps over (64-row group, column phase): rows along the lanes
      // (conflict-free shared memory), two per lane
      const int nrr = r1 - rs, ngr = (nrr + 63) / 64, nph = (GP_THREADS / 32) / (ngr < GP_THREADS / 32 ? ngr : GP_THREADS / 32);
      const int nwu = ngr < GP_THREADS / 32 ? ngr : GP_THREADS / 32;  // row groups worked on at a time
      const int wg = warp % nwu, ph = warp / nwu;
      if (ph < nph)
        for (int gq = wg; gq < ngr; gq += nwu) {
          const int i0 = gq * 64 + lane, i1 = i0 + 32;
          const bool u0 = i0 < nrr, u1 = i1 < nrr;
          T* c0 = tile + (rs - r0) + i0;
          T* c1 = c0 + 32;
          const T l0 = u0 ? c0[jj * per] : T(0), l1 = u1 ? c1[jj * per] : T(0);
          for (int k = jj + 1 + ph; k < jb; k += nph) {
            const T p = prow[k];
            if (u0) c0[k * per] = fma(-l0, p, c0[k * per]);
            if (u1) c1[k * per] = fma(-l1, p, c1[k * per]);
          }
        }
    }
    __syncthreads();
  }
  for (int k = warp; k < jb; k += GP_THREADS / 32)
    for (int r = lane; r < nr; r += 32) A[static_cast<long long>(j0 + k) * ld + r0 + r] = tile[k * per + r];
  // the panel's row moves for the swaps outside it (the tile is free now)
  if (b == 0) {
    __syncthreads();
    if (warp == 0) {
      int* rows = reinterpret_cast<int*>(gp_raw);
      swap_map_warp(s_piv, j0, jb, map, rows, rows + 256, rows + 512, rows + 512 + SWAP_HASH,
                    rows + 512 + 2 * SWAP_HASH);
    }
  }
}

// ---- panel on one 16-CTA cluster (FP32 factors) --------------------------
// The same algorithm as panel_grid_kernel with the exchange in distributed
// shared memory: CTA r of the cluster keeps rows [j0 + r*per, ...) of the
// panel in its shared memory, row by row (stride cp_row_stride(jb) floats,
// so that a row's 16-column inner block is four aligned 128-bit words and
// eight consecutive rows hit distinct banks).  While a 16-column inner block is
// worked on, its columns live in the registers of the rows' threads.  Per
// column, one block barrier and one exchange:
//  - every thread already holds its best candidate for the column (found
//    while updating it in the previous column step); a warp reduction, the
//    winner's block columns through shared memory and one block barrier give
//    the CTA's candidate;
//  - warp 0 pushes (value, the row's inner block) and warp 2 the row number
//    into every CTA's receive slot, and warp 1 of the owner of row j pushes
//    row j's inner block; the CTA keeps its candidate's full row (copied by
//    warp 2 first) and row j locally;
//  - when its slot is complete every warp picks the winner from its own
//    receive slot (same order everywhere); each thread then swaps, scales
//    and updates the inner block of its rows and tracks its candidate for
//    column j + 1, all in one pass; the multipliers go to the tile;
//  - the other columns of the two swapped rows are fetched from the owners'
//    shared memory off the critical path.
// Receive slots, candidate rows and row j are double-buffered by column
// parity: a CTA can only overwrite a slot after every CTA has pushed the next
// column, i.e. has finished reading it.
// Bound: latency, about 3,200 cycles a column (376 rows a CTA, 96 columns): the
// CTA's candidate 550, pushing 600, waiting 500, the winner 250, the column step
// 430, the block ends 720.  With the block in shared memory a step took 850 (its
// bandwidth), arg-max by shuffles instead of redux 900 more, the U12 columns of a
// block end through shared memory 300, and the candidate's row copy before the
// pushes of the same warp 100: 224 -> 151 us per panel at N = 6,001, 235 -> 151 us
// on average at N = 12,331.
constexpr int CP_CL = 16;
constexpr int CP_THREADS = 512;  // most; see cp_threads
constexpr int CP_WARPS = CP_THREADS / 32;
constexpr size_t CP_MAX_SMEM = 212 * 1024;
// Threads for `per` rows a CTA: whole rounds of the rows, at most 448 a round
// (771 rows: two rounds of 416 instead of three of 384), no fewer than 256.
constexpr int cp_threads(int per) {
  const int rounds = (per + 447) / 448, t = ((per + rounds - 1) / rounds + 31) / 32 * 32;
  return t < 256 ? 256 : t;
}
constexpr int CP_IB = 16;  // inner block: columns updated per column step

// Row stride (floats) of the panel in shared memory: whole 16-column inner
// blocks plus 4, i.e. an odd number of 16-byte words.
__host__ __device__ constexpr int cp_row_stride(int jb) { return ((jb + 15) / 16) * 16 + 4; }

// |v| as an integer of the same order: 0 for NaN (never a pivot), else its bits
// + 1.  Arg-max are then two redux instructions (largest key, lowest row).
__device__ __forceinline__ unsigned cp_key(float v) {
  const unsigned k = __float_as_uint(v) & 0x7fffffffu;
  return k > 0x7f800000u ? 0u : k + 1u;
}
__device__ __forceinline__ void cp_warp_best(unsigned& key, int& row) {
  const unsigned m = __reduce_max_sync(0xffffffffu, key);
  row = __reduce_min_sync(0xffffffffu, key == m ? row : 0x7fffffff);
  key = m;
}

struct CpSlot {
  float4 seg[CP_CL][CP_IB / 4];  // candidate rows' inner blocks, by source CTA
  float4 jseg[CP_IB / 4];        // row j's inner block
  unsigned v[CP_CL];             // keys of the candidates, by source CTA
  int i[CP_CL];                  // candidate rows (N: none), by source CTA
};

// The per-column exchange of the cluster panel: each CTA's candidate (and the
// owner's row j) go to every CTA's receive slot by st.async, which completes
// on that CTA's mbarrier for the slot (its complete-tx has release semantics
// at cluster scope); a CTA waits on its own mbarrier (acquire at cluster
// scope), bounded by wait_ns.  False (and *err set) when the wait ran out.
__device__ __forceinline__ unsigned cp_smem(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ unsigned cp_mapa(unsigned a, unsigned rank) {
  unsigned d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  return d;
}
__device__ __forceinline__ void cp_push4(unsigned dst, float4 v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)),
               "r"(__float_as_uint(v.w)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cp_push1(unsigned dst, unsigned v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cp_arm(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cp_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool cp_wait(unsigned long long* bar, unsigned parity, unsigned long long wait_ns,
                                        int* err) {
  const unsigned a = cp_smem(bar);
  unsigned long long t0 = 0;
  for (int spin = 0;; spin++) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 "
        "%0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if (spin == 0) {
      t0 = globaltimer_ns();
    } else if ((spin & 15) == 0 && globaltimer_ns() - t0 > wait_ns) {
      atomicExch(err, 1);
      return false;
    }
  }
}

template <int RPT>
__global__ void __launch_bounds__(CP_THREADS, 1) panel_cluster16_kernel(float* __restrict__ A, long long ld, int N,
                                                                     int j0, int jb, int per,
                                                                     int* __restrict__ ipiv,
                                                                     int* __restrict__ info,
                                                                     int* __restrict__ swap_map,
                                                                     int* __restrict__ err,
                                                                     unsigned long long wait_ns, unsigned stall) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char cp_raw[];
  float* tile = reinterpret_cast<float*>(cp_raw);  // tile[r * S + k]
  __shared__ int pivs[128];  // the panel's pivots (CTA 0)
  __shared__ __align__(16) float cand_row[2][128];
  __shared__ __align__(16) float jrow[2][128];
  __shared__ __align__(16) CpSlot recv[2];
  __shared__ __align__(16) float ublk[CP_IB][128];  // rows of the current inner block (L11 | A12 -> U12)
  __shared__ unsigned wv[CP_WARPS];
  __shared__ int wi[CP_WARPS];
  __shared__ __align__(16) float4 wseg[CP_WARPS][CP_IB / 4], jbuf[CP_IB / 4];  // the warps' candidates, row j
  __shared__ __align__(8) unsigned long long xmb[2];  // the exchange's mbarriers, one per receive slot
  const int S = cp_row_stride(jb);
  const int rank = static_cast<int>(cluster.block_rank());
  const int ncl = static_cast<int>(cluster.num_blocks());  // 2, 4, 8 or 16 CTAs
  const int tid = threadIdx.x, bd = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int r0 = j0 + rank * per;
  const int r1 = (r0 + per < N) ? r0 + per : N;
  const int nr = r1 > r0 ? r1 - r0 : 0;
  for (int e = tid; e < jb * nr; e += bd) {
    int k = e / nr, r = e % nr;
    tile[r * S + k] = A[static_cast<long long>(j0 + k) * ld + r0 + r];
  }
  // bytes one column's exchange brings to each CTA: every CTA's candidate
  // (its 16-column segment, value and row) and the owner's segment of row j;
  // stall_waits asks for bytes that never come
  const unsigned xbytes = static_cast<unsigned>(ncl) * (4 * 16 + 8) + 4 * 16 + (stall ? 16u : 0u);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cp_smem(&xmb[0])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cp_smem(&xmb[1])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cp_arm(&xmb[0], xbytes);
    cp_arm(&xmb[1], xbytes);
  }
  bool dead = false;  // this thread's exchange wait ran out: no more waits
  cluster.sync();     // every CTA's mbarriers exist before the first push
  for (int b0 = 0; b0 < jb; b0 += CP_IB) {
    const int be = (b0 + CP_IB < jb) ? b0 + CP_IB : jb;
    const int nb = be - b0;
    // The inner block of this thread's rows stays in registers for the
    // block's columns, t[r][0] being the current column (each step shifts the
    // rest down); and the thread's candidate for the block's first column.
    float t[RPT][CP_IB];
    unsigned best = 0;
    int bi = N;
#pragma unroll
    for (int r = 0; r < RPT; r++) {
      const int li = tid + r * bd;
#pragma unroll
      for (int c = 0; c < CP_IB / 4; c++) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (li < nr) x = *reinterpret_cast<const float4*>(tile + static_cast<size_t>(li) * S + b0 + 4 * c);
        t[r][4 * c] = x.x;
        t[r][4 * c + 1] = x.y;
        t[r][4 * c + 2] = x.z;
        t[r][4 * c + 3] = x.w;
      }
      if (li < nr && r0 + li >= j0 + b0) {
        const unsigned key = cp_key(t[r][0]);
        if (key > best) {  // rows ascend: ties stay with the lower one
          best = key;
          bi = r0 + li;
        }
      }
    }
    for (int jj = b0; jj < be; jj++) {
      const int j = j0 + jj;
      const int slot = jj & 1;
      const int q0 = jj - b0;  // column jj within the inner block
      {
        const int own = bi;
        cp_warp_best(best, bi);
        const bool cand = best != 0 && own == bi;
#pragma unroll
        for (int r = 0; r < RPT; r++) {
          const int i = r0 + tid + r * bd;
          if (cand && i == bi) {
#pragma unroll
            for (int c = 0; c < CP_IB / 4; c++)
              wseg[warp][c] = make_float4(t[r][4 * c], t[r][4 * c + 1], t[r][4 * c + 2], t[r][4 * c + 3]);
          }
          if (i == j && tid + r * bd < nr) {
#pragma unroll
            for (int c = 0; c < CP_IB / 4; c++)
              jbuf[c] = make_float4(t[r][4 * c], t[r][4 * c + 1], t[r][4 * c + 2], t[r][4 * c + 3]);
          }
        }
      }
      if (lane == 0) {
        wv[warp] = best;
        wi[warp] = bi;
      }
      __syncthreads();  // also orders the previous column step's tile writes
      if (warp == 0 || warp == 2) {
        unsigned cv = (lane < (bd >> 5)) ? wv[lane] : 0u;
        int ci = (lane < (bd >> 5)) ? wi[lane] : N;
        const unsigned wkey = cv;
        const int wrow = ci;
        cp_warp_best(cv, ci);
        if (warp == 0) {
          const int from = __ffs(__ballot_sync(0xffffffffu, wkey == cv && wrow == ci)) - 1;
          const float4* src = wseg[from < CP_WARPS ? from : 0];  // any words when there is no candidate
          // (destination CTA, half of the inner block)
          for (int e = lane; e < 2 * ncl; e += 32) {
            const unsigned d = static_cast<unsigned>(e >> 1);
            const int c0 = (e & 1) * 2;
            const unsigned bar = cp_mapa(cp_smem(&xmb[slot]), d);
            cp_push4(cp_mapa(cp_smem(&recv[slot].seg[rank][c0]), d), src[c0], bar);
            cp_push4(cp_mapa(cp_smem(&recv[slot].seg[rank][c0 + 1]), d), src[c0 + 1], bar);
            if ((e & 1) == 0) cp_push1(cp_mapa(cp_smem(&recv[slot].v[rank]), d), cv, bar);
          }
        } else {
          // the candidate's other columns, then its row number: the (releasing)
          // push of the number comes after the whole row copy
          if (cv == 0) ci = N;
          if (ci < N)
            for (int k = lane; k < jb; k += 32) cand_row[slot][k] = tile[static_cast<size_t>(ci - r0) * S + k];
          __syncwarp();
          if (lane < ncl)
            cp_push1(cp_mapa(cp_smem(&recv[slot].i[rank]), lane), static_cast<unsigned>(ci),
                     cp_mapa(cp_smem(&xmb[slot]), lane));
        }
      } else if (warp == 1 && j >= r0 && j < r1) {
        for (int k = lane; k < jb; k += 32) jrow[slot][k] = tile[(j - r0) * S + k];
        __syncwarp();
        const float4* src = jbuf;
        for (int e = lane; e < 2 * ncl; e += 32) {
          const unsigned d = static_cast<unsigned>(e >> 1);
          const int c0 = (e & 1) * 2;
          const unsigned bar = cp_mapa(cp_smem(&xmb[slot]), d);
          cp_push4(cp_mapa(cp_smem(&recv[slot].jseg[c0]), d), src[c0], bar);
          cp_push4(cp_mapa(cp_smem(&recv[slot].jseg[c0 + 1]), d), src[c0 + 1], bar);
        }
      }
      // every CTA's push of this column; the slot's next phase is column jj + 2
      // (its pushes come only after this CTA's own push of column jj + 1)
      if (!dead) dead = !cp_wait(&xmb[slot], static_cast<unsigned>(jj >> 1) & 1u, wait_ns, err);
      if (tid == 0 && !dead) cp_arm(&xmb[slot], xbytes);
      // the winner, from this CTA's own receive slot: every warp reduces the
      // candidates across its lanes (same result everywhere)
      const unsigned mine = lane < ncl ? recv[slot].v[lane] : 0u;
      unsigned gv = mine;
      int gi = lane < ncl ? recv[slot].i[lane] : N;
      const int row = gi;
      cp_warp_best(gv, gi);
      // the CTA it came from (rows are distinct)
      int tag = __ffs(__ballot_sync(0xffffffffu, mine == gv && row == gi)) - 1;
      // nothing usable below the diagonal: no swap.  (A winner is always a
      // row at or below j; a thread whose exchange wait ran out may read a
      // stale slot, and the row-move list must still hold rows of the panel.)
      if (gi < j || gi >= N) {
        gi = j;
        tag = -1;
      }
      if (rank == 0 && tid == 0) {
        ipiv[j] = gi;
        pivs[jj] = gi;
        if (gv <= 1u && *info == 0) *info = j + 1;  // zero (or NaN) pivot
      }
      // the pivot row's inner block
      const float4* p4 = (tag >= 0) ? recv[slot].seg[tag] : recv[slot].jseg;
      float ps[CP_IB];
#pragma unroll
      for (int c = 0; c < CP_IB / 4; c++) {
        const float4 x = p4[c];
        ps[4 * c] = x.x;
        ps[4 * c + 1] = x.y;
        ps[4 * c + 2] = x.z;
        ps[4 * c + 3] = x.w;
      }
      const float piv = ps[0];
      const bool nonzero = piv != 0.0f;
      const float inv = nonzero ? 1.0f / piv : 0.0f;
      // the column step on this thread's rows: row gi takes row j's block, the
      // multiplier goes to its place in the tile, the rest is updated and
      // shifted down; and the thread's candidate for the next column
      best = 0;
      bi = N;
#pragma unroll
      for (int r = 0; r < RPT; r++) {
        const int li = tid + r * bd, i = r0 + li;
        if (li >= nr || i <= j) continue;
        if (i == gi) {
#pragma unroll
          for (int c = 0; c < CP_IB / 4; c++) {
            const float4 x = recv[slot].jseg[c];
            t[r][4 * c] = x.x;
            t[r][4 * c + 1] = x.y;
            t[r][4 * c + 2] = x.z;
            t[r][4 * c + 3] = x.w;
          }
        }
        const float l = nonzero ? t[r][0] * inv : t[r][0];
        tile[static_cast<size_t>(li) * S + jj] = l;
        if (nonzero) {
#pragma unroll
          for (int q = 1; q < CP_IB; q++) t[r][q - 1] = fmaf(-l, ps[q], t[r][q]);
        } else {
#pragma unroll
          for (int q = 1; q < CP_IB; q++) t[r][q - 1] = t[r][q];
        }
        t[r][CP_IB - 1] = 0.0f;
        if (q0 + 1 < nb) {
          const unsigned key = cp_key(t[r][0]);
          if (key > best) {
            best = key;
            bi = i;
          }
        }
      }
      // row j becomes the pivot row: its columns jj .. be - 1
      if (j >= r0 && j < r1 && tid < be - jj)
        tile[static_cast<size_t>(j - r0) * S + jj + tid] = reinterpret_cast<const float*>(p4)[tid];
      // the swapped rows' other columns, from the owners' shared memory
      if (gi != j) {
        if (gi >= r0 && gi < r1) {
          const float* src = cluster.map_shared_rank(&jrow[slot][0], (j - j0) / per);
          for (int k = tid; k < jb; k += bd)
            if (k < jj || k >= be) tile[(gi - r0) * S + k] = src[k];
        }
        if (j >= r0 && j < r1) {
          const float* src = cluster.map_shared_rank(&cand_row[slot][0], tag);
          for (int k = tid; k < jb; k += bd)
            if (k < jj || k >= be) tile[(j - r0) * S + k] = src[k];
        }
      }
    }
    if (be < jb) {
      // Rows j0+b0 .. j0+be-1 are final in columns b0..be-1 (L11 below the
      // diagonal); every CTA fetches them whole and forms
      // U12 = L11^{-1} A12 for columns be..jb-1.
      cluster.sync();
      // (the columns from b0 on, by 16-byte words, all loads before the stores;
      // nb == CP_IB here, and padding columns come along)
      {
        const int words = S / 4 - 1 - b0 / 4, total = CP_IB * words;
        float4 w[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int e = tid + u * bd;
          if (e < total) {
            const int t = e / words, k4 = e - t * words, row = b0 + t, owner = row / per;
            w[u] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(tile, owner) +
                                                    static_cast<size_t>(row - owner * per) * S + b0 + 4 * k4);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int e = tid + u * bd;
          if (e < total) *reinterpret_cast<float4*>(&ublk[e / words][b0 + 4 * (e % words)]) = w[u];
        }
      }
      __syncthreads();
      for (int k = be + tid; k < jb; k += bd) {  // one column of U12 per thread, in registers
        float u[CP_IB];
#pragma unroll
        for (int t = 0; t < CP_IB; t++) u[t] = ublk[t][k];
#pragma unroll
        for (int t = 1; t < CP_IB; t++) {
          float acc = u[t];
#pragma unroll
          for (int q = 0; q < t; q++) acc = fmaf(-ublk[t][b0 + q], u[q], acc);
          u[t] = acc;
          ublk[t][k] = acc;
        }
      }
      cluster.sync();  // remote reads of the block rows are done
      // owners store U12; rows below the block get the rank-16 update, one
      // row per thread with its 16 multipliers in registers and four
      // columns per step
      for (int e = tid; e < nb * (jb - be); e += bd) {
        const int t = e / (jb - be), k = be + e % (jb - be);
        const int row = j0 + b0 + t;
        if (row >= r0 && row < r1) tile[(row - r0) * S + k] = ublk[t][k];
      }
      const int rs = (r0 > j0 + be) ? r0 : j0 + be;
      for (int i = rs + tid; i < r1; i += bd) {
        const int li = i - r0;
        const float4* lrow = reinterpret_cast<const float4*>(tile + static_cast<size_t>(li) * S + b0);
        float l[CP_IB];
#pragma unroll
        for (int c = 0; c < CP_IB / 4; c++) {
          const float4 x = lrow[c];
          l[4 * c] = x.x;
          l[4 * c + 1] = x.y;
          l[4 * c + 2] = x.z;
          l[4 * c + 3] = x.w;
        }
        float4* arow = reinterpret_cast<float4*>(tile + static_cast<size_t>(li) * S);
        // (inside this branch the block is full: nb == CP_IB; columns past
        // jb up to the stride are padding, updated but never read)
        for (int k4 = be / 4; k4 < (jb + 3) / 4; k4++) {
          float4 acc = arow[k4];
#pragma unroll
          for (int q = 0; q < CP_IB; q++) {
            const float4 u = *reinterpret_cast<const float4*>(&ublk[q][4 * k4]);
            acc.x = fmaf(-l[q], u.x, acc.x);
            acc.y = fmaf(-l[q], u.y, acc.y);
            acc.z = fmaf(-l[q], u.z, acc.z);
            acc.w = fmaf(-l[q], u.w, acc.w);
          }
          arow[k4] = acc;
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  for (int e = tid; e < jb * nr; e += bd) {
    int k = e / nr, r = e % nr;
    A[static_cast<long long>(j0 + k) * ld + r0 + r] = tile[r * S + k];
  }
  cluster.sync();  // remote readers of this CTA's shared memory are done
  // the panel's row moves for the swaps outside it (ublk is free now)
  if (swap_map && rank == 0 && warp == 0) {
    int* rows = reinterpret_cast<int*>(&ublk[0][0]);
    swap_map_warp(pivs, j0, jb, swap_map, rows, rows + 256, rows + 512, rows + 512 + SWAP_HASH,
                  rows + 512 + 2 * SWAP_HASH);
  }
}

// Widest panel (96, 64 or 32 columns) whose rows fit in the shared memory of
// one 16-CTA cluster; 0 when none does.
// Widest panel (96, 64 or 32 columns, no narrower than min_w) whose rows fit
// the shared memory of one 16-CTA cluster; 0 when none does.
static int cluster_panel_width(int rows, int min_w = 32) {
  const int per = (rows + CP_CL - 1) / CP_CL;
  for (int w : {96, 64, 32})
    if (w >= min_w && static_cast<size_t>(per) * cp_row_stride(w) * sizeof(float) <= CP_MAX_SMEM) return w;
  return 0;
}

// True when the cooperative grid kernel on `nsm` SMs holds a panel of this
// height and width in shared memory (panel_grid's own test).
static bool grid_panel_fits(int rows, int jb, int nsm, size_t elem) {
  int nblk = (rows + GP_MIN_ROWS - 1) / GP_MIN_ROWS;
  if (nblk > nsm) nblk = nsm;
  if (nblk > 32 * GP_POLL_WARPS) nblk = 32 * GP_POLL_WARPS;
  const int per = (rows + nblk - 1) / nblk;
  return static_cast<size_t>(per) * jb * elem <= GP_MAX_SMEM;
}

// Launches the cluster panel on the smallest cluster (2, 4, 8 or 16 CTAs)
// whose shared memory holds the panel; false when none does or the GPU
// cannot host a 16-CTA cluster (the caller then uses the cooperative grid
// kernel).
static bool panel_cluster16(Context* ctx, float* A, long long ld, int N, int j0, int jb, int* ipiv, int* info,
                            int* swap_map, int* err, unsigned long long wait_ns, unsigned stall) {
  const int rows = N - j0;
  int ncl = 2;
  while (ncl < CP_CL &&
         static_cast<size_t>((rows + ncl - 1) / ncl) * cp_row_stride(jb) * sizeof(float) > CP_MAX_SMEM)
    ncl *= 2;
  const int per = (rows + ncl - 1) / ncl;
  const size_t smem = static_cast<size_t>(per) * cp_row_stride(jb) * sizeof(float);
  if (smem > CP_MAX_SMEM) return false;
  static bool usable = false;
  static std::once_flag probe;
  std::call_once(probe, [] {
    auto prepare = [](auto* kernel) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
          cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(CP_MAX_SMEM)) !=
              cudaSuccess)
        return false;
      cudaLaunchConfig_t q = {};
      q.gridDim = dim3(CP_CL, 1, 1);
      q.blockDim = dim3(CP_THREADS, 1, 1);
      q.dynamicSmemBytes = CP_MAX_SMEM;
      cudaLaunchAttribute qa[1];
      qa[0].id = cudaLaunchAttributeClusterDimension;
      qa[0].val.clusterDim.x = CP_CL;
      qa[0].val.clusterDim.y = 1;
      qa[0].val.clusterDim.z = 1;
      q.attrs = qa;
      q.numAttrs = 1;
      int nclusters = 0;
      return cudaOccupancyMaxActiveClusters(&nclusters, kernel, &q) == cudaSuccess && nclusters > 0;
    };
    usable = prepare(panel_cluster16_kernel<1>) && prepare(panel_cluster16_kernel<2>) &&
             prepare(panel_cluster16_kernel<4>);
    cudaGetLastError();  // clear a refused attribute or query
  });
  if (!usable) return false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncl, 1, 1);
  cfg.blockDim = dim3(cp_threads(per), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream();
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ncl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int rpt = (per + static_cast<int>(cfg.blockDim.x) - 1) / static_cast<int>(cfg.blockDim.x);
  auto* kernel = rpt == 1 ? panel_cluster16_kernel<1> : rpt == 2 ? panel_cluster16_kernel<2> : panel_cluster16_kernel<4>;
  if (rpt > 4) return false;
  cuda_check(cudaLaunchKernelEx(&cfg, kernel, A, ld, N, j0, jb, per, ipiv, info, swap_map, err, wait_ns, stall),
             "panel cluster kernel");
  ctx->launches += 1;
  return true;
}

// Applies a panel's row moves to every column outside the panel, one warp
// per column: all sources are read into registers before any write.
constexpr int SWAP_PER_LANE = 8;  // 2 jb <= 256 = 32 x 8 moves
template <class T>
__global__ void laswp_map(T* __restrict__ A, long long ld, int N, int j0, int jb, const int* __restrict__ map,
                          int* __restrict__ perm) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int ncol = N - jb;
  if (warp > ncol) return;
  if (warp == ncol) {  // the pivot order (P b)[i] = b[perm[i]] moves like a column
    const int n = map[0];
    int v[SWAP_PER_LANE];
#pragma unroll
    for (int q = 0; q < SWAP_PER_LANE; q++)
      if (lane + 32 * q < n) v[q] = perm[map[1 + 2 * jb + lane + 32 * q]];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < SWAP_PER_LANE; q++)
      if (lane + 32 * q < n) perm[map[1 + lane + 32 * q]] = v[q];
    return;
  }
  const int c = (warp < j0) ? warp : warp + jb;
  T* col = A + static_cast<long long>(c) * ld;
  const int n = map[0];
  const int* dst = map + 1;
  const int* src = map + 1 + 2 * jb;
  T v[SWAP_PER_LANE];
#pragma unroll
  for (int q = 0; q < SWAP_PER_LANE; q++) {
    int t = lane + 32 * q;
    if (t < n) v[q] = col[src[t]];
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < SWAP_PER_LANE; q++) {
    int t = lane + 32 * q;
    if (t < n && dst[t] != src[t]) col[dst[t]] = v[q];
  }
}

template <class T>
static bool panel_grid(Context* ctx, T* A, long long ld, int N, int j0, int jb, int* ipiv, int* info, int* map,
                       int nsm, const PanelSlots<T>& slots) {
  const int rows = N - j0;
  int nblk = (rows + GP_MIN_ROWS - 1) / GP_MIN_ROWS;
  if (nblk > nsm) nblk = nsm;
  if (nblk > 32 * GP_POLL_WARPS) nblk = 32 * GP_POLL_WARPS;
  const int per = (rows + nblk - 1) / nblk;
  nblk = (rows + per - 1) / per;
  size_t smem = static_cast<size_t>(per) * jb * sizeof(T);
  if (smem > GP_MAX_SMEM) return false;
  if (smem < GP_MIN_SMEM) smem = GP_MIN_SMEM;  // the row moves are listed there at the end
  static std::once_flag attr;
  std::call_once(attr, [] {
    cuda_check(cudaFuncSetAttribute(panel_grid_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(GP_MAX_SMEM)),
               "cudaFuncSetAttribute(panel)");
  });
  cudaStream_t s = ctx->stream();
  cuda_check(cudaMemsetAsync(slots.count, 0, sizeof(unsigned), s), "memset arrivals");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nblk, 1, 1);
  cfg.blockDim = dim3(GP_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cuda_check(cudaLaunchKernelEx(&cfg, panel_grid_kernel<T>, A, ld, N, j0, jb, per, ipiv, info, map, slots),
             "panel grid kernel");
  ctx->launches += 1;
  return true;
}

template <class T>
// Factors one panel; returns true when the panel kernel also wrote the
// panel's row-move list into swap_map (not the cluster that works in global
// memory).
static bool panel_factor(Context* ctx, T* A, long long ld, int N, int j0, int jb, int* ipiv, int* info, int nsm,
                         void* slot_mem, int* swap_map) {
  cudaStream_t s = ctx->stream();
  ProfScope ps(ctx, Context::PROF_LU_PANEL, 2.0 * sizeof(T) * jb * (N - j0));
  if (jb > 128) throw KdError(KD_ERR_ARG, "panel width above 128");
  PanelSlots<T> slots;
  {
    char* p = static_cast<char*>(slot_mem);
    slots.cand_rows = reinterpret_cast<T*>(p);
    p += sizeof(double) * 2 * 128 * static_cast<size_t>(nsm);
    slots.rec = reinterpret_cast<PanelRecord*>(p);
    p += sizeof(PanelRecord) * 2 * static_cast<size_t>(nsm);
    slots.jrow = reinterpret_cast<T*>(p);
    p += sizeof(double) * 2 * 128;
    slots.count = reinterpret_cast<unsigned*>(p);
    slots.err = reinterpret_cast<int*>(p + 16);
    slots.wait_ns = ctx->grid_wait_ns;
    slots.stall = ctx->stall_waits ? 1u : 0u;
  }
  if constexpr (std::is_same<T, float>::value) {
    if (panel_cluster16(ctx, A, ld, N, j0, jb, ipiv, info, swap_map, slots.err, slots.wait_ns, slots.stall)) return true;
  }
  if (panel_grid<T>(ctx, A, ld, N, j0, jb, ipiv, info, swap_map, nsm < ctx->sms() ? nsm : ctx->sms(), slots)) return true;
  // Panels too tall for the shared memory of the GPU: one 8-CTA cluster
  // working on the panel in global memory.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(PANEL_CL, 1, 1);
  cfg.blockDim = dim3(PANEL_THREADS, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PANEL_CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cuda_check(cudaLaunchKernelEx(&cfg, panel_cluster_kernel<T>, A, ld, N, j0, jb, ipiv, info), "panel cluster kernel");
  ctx->launches += 1;
  return false;
}

static void launch_trsm_chunk(Context* ctx, float* A, long long ld, int j0, int jb, int c0, int c1) {
  static std::once_flag attr;
  std::call_once(attr, [] {
    cuda_check(cudaFuncSetAttribute(trsm_chunk_f32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(TS_SMEM)),
               "cudaFuncSetAttribute(trsm)");
  });
  trsm_chunk_f32<<<blocks(c1 - c0, TS_COLS), TS_THREADS, TS_SMEM, ctx->stream()>>>(A, ld, j0, jb, c0, c1);
  ctx->launches += 1;
  cuda_check(cudaGetLastError(), "trsm kernel");
}

// The row exchanges of a factored panel in every other column.
template <class T>
static void exchange_rows(Context* ctx, T* A, long long ld, int N, int j0, int jb, const int* ipiv, int* map,
                          bool map_ready, int* perm) {
  cudaStream_t s = ctx->stream();
  if (!map_ready) {
    build_swap_map<<<1, 32, 0, s>>>(ipiv, j0, jb, map);
    ctx->launches += 1;
  }
  laswp_map<T><<<blocks(static_cast<long long>(N - jb + 1) * 32, 256), 256, 0, s>>>(A, ld, N, j0, jb, map, perm);
  ctx->launches += 1;
}

template <class T>
static void trsm_and_swaps(Context* ctx, T* A, long long ld, int N, int j0, int jb, const int* ipiv, int* map,
                           bool map_ready, int* perm) {
  cudaStream_t s = ctx->stream();
  ProfScope ps(ctx, Context::PROF_LU_SWAP_TRSM, 2.0 * sizeof(T) * jb * (N - j0 - jb));
  exchange_rows<T>(ctx, A, ld, N, j0, jb, ipiv, map, map_ready, perm);
  if (j0 + jb < N) {
    if constexpr (std::is_same<T, float>::value) {
      launch_trsm_chunk(ctx, A, ld, j0, jb, j0 + jb, N);
    } else {
      static std::once_flag attr_set;
      std::call_once(attr_set, [] {
        cuda_check(cudaFuncSetAttribute(trsm_chunk_f64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(TD_SMEM)),
                   "cudaFuncSetAttribute(trsm)");
      });
      trsm_chunk_f64<<<blocks(N - j0 - jb, TD_COLS), TD_THREADS, TD_SMEM, s>>>(A, ld, j0, jb, j0 + jb, N);
      ctx->launches += 1;
    }
  }
  cuda_check(cudaGetLastError(), "laswp/trsm kernels");
}

// Trailing updates of at least this many rows go to the sliced tensor-core
// product, smaller ones to the library's FP64 GEMM, whose single launch is as
// fast there (all updates of an N = 500 factorisation: 0.20 against 0.23 ms; N =
// 1,000: 0.48 against 0.93; N = 2,000: 1.2 against 5.5).
constexpr int F64_SLICED_MIN = 256;

void DenseLU::factor_fp64(double* A, long long ld, int N) {
  const int NB = nb > 96 ? 96 : nb;  // L11 + one column tile fit in shared memory
  cudaStream_t s = ctx_->stream();
  cuda_check(cudaMemsetAsync(d_info_, 0, sizeof(int), s), "memset info");
  for (int j0 = 0; j0 < N; j0 += NB) {
    int jb = (N - j0 < NB) ? N - j0 : NB;
    const bool map_ready = panel_factor<double>(ctx_, A, ld, N, j0, jb, ipiv_, d_info_, nsm_, slot_mem_, swap_map_);
    trsm_and_swaps<double>(ctx_, A, ld, N, j0, jb, ipiv_, swap_map_, map_ready, perm_);
    int m = N - j0 - jb;
    if (m > 0) {
      // A22 -= A21 * A12
      const double one = 1.0, mone = -1.0;
      ProfScope ps(ctx_, Context::PROF_LU_GEMM, 2.0 * m * m * jb);
      double* A21 = A + static_cast<long long>(j0) * ld + j0 + jb;
      double* A12 = A + static_cast<long long>(j0 + jb) * ld + j0;
      double* A22 = A + static_cast<long long>(j0 + jb) * ld + j0 + jb;
      if (m >= F64_SLICED_MIN && f64_sliced_update_possible(jb)) {
        f64_sliced_update(ctx_, m, m, jb, A21, ld, A12, ld, A22, ld);
        continue;
      }
      if (cublasDgemm(blas_, CUBLAS_OP_N, CUBLAS_OP_N, m, m, jb, &mone, A21, static_cast<int>(ld), A12,
                      static_cast<int>(ld), &one, A22, static_cast<int>(ld)) != CUBLAS_STATUS_SUCCESS)
        throw KdError(KD_ERR_CUDA, "cublasDgemm failed");
      ctx_->launches++;
    }
  }
}

void DenseLU::factor_f32(float* A, long long ld, int N, bool tf32) {
  const int NB = nb > 96 ? 96 : nb;
  cudaStream_t s = ctx_->stream();
  cuda_check(cudaMemsetAsync(d_info_, 0, sizeof(int), s), "memset info");
  // Panel width (blocked LU allows any widths).  A cluster panel of 96 or
  // 64 columns when its rows fit one 16-CTA cluster.  Taller panels: 96
  // columns on the cooperative grid when it holds them, since each panel
  // costs one pass of the trailing matrix through HBM in the update and a
  // 32-column panel triples that traffic; a 32-column cluster panel when the
  // grid cannot (a context limited to a share of the SMs).
  const int nsm_eff = nsm_ < ctx_->sms() ? nsm_ : ctx_->sms();
  auto on_cluster = [&](int rows) {
    if (NB != 96) return false;
    if (cluster_panel_width(rows, 64) > 0) return true;
    return !grid_panel_fits(rows, 96, nsm_eff, sizeof(float)) && cluster_panel_width(rows) > 0;
  };
  // A panel on the grid has no look-ahead, so it may as well be two: 192 columns
  // as two halves of 96, the right one brought up to date between them, and one
  // trailing update with k = 192 for both, which streams the trailing matrix
  // through HBM half as often.  N = 40,081: updates 362 -> 294 ms with all of the
  // right halves' extra products, the factorisation 519 -> 452 ms.  (Cluster
  // panels stay at 96 or 64: their updates run beside the next panel.)
  const int NW = 2 * NB;
  auto wide = [&](int rows) {
    return tf32 && tf32_terms == 3 && rows > NW && !on_cluster(rows) &&
           grid_panel_fits(rows, NB, nsm_eff, sizeof(float)) &&
           tf32x3_gemm_possible(NW, A, ld, 4, 4);  // panels start at multiples of 4, so A stands for every C
  };
  auto width = [&](int j0) {
    const int rows = N - j0;
    int w = NB;
    if (on_cluster(rows)) w = cluster_panel_width(rows);
    else if (wide(rows)) w = NW;
    return (rows < w) ? rows : w;
  };
  auto at = [&](int row, int col) { return A + static_cast<long long>(col) * ld + row; };
  auto panel = [&](int j0, int jb) {
    return panel_factor<float>(ctx_, A, ld, N, j0, jb, ipiv_, d_info_, nsm_, slot_mem_, swap_map_);
  };
  // Factors the panel of jb columns; of a wide one both halves, with the left
  // half's row exchanges in every column.
  auto factor_panel = [&](int j0, int jb) {
    const bool left = panel(j0, jb <= NB ? jb : NB);
    if (jb <= NB) return left;
    {
      ProfScope ps(ctx_, Context::PROF_LU_SWAP_TRSM, 2.0 * sizeof(float) * NB * (N - j0 - NB));
      exchange_rows<float>(ctx_, A, ld, N, j0, NB, ipiv_, swap_map_, left, perm_);
      launch_trsm_chunk(ctx_, A, ld, j0, NB, j0 + NB, j0 + jb);
    }
    gemm_update_f32(ctx_, blas_, N - j0 - NB, jb - NB, NB, at(j0 + NB, j0), ld, at(j0, j0 + NB), ld,
                    at(j0 + NB, j0 + NB), ld, tf32, static_cast<int>(ld - j0 - NB), tf32_terms);
    return panel(j0 + NB, jb - NB);
  };
  // The (right half's) row exchanges and U12 = L11^-1 A12 over the trailing columns.
  auto finish_panel = [&](int j0, int jb, bool ready) {
    if (jb <= NB) {
      trsm_and_swaps<float>(ctx_, A, ld, N, j0, jb, ipiv_, swap_map_, ready, perm_);
      return;
    }
    const int c0 = j0 + jb;
    {
      ProfScope ps(ctx_, Context::PROF_LU_SWAP_TRSM, 2.0 * sizeof(float) * NB * (N - c0));
      exchange_rows<float>(ctx_, A, ld, N, j0 + NB, jb - NB, ipiv_, swap_map_, ready, perm_);
      if (c0 < N) launch_trsm_chunk(ctx_, A, ld, j0, NB, c0, N);
    }
    if (c0 >= N) return;
    gemm_update_f32(ctx_, blas_, jb - NB, N - c0, NB, at(j0 + NB, j0), ld, at(j0, c0), ld, at(j0 + NB, c0), ld, tf32,
                    jb - NB, tf32_terms);
    ProfScope ps(ctx_, Context::PROF_LU_SWAP_TRSM, 2.0 * sizeof(float) * (jb - NB) * (N - c0));
    launch_trsm_chunk(ctx_, A, ld, j0 + NB, jb - NB, c0, N);
  };
  // Look-ahead (tensor-core update only): the columns of the next panel are
  // updated first, then the rest of the trailing update runs on a side
  // stream as 16-CTA clusters that leave one GPC free, while the next panel
  // is factored on the main stream; the next row exchanges wait for both.
  // A panel on the cooperative grid needs every SM, so it cannot run beside
  // the update: look-ahead only when the next panel fits a cluster.
  const bool lookahead = tf32 && tf32_update_max_clusters16() >= 2;
  int j0 = 0, jb = width(0);
  bool map_ready = factor_panel(j0, jb);
  bool side_pending = false;
  for (;;) {
    if (side_pending) {
      ctx_->join();
      side_pending = false;
    }
    finish_panel(j0, jb, map_ready);
    const int m = N - j0 - jb;
    if (m <= 0) break;
    const int j0n = j0 + jb, jbn = width(j0n);
    float* A21 = A + static_cast<long long>(j0) * ld + j0 + jb;
    float* A12 = A + static_cast<long long>(j0 + jb) * ld + j0;
    float* A22 = A + static_cast<long long>(j0 + jb) * ld + j0 + jb;
    // rows N .. ld of the working matrix are padding
    const int writable = static_cast<int>(ld - j0 - jb);
    if (lookahead && m > jbn && on_cluster(N - j0n)) {
      gemm_update_f32(ctx_, blas_, m, jbn, jb, A21, ld, A12, ld, A22, ld, tf32, writable, tf32_terms);
      ctx_->fork(1);
      ctx_->use(0);
      gemm_update_f32(ctx_, blas_, m, m - jbn, jb, A21, ld, A12 + static_cast<long long>(jbn) * ld, ld,
                      A22 + static_cast<long long>(jbn) * ld, ld, tf32, writable, tf32_terms, true);
      ctx_->use(-1);
      side_pending = true;
    } else {
      gemm_update_f32(ctx_, blas_, m, m, jb, A21, ld, A12, ld, A22, ld, tf32, writable, tf32_terms);
    }
    map_ready = factor_panel(j0n, jbn);
    j0 = j0n;
    jb = jbn;
  }
  if (side_pending) ctx_->join();
}

// Static-pivot factorisation of the FP32 working copy, whose rows are
// already in the pivot order of an earlier factorisation.  Panels are 192
// columns wide, each made of two 96-column halves: the left half is factored
// (panel_nopiv_kernel: the diagonal block and L21 in one launch), its U12
// over the right half solved, the right half updated below it, then
// factored.  The U12 solve of a wide panel goes the same way by halves, and
// the trailing update runs with k = 192 on the tensor cores, which streams
// the trailing matrix through HBM half as often as 96-column panels would.
// Columns that do not fill a wide panel take 96-column panels.  No row
// exchanges, no grid-wide synchronisation.
void DenseLU::factor_f32_nopiv(float* A, long long ld, int N, bool tf32) {
  cudaStream_t s = ctx_->stream();
  cuda_check(cudaMemsetAsync(d_info_, 0, sizeof(int), s), "memset info");
  const int NB = NP_NB, NW = 2 * NP_NB;
  auto at = [&](int row, int col) { return A + static_cast<long long>(col) * ld + row; };
  auto panel = [&](int j0, int jb) {
    const int m = N - j0 - jb;
    ProfScope ps(ctx_, Context::PROF_LU_PANEL_STATIC, 2.0 * sizeof(float) * jb * (N - j0));
    // at most NP_MAX_CTAS CTAs: the SMs left beside the trailing update's
    // 16-CTA clusters; equal shares in whole 128-byte lines
    int rows = ((m + NP_MAX_CTAS - 1) / NP_MAX_CTAS + 31) / 32 * 32;
    if (rows < NP_MIN_ROWS) rows = NP_MIN_ROWS;
    const int grid = m > 0 ? blocks(m, rows) : 1;
    static std::once_flag attr;
    std::call_once(attr, [] {
      cuda_check(cudaFuncSetAttribute(panel_nopiv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NP_XS_BYTES),
                 "panel_nopiv smem");
    });
    panel_nopiv_kernel<<<grid, NP_THREADS, NP_XS_BYTES, ctx_->stream()>>>(A, ld, N, j0, jb, rows, d_info_, np_done_);
    ctx_->launches++;
  };
  auto trsm = [&](int j0, int jb, int c0, int c1) {
    ProfScope ps(ctx_, Context::PROF_LU_SWAP_TRSM, 2.0 * sizeof(float) * jb * (c1 - c0));
    launch_trsm_chunk(ctx_, A, ld, j0, jb, c0, c1);
  };
  // a panel of jb <= 96 columns, or a wide one of 192 as two halves
  auto wide_panel = [&](int j0, int jb) {
    if (jb <= NB) {
      panel(j0, jb);
      return;
    }
    panel(j0, NB);
    trsm(j0, NB, j0 + NB, j0 + jb);
    const int mr = N - j0 - NB;
    gemm_update_f32(ctx_, blas_, mr, jb - NB, NB, at(j0 + NB, j0), ld, at(j0, j0 + NB), ld, at(j0 + NB, j0 + NB), ld,
                    tf32, static_cast<int>(ld - j0 - NB), tf32_terms, 0, NP_MAX_CTAS);
    panel(j0 + NB, jb - NB);
  };
  // U12 = L11^-1 A12 for the panel's rows over columns [c0, c1)
  auto wide_trsm = [&](int j0, int jb, int c0, int c1) {
    if (jb <= NB) {
      trsm(j0, jb, c0, c1);
      return;
    }
    trsm(j0, NB, c0, c1);
    gemm_update_f32(ctx_, blas_, jb - NB, c1 - c0, NB, at(j0 + NB, j0), ld, at(j0, c0), ld, at(j0 + NB, c0), ld, tf32,
                    jb - NB, tf32_terms);
    trsm(j0 + NB, jb - NB, c0, c1);
  };
  auto width = [&](int j0) { return N - j0 >= NW ? NW : (N - j0 < NB ? N - j0 : NB); };
  // Look-ahead (tensor-core update): the next panel's columns are updated
  // first, then the rest of the trailing update runs on a side stream as
  // every 16-CTA cluster the GPU holds, while the next panel is factored on
  // the main stream on the SMs left; the next U12 solve waits for both.
  const bool lookahead = tf32 && tf32_update_max_clusters16() >= 2;
  int j0 = 0, jb = width(0);
  wide_panel(j0, jb);
  bool side_pending = false;
  for (;;) {
    if (side_pending) {
      ctx_->join();
      side_pending = false;
    }
    const int m = N - j0 - jb;
    if (m <= 0) break;
    wide_trsm(j0, jb, j0 + jb, N);
    const int j0n = j0 + jb, jbn = width(j0n);
    float* A21 = at(j0 + jb, j0);
    float* A12 = at(j0, j0 + jb);
    float* A22 = at(j0 + jb, j0 + jb);
    const int writable = static_cast<int>(ld - j0 - jb);
    if (lookahead && m > jbn) {
      gemm_update_f32(ctx_, blas_, m, jbn, jb, A21, ld, A12, ld, A22, ld, tf32, writable, tf32_terms);
      ctx_->fork(1);
      ctx_->use(0);
      gemm_update_f32(ctx_, blas_, m, m - jbn, jb, A21, ld, A12 + static_cast<long long>(jbn) * ld, ld,
                      A22 + static_cast<long long>(jbn) * ld, ld, tf32, writable, tf32_terms, 2);
      ctx_->use(-1);
      side_pending = true;
    } else {
      gemm_update_f32(ctx_, blas_, m, m, jb, A21, ld, A12, ld, A22, ld, tf32, writable, tf32_terms);
    }
    wide_panel(j0n, jbn);
    j0 = j0n;
    jb = jbn;
  }
  if (side_pending) ctx_->join();
  cuda_check(cudaGetLastError(), "static-pivot factorisation");
}

// FP32 working copy of the FP64 matrix (equilibrated, rows in the order
// `perm` when it is given) and its factorisation: with perm, the
// static-pivot path; without, partial pivoting.
void DenseLU::factor_mixed(double* A, long long ld, int N, int mode, const int* perm) {
  double* rs = eq_buf_;
  double* cs = eq_buf_ + N;
  unsigned long long* rmax = reinterpret_cast<unsigned long long*>(eq_buf_ + 2 * static_cast<size_t>(N));
  cudaStream_t st = ctx_->stream();
  const size_t column = sizeof(float) * static_cast<size_t>(N);
  const bool keep = perm && column <= SC_MAX_SMEM;
  if (keep) {
    static std::once_flag attr;
    std::call_once(attr, [] {
      cuda_check(cudaFuncSetAttribute(scale_convert_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(SC_MAX_SMEM)),
                 "cudaFuncSetAttribute(working copy)");
      cuda_check(cudaFuncSetAttribute(scale_convert_kernel<true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      cudaSharedmemCarveoutMaxShared),
                 "cudaFuncSetAttribute(working copy)");
    });
  }
  auto convert = [&](const double* r, double* c) {
    if (keep)
      scale_convert_kernel<true><<<N, SC_THREADS, column, st>>>(A, ld, r, N, c, A32_, ld32_, perm);
    else
      scale_convert_kernel<false><<<N, SC_THREADS, 0, st>>>(A, ld, r, N, c, A32_, ld32_, perm);
  };
  if (equilibrate) {
    cuda_check(cudaMemsetAsync(rmax, 0, sizeof(unsigned long long) * N, st), "memset row max");
    const int rb = blocks(N, 256);
    int nch = (4 * nsm_ + rb - 1) / rb;
    if (nch < 1) nch = 1;
    const int chunk = (N + nch - 1) / nch;
    nch = (N + chunk - 1) / chunk;
    row_absmax_kernel<<<dim3(rb, nch), 256, 0, st>>>(A, ld, N, chunk, rmax);
    row_scale_kernel<<<rb, 256, 0, st>>>(rmax, N, rs);
    convert(rs, cs);
    ctx_->launches += 3;
  } else {
    convert(nullptr, nullptr);
    ctx_->launches++;
  }
  scaled_ = equilibrate;
  iota_kernel<<<blocks(N, 256), 256, 0, st>>>(ipiv_, N);
  if (!perm) iota_kernel<<<blocks(N, 256), 256, 0, st>>>(perm_, N);
  ctx_->launches++;
  if (perm) {
    factor_f32_nopiv(A32_, ld32_, N, mode == LU_TF32_IR);
    prepare_solves<float>(A32_, ld32_, N);
  } else {
    factor_f32(A32_, ld32_, N, mode == LU_TF32_IR);
    prepare_solves<float>(A32_, ld32_, N);
  }
  nopiv_ = perm != nullptr;
}

int DenseLU::read_info() {
  int info = 0;
  cuda_check(cudaMemcpyAsync(&info, d_info_, sizeof(int), cudaMemcpyDeviceToHost, ctx_->stream()), "D2H info");
  cuda_check(cudaStreamSynchronize(ctx_->stream()), "sync after LU");
  return info;
}

void DenseLU::factor(double* A, long long ld, int N, int mode) {
  if (N <= 0) throw KdError(KD_ERR_ARG, "empty matrix");
  double t0 = now_ms();
  mode_ = mode;
  N_ = N;
  ld_ = ld;
  A_ = A;
  if (static_cast<size_t>(N) > ipiv_cap_) {
    cudaFree(ipiv_);
    cuda_check(cudaMalloc(&ipiv_, sizeof(int) * N), "cudaMalloc(ipiv)");
    ipiv_cap_ = N;
  }
  if (static_cast<size_t>(N) > perm_cap_) {
    cudaFree(perm_);
    cudaFree(tri_work_);
    cuda_check(cudaMalloc(&perm_, sizeof(int) * N), "cudaMalloc(perm)");
    // two FP64 vectors, then two FP32 vectors (the chained sweeps' copies)
    cuda_check(cudaMalloc(&tri_work_, sizeof(double) * 3 * (((static_cast<size_t>(N) + 31) / 32) * 32)),
               "cudaMalloc(tri work)");
    perm_cap_ = N;
  }
  stats = LuStats();
  stats.flops = static_cast<long long>(2.0 / 3.0 * double(N) * N * N);
  iota_kernel<<<blocks(N, 256), 256, 0, ctx_->stream()>>>(ipiv_, N);
  ctx_->launches++;
  if (mode == LU_FP64) {
    iota_kernel<<<blocks(N, 256), 256, 0, ctx_->stream()>>>(perm_, N);
    factor_fp64(A, ld, N);
    prepare_solves<double>(A, ld, N);
    nopiv_ = false;
  } else {
    ld32_ = ((static_cast<long long>(N) + 31) / 32) * 32;  // 128-byte aligned columns
    const size_t need = static_cast<size_t>(ld32_) * N;
    if (need > a32_cap_) {
      cudaFree(A32_);
      cuda_check(cudaMalloc(&A32_, need * sizeof(float)), "cudaMalloc(A32)");
      a32_cap_ = need;
    }
    if (static_cast<size_t>(N) > eq_cap_) {
      cudaFree(eq_buf_);
      cuda_check(cudaMalloc(&eq_buf_, sizeof(double) * 3 * static_cast<size_t>(N)), "cudaMalloc(equilibration)");
      eq_cap_ = N;
    }
    // later factorisations of a matrix of the same size reuse the pivot
    // order of the last partial-pivoting factorisation (static pivoting)
    const bool reuse = reuse_pivots && perm_n_ == N;
    factor_mixed(A, ld, N, mode, reuse ? perm_ : nullptr);
    if (reuse && read_info() != 0) {
      // a zero or non-finite pivot in that order: factor with partial pivoting
      stats.static_pivot_fallback = 1;
      perm_n_ = 0;
      factor_mixed(A, ld, N, mode, nullptr);
    }
  }
  int info = read_info();
  stats.t_factor_ms = now_ms() - t0;
  int perr = 0;
  cuda_check(cudaMemcpyAsync(&perr, panel_err_, sizeof(int), cudaMemcpyDeviceToHost, ctx_->stream()),
             "D2H panel flag");
  cuda_check(cudaStreamSynchronize(ctx_->stream()), "sync panel flag");
  if (perr) {
    cuda_check(cudaMemsetAsync(panel_err_, 0, sizeof(int), ctx_->stream()), "reset panel flag");
    throw KdError(KD_ERR_TIMEOUT, "panel factorisation: a grid barrier wait ran out (or a cluster panel's exchange wait)");
  }
  if (mode != LU_FP32_IR && tf32_gemm_error_flag(ctx_))
    throw KdError(KD_ERR_TIMEOUT, "tensor-core trailing update timed out waiting for its MMAs");
  if (info != 0) throw KdError(KD_ERR_SINGULAR, "Jacobian is singular (zero pivot at column " + std::to_string(info) + ")");
  if (!nopiv_) perm_n_ = N;  // perm_ holds this factorisation's pivot order
  stats.static_pivots = nopiv_ ? 1 : 0;
}

// x = xscale (LU)^-1 (bscale b), or with the transposed factors: two sweeps,
// one launch each, and the pivot order's permutation.  Scales null: 1 (FP64
// factors: always).
template <class T>
void DenseLU::tri_solve(const T* LU, long long ld, int N, const double* b, double* x, int trans, const double* bscale,
                        const double* xscale) {
  cudaStream_t s = ctx_->stream();
  // work of one sweep: the triangle of the factors it reads
  const double sweep_bytes = 0.5 * sizeof(T) * N * static_cast<double>(N);
  const int nblk = (N + TB - 1) / TB;
  const size_t rnd = ((static_cast<size_t>(N) + 31) / 32) * 32;
  double* w1 = tri_work_;
  double* w2 = tri_work_ + rnd;  // 256-byte aligned second vector
  constexpr bool kF = std::is_same<T, float>::value;
  constexpr int RC = kF ? CH_RF : CH_R;
  static std::once_flag ch_attr;
  std::call_once(ch_attr, [] {
    auto smem = [](auto* kernel, size_t bytes) {
      cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)),
                 "cudaFuncSetAttribute(chain sweep)");
    };
    if constexpr (kF) smem(trsv_group, sizeof(TgShared));
    else smem(trsv_chain<T, false, RC>, CH_SMEM<RC>);
    smem(trsv_chain<T, true, RC>, CH_SMEM<RC>);
  });
  // one group of blocks per CTA while the device holds that many CTAs;
  // more groups go round the context's SMs.  The sums' order does not depend
  // on the grid, so concurrent and serial solves agree bit for bit.
  const bool groups = kF && !trans;
  const int R = groups ? TG : RC;
  const int gch = (nblk + R - 1) / R;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(gch <= nsm_ ? gch : ctx_->sms(), 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = groups ? sizeof(TgShared) : CH_SMEM<RC>;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const unsigned stall = ctx_->stall_waits ? 1u : 0u;
  // FP32 copies of the two sweeps' outputs (group sweeps only)
  float* yf = reinterpret_cast<float*>(tri_work_ + 2 * rnd);
  if (groups)
    cuda_check(cudaMemsetAsync(yf, 0xff, 2 * rnd * sizeof(float), s), "memset sweep outputs");
  else if (kF)
    cuda_check(cudaMemsetAsync(w1, 0xff, 2 * rnd * sizeof(double), s), "memset sweep outputs");
  else
    cuda_check(cudaMemsetAsync(tri_bar_, 0, 2 * sizeof(unsigned), s), "memset sweep progress");
  if (kF && trans) prepare_transposed();
  // sweep number k over L (or its transpose) or U; scales on entry, and on exit
  // where x is not read back by the sweep itself
  auto sweep = [&](int k, bool over_l, const double* in, const double* iscale, double* out, const double* oscale,
                   const char* what) {
    ProfScope ps(ctx_, Context::PROF_LU_SOLVE, sweep_bytes);
    const int ascending = k == 0 ? 1 : 0;
    if constexpr (kF)
      if (groups) {
        cuda_check(cudaLaunchKernelEx(&cfg, trsv_group, LU, ld, N, in, iscale, out, oscale, yf + k * rnd,
                                      over_l ? dinv2_l_ : dinv2_u_, over_l ? group_x_l_ : group_x_u_, ascending,
                                      panel_err_, ctx_->grid_wait_ns, stall),
                   what);
        return;
      }
    auto* kernel = trsv_chain<T, true, RC>;
    if constexpr (!kF)
      if (!trans) kernel = trsv_chain<T, false, RC>;
    cuda_check(cudaLaunchKernelEx(&cfg, kernel, LU, ld, N, in, iscale, out, over_l ? dinv_l_ : dinv_u_, ascending,
                                  tri_bar_ + k, panel_err_, ctx_->grid_wait_ns, stall),
               what);
  };
  if (!trans) {
    // L y = P b, then U x = y
    gather_perm<<<blocks(N, 256), 256, 0, s>>>(b, perm_, bscale, N, w1);
    sweep(0, true, w1, nullptr, w2, nullptr, "forward sweep");
    sweep(1, false, w2, nullptr, x, xscale, "backward sweep");
  } else {
    // A^T = U^T L^T P: U^T y = b (forward), L^T z = y (backward), x = P^T z
    sweep(0, false, b, bscale, w2, nullptr, "forward transposed sweep");
    sweep(1, true, w2, nullptr, w1, nullptr, "backward transposed sweep");
    scatter_perm<<<blocks(N, 256), 256, 0, s>>>(w1, perm_, xscale, N, x);
  }
  ctx_->launches += 3;
  cuda_check(cudaGetLastError(), "triangular solve");
}

void DenseLU::solve_fp64(const double* LU, long long ld, int N, double* b, int trans) {
  tri_solve<double>(LU, ld, N, b, b, trans, nullptr, nullptr);
}

void DenseLU::solve_f32(const double* b, double* x, int trans) {
  // M^-1 b = D_c (LU)^-1 (D_r b) with the equilibrated factors LU of
  // P D_r A D_c; transposed, M^-T b = D_r (LU)^-T (D_c b)
  const double* first = trans ? eq_buf_ + N_ : eq_buf_;
  const double* last = trans ? eq_buf_ : eq_buf_ + N_;
  tri_solve<float>(A32_, ld32_, N_, b, x, trans, scaled_ ? first : nullptr, scaled_ ? last : nullptr);
}

// A sweep that gave up is reported first (its garbage also stops the
// refinement), and its flag is cleared so the context stays usable.
void DenseLU::check_sweeps() {
  cuda_check(cudaStreamSynchronize(ctx_->stream()), "sync after solve");
  int perr = 0;
  cuda_check(cudaMemcpyAsync(&perr, panel_err_, sizeof(int), cudaMemcpyDeviceToHost, ctx_->stream()),
             "D2H sweep flag");
  cuda_check(cudaStreamSynchronize(ctx_->stream()), "sync sweep flag");
  if (perr) {
    cuda_check(cudaMemsetAsync(panel_err_, 0, sizeof(int), ctx_->stream()), "reset sweep flag");
    cuda_check(cudaStreamSynchronize(ctx_->stream()), "sync sweep flag reset");
    throw KdError(KD_ERR_TIMEOUT, "triangular solve: a grid barrier wait ran out");
  }
}

void DenseLU::ensure_bsave() {
  if (static_cast<size_t>(N_) > bsave_cap_) {
    cudaFree(bsave_);
    bsave_ = nullptr;
    cuda_check(cudaMalloc(&bsave_, sizeof(double) * N_), "cudaMalloc(rhs copy)");
    bsave_cap_ = N_;
  }
}

void DenseLU::ensure_dinv(size_t need) {
  if (need <= dinv_cap_) return;
  cudaFree(dinv_l_);
  cudaFree(dinv_u_);
  dinv_l_ = dinv_u_ = nullptr;
  dinv_cap_ = 0;
  cuda_check(cudaMalloc(&dinv_l_, need * sizeof(double)), "cudaMalloc(Linv)");
  cuda_check(cudaMalloc(&dinv_u_, need * sizeof(double)), "cudaMalloc(Uinv)");
  dinv_cap_ = need;
}

template <class T>
void DenseLU::invert_blocks(const T* LU, long long ld, int N, double* linv, double* uinv, float2* linv2,
                            float2* uinv2) {
  constexpr size_t smem = sizeof(double) * (TB * TB + TB * (TB + 1));
  static std::once_flag attr_set;
  std::call_once(attr_set, [] {
    cuda_check(cudaFuncSetAttribute(invert_diag_blocks<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(smem)),
               "cudaFuncSetAttribute(diagonal inverses)");
  });
  invert_diag_blocks<T><<<dim3((N + TB - 1) / TB, 2), ID_THREADS, smem, ctx_->stream()>>>(LU, ld, N, linv, uinv, linv2,
                                                                                         uinv2);
  ctx_->launches++;
}

// The FP64 inverses of the diagonal blocks of FP32 factors, which only their
// transposed sweeps read: made when the first of them needs them.
void DenseLU::prepare_transposed() {
  if (transposed_ready_) return;
  ensure_dinv(static_cast<size_t>((N_ + TB - 1) / TB) * TB * TB);
  invert_blocks<float>(A32_, ld32_, N_, dinv_l_, dinv_u_, nullptr, nullptr);
  transposed_ready_ = true;
}

// After factorisation: inverses of the 64 x 64 diagonal blocks of L (unit lower)
// and U, and with FP32 factors of the groups.
template <class T>
void DenseLU::prepare_solves(const T* LU, long long ld, int N) {
  const int nblk = (N + TB - 1) / TB;
  const size_t need = static_cast<size_t>(nblk) * TB * TB;
  constexpr bool kF = std::is_same<T, float>::value;
  transposed_ready_ = false;
  if constexpr (kF) {
    if (need > dinv2_cap_) {
      cudaFree(dinv2_l_);
      cudaFree(dinv2_u_);
      dinv2_l_ = dinv2_u_ = nullptr;
      dinv2_cap_ = 0;
      cuda_check(cudaMalloc(&dinv2_l_, need * sizeof(float2)), "cudaMalloc(Linv pairs)");
      cuda_check(cudaMalloc(&dinv2_u_, need * sizeof(float2)), "cudaMalloc(Uinv pairs)");
      dinv2_cap_ = need;
    }
    invert_blocks<float>(LU, ld, N, nullptr, nullptr, dinv2_l_, dinv2_u_);
  } else {
    ensure_dinv(need);
    invert_blocks<double>(LU, ld, N, dinv_l_, dinv_u_, nullptr, nullptr);
  }
  if constexpr (std::is_same<T, float>::value) {
    const int ng = (nblk + TG - 1) / TG;
    const size_t gx = static_cast<size_t>(ng) * TB * TB;
    if (gx > group_x_cap_) {
      cudaFree(group_x_l_);
      cudaFree(group_x_u_);
      group_x_l_ = group_x_u_ = nullptr;
      group_x_cap_ = 0;
      cuda_check(cudaMalloc(&group_x_l_, gx * sizeof(float2)), "cudaMalloc(group inverses)");
      cuda_check(cudaMalloc(&group_x_u_, gx * sizeof(float2)), "cudaMalloc(group inverses)");
      group_x_cap_ = gx;
    }
    static std::once_flag gi_attr;
    std::call_once(gi_attr, [] {
      cuda_check(cudaFuncSetAttribute(invert_groups, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(GI_SMEM)),
                 "cudaFuncSetAttribute(group inverses)");
    });
    if (nblk > 1) {
      invert_groups<<<dim3(ng, 2), 256, GI_SMEM, ctx_->stream()>>>(LU, ld, N, dinv2_l_, dinv2_u_, group_x_l_, group_x_u_);
      ctx_->launches++;
    } else {  // one block: nothing beside it
      cuda_check(cudaMemsetAsync(group_x_l_, 0, gx * sizeof(float2), ctx_->stream()), "memset group inverses");
      cuda_check(cudaMemsetAsync(group_x_u_, 0, gx * sizeof(float2), ctx_->stream()), "memset group inverses");
    }
  }
  cuda_check(cudaGetLastError(), "solve preparation");
}

// Right-preconditioned GMRES(m) in FP64 with the FP32 LU as preconditioner:
// solves A x = b to a relative residual below gmres_tol.  Small dense
// Hessenberg algebra runs on the host (m <= 50), vectors stay on the device.
void DenseLU::gemv(const double* x, double* y, double alpha, double beta, const double* b, int trans) {
  const int N = N_;
  cudaStream_t s = ctx_->stream();
  if (trans) {
    gemv_t_kernel<<<blocks(N, GEMVT_WARPS), GEMVT_WARPS * 32, 0, s>>>(A_, ld_, N, x, alpha, beta, b, y);
    ctx_->launches++;
    return;
  }
  const int rb = blocks(N, GEMV_ROWS);
  int nchunk = (16 * nsm_ + rb - 1) / rb;  // the device's SMs: the split of the sums stays fixed
  if (nchunk > GEMV_MAX_CHUNKS) nchunk = GEMV_MAX_CHUNKS;
  if (nchunk > (N + 15) / 16) nchunk = (N + 15) / 16;  // shorter chunks cost more in gemv_finish than they save
  if (nchunk < 1) nchunk = 1;
  const int chunk = (N + nchunk - 1) / nchunk;
  nchunk = (N + chunk - 1) / chunk;
  const size_t need = static_cast<size_t>(GEMV_MAX_CHUNKS) * N;
  if (need > part_cap_) {
    cudaFree(part_);
    cuda_check(cudaMalloc(&part_, need * sizeof(double)), "cudaMalloc(gemv partials)");
    part_cap_ = need;
  }
  gemv_partial<<<dim3(rb, nchunk), GEMV_ROWS, 0, s>>>(A_, ld_, N, x, chunk, part_);
  gemv_finish<<<blocks(N, 32), 32 * GEMV_SHARES, 0, s>>>(part_, nchunk, N, alpha, beta, b, y);
  ctx_->launches += 2;
}

void DenseLU::gmres_ir(double* b, int trans) {
  // Right-preconditioned GMRES(m), M^-1 = the FP32 factors.  The basis is
  // orthogonalised by classical Gram-Schmidt run twice (CGS2): per
  // iteration two passes of dot products and one norm on the device, one
  // copy of the results to the host; the small Hessenberg least-squares
  // problem is solved on the host.  At most gmres_restarts cycles.  With
  // trans the operator is A^T and the preconditioner M^-T.
  const int N = N_;
  const int m = gmres_max_iter;
  cudaStream_t s = ctx_->stream();
  const int nb = blocks(N, VA_THREADS);
  const size_t hn_at = 2 * static_cast<size_t>(m + 1);  // projections of both passes, then the CTAs' shares of |w|^2
  ensure_work(static_cast<size_t>(N) * (m + 4) + hn_at + nb);
  if (hproj_cap_ < hn_at + nb) {
    if (hproj_) cudaFreeHost(hproj_);
    hproj_ = nullptr;
    hproj_cap_ = 0;
    cuda_check(cudaMallocHost(&hproj_, (hn_at + nb) * sizeof(double)), "cudaMallocHost(projections)");
    hproj_cap_ = hn_at + nb;
  }
  double* V = work_;  // m + 1 basis vectors
  double* w = work_ + static_cast<size_t>(N) * (m + 1);
  double* x = w + N;
  double* r = x + N;
  double* dproj = r + N;  // [0, m+1): first pass, [m+1, 2m+2): second pass, then |w|^2's shares
  auto copy_scaled = [&](const double* src, double alpha, double* dst) {
    scaled_copy<<<nb, VA_THREADS, 0, s>>>(N, alpha, src, dst, 0);
    ctx_->launches++;
  };
  auto add_scaled = [&](const double* src, double alpha, double* dst) {
    scaled_copy<<<nb, VA_THREADS, 0, s>>>(N, alpha, src, dst, 1);
    ctx_->launches++;
  };
  auto host_norm = [&] {
    double sum = 0.0;
    for (int i = 0; i < nb; i++) sum += hproj_[hn_at + i];
    return std::sqrt(sum);
  };
  auto norm = [&](const double* v) {
    sum_squares<<<nb, VA_THREADS, 0, s>>>(v, N, dproj + hn_at);
    ctx_->launches++;
    cuda_check(cudaMemcpyAsync(hproj_ + hn_at, dproj + hn_at, nb * sizeof(double), cudaMemcpyDeviceToHost, s),
               "D2H norm");
    cuda_check(cudaStreamSynchronize(s), "sync norm");
    return host_norm();
  };
  cuda_check(cudaMemsetAsync(x, 0, sizeof(double) * N, s), "memset x");
  const double bnorm = norm(b);
  if (bnorm == 0) return;
  int total_it = 0;
  bool checked = false;
  for (int restart = 0; restart < gmres_restarts; restart++) {
    // r = b - A x (x = 0 on the first cycle: r = b, no matvec)
    if (restart == 0) {
      cuda_check(cudaMemcpyAsync(r, b, sizeof(double) * N, cudaMemcpyDeviceToDevice, s), "copy b");
    } else {
      ProfScope ps(ctx_, Context::PROF_GMRES, 8.0 * double(N) * N);
      gemv(x, r, -1.0, 1.0, b, trans);
    }
    const double beta = norm(r);
    stats.final_rel_residual = beta / bnorm;
    if (beta / bnorm < gmres_tol) {
      checked = true;  // of this very x
      break;
    }
    std::vector<double> H(static_cast<size_t>(m + 1) * m, 0.0), cs(m), sn(m), g(m + 1, 0.0);
    g[0] = beta;
    copy_scaled(r, 1.0 / beta, V);
    int k = 0;
    for (; k < m; k++) {
      // w = A M^-1 v_k
      solve_f32(V + static_cast<size_t>(k) * N, r, trans);
      {
        ProfScope ps(ctx_, Context::PROF_GMRES, 8.0 * double(N) * N);
        gemv(r, w, 1.0, 0.0, nullptr, trans);
      }
      // two passes of w -= V (V^T w) over v_0 .. v_k, then |w|^2
      const int kk = k + 1;
      for (int pass = 0; pass < 2; pass++) {
        double* h = dproj + static_cast<size_t>(pass) * (m + 1);
        basis_dots<<<kk, VD_THREADS, 0, s>>>(V, N, w, h);
        basis_subtract<<<nb, VA_THREADS, 0, s>>>(V, N, kk, h, w, pass ? dproj + hn_at : nullptr);
        ctx_->launches += 2;
      }
      cuda_check(cudaMemcpyAsync(hproj_, dproj, (hn_at + nb) * sizeof(double), cudaMemcpyDeviceToHost, s),
                 "D2H projections");
      cuda_check(cudaStreamSynchronize(s), "sync projections");
      const double hn = host_norm();
      for (int i = 0; i <= k; i++) H[static_cast<size_t>(i) * m + k] = hproj_[i] + hproj_[m + 1 + i];
      H[static_cast<size_t>(k + 1) * m + k] = hn;
      if (hn > 0) copy_scaled(w, 1.0 / hn, V + static_cast<size_t>(k + 1) * N);
      for (int i = 0; i < k; i++) {
        const double t = cs[i] * H[i * m + k] + sn[i] * H[(i + 1) * m + k];
        H[(i + 1) * m + k] = -sn[i] * H[i * m + k] + cs[i] * H[(i + 1) * m + k];
        H[i * m + k] = t;
      }
      const double a = H[k * m + k], c = H[(k + 1) * m + k];
      const double d = std::sqrt(a * a + c * c);
      cs[k] = d > 0 ? a / d : 1.0;
      sn[k] = d > 0 ? c / d : 0.0;
      H[k * m + k] = d;
      H[(k + 1) * m + k] = 0;
      g[k + 1] = -sn[k] * g[k];
      g[k] = cs[k] * g[k];
      total_it++;
      if (std::fabs(g[k + 1]) / bnorm < gmres_tol || hn == 0) {
        k++;
        break;
      }
    }
    // y = H^-1 g, x += M^-1 V y
    std::vector<double> y(k, 0.0);
    for (int i = k - 1; i >= 0; i--) {
      double sum = g[i];
      for (int j = i + 1; j < k; j++) sum -= H[i * m + j] * y[j];
      y[i] = sum / H[i * m + i];
    }
    if (k == 0) cuda_check(cudaMemsetAsync(w, 0, sizeof(double) * N, s), "memset w");
    for (int i0 = 0; i0 < k; i0 += COMBINE_MAX) {
      CombineCoefs c;
      const int n = std::min(COMBINE_MAX, k - i0);
      for (int i = 0; i < n; i++) c.c[i] = y[i0 + i];
      basis_combine<<<nb, VA_THREADS, 0, s>>>(V + static_cast<size_t>(i0) * N, N, n, c, w, i0 > 0);
      ctx_->launches++;
    }
    solve_f32(w, r, trans);
    add_scaled(r, 1.0, x);
  }
  if (!checked) {
    {
      ProfScope ps(ctx_, Context::PROF_GMRES, 8.0 * double(N) * N);
      gemv(x, r, -1.0, 1.0, b, trans);
    }
    stats.final_rel_residual = norm(r) / bnorm;
  }
  stats.refine_iters = total_it;
  cuda_check(cudaMemcpyAsync(b, x, sizeof(double) * N, cudaMemcpyDeviceToDevice, s), "copy x");
}

void DenseLU::solve(double* b, int trans) {
  double t0 = now_ms();
  if (mode_ == LU_FP64) {
    solve_fp64(A_, ld_, N_, b, trans);
  } else if (trans) {
    // A^T x = b: GMRES on A^T preconditioned by the transposed factors
    // (no fallback to new factors: the caller decides)
    gmres_ir(b, 1);
    check_sweeps();
  } else {
    if (nopiv_) {
      ensure_bsave();
      cuda_check(cudaMemcpyAsync(bsave_, b, sizeof(double) * N_, cudaMemcpyDeviceToDevice, ctx_->stream()),
                 "keep right-hand side");
    }
    gmres_ir(b);
    check_sweeps();
    if (nopiv_) {
      if (!(stats.final_rel_residual < 1e-10)) {
        // the reused pivot order does not precondition this matrix: factor
        // it with partial pivoting and solve again
        stats.static_pivot_fallback = 1;
        perm_n_ = 0;
        factor_mixed(A_, ld_, N_, mode_, nullptr);
        const int info = read_info();
        if (info != 0)
          throw KdError(KD_ERR_SINGULAR, "Jacobian is singular (zero pivot at column " + std::to_string(info) + ")");
        perm_n_ = N_;
        cuda_check(cudaMemcpyAsync(b, bsave_, sizeof(double) * N_, cudaMemcpyDeviceToDevice, ctx_->stream()),
                   "restore right-hand side");
        gmres_ir(b);
        check_sweeps();
      } else if (stats.refine_iters > pivoted_iters_ + 4) {
        perm_n_ = 0;  // the order has drifted: the next factorisation pivots again
      }
    }
    if (!nopiv_) pivoted_iters_ = stats.refine_iters;
  }
  check_sweeps();
  if (mode_ != LU_FP64 && !(stats.final_rel_residual < 1e-10))
    throw KdError(KD_ERR_NOCONV, "GMRES-IR did not converge (relative residual " +
                                     std::to_string(stats.final_rel_residual) + ")");
  stats.t_solve_ms = now_ms() - t0;
}

}  // namespace kd
