// Trailing update of the FP64 LU, C -= A * B, on the tcgen05 tensor cores by
// exact products of 8-bit slices (the error-free splitting of Ozaki, Ogita,
// Oishi and Rump, Numer. Algorithms 59, 2012, in fixed point), entry by entry
// only where that loses nothing against a product in FP64.
//
// This GPU's FP64 pipe gives 1.1 TFLOP/s; its bf16 tensor cores 1,700 times
// that.  Each operand entry becomes a 62-bit fixed-point number F relative to
// the largest entry of its row of A (column of B), F = sum_s d_s 2^(8(8-s)),
// s = 1..8, with d_s in [-128, 127]: eight bf16 matrices of integers.  The
// product of slices i and j has integer entries, summed exactly in FP32: an
// order o = i + j adds at most 8 pairs of k <= 128 products below 2^14, at
// most 2^24 in all.  Orders 2..9 (36 of the 64 pairs) are kept.  Before
// splitting, row k of B is scaled by a power of two and column k of A by its
// inverse so that the mean exponents of their nonzero entries agree: then the k
// that are large in A's rows are those that are large in B's columns, and rows of
// B of very different sizes (a Jacobian's second derivatives beside its boundary
// rows) do not cost each other digits.  (With the largest entry of row k of B at 1
// instead, one outlier moved the whole row: of a matrix of 8,000 rows over six
// decades 54 million entries had to be listed below, 0.7 million now.)
//
// Error.  With R the bound 2^(row's scale + column's scale) of the products of
// an entry, the orders left out and the rounding of the digits come to about
// 2^-59 R (96 random digits; the 2^-63 of each entry's last digit is less), and
// the sum is rounded to FP64 once.  An FP64 product errs by about 2^-53 of
// sum_k |a_k b_k|, and the subtraction by 2^-53 of the result, so an entry is
// taken from the slices only where one of the two is at least 2^-4 R or so:
//   three or more k have |a_k| >= 2^-3 and |b_k| >= 2^-3 of their row's and
//   column's scale (bit masks made while packing), or
//   the sum itself, or the updated entry, is at least 2^-4 R in size.
// Every other entry, and every entry of a row or column with Inf or NaN, is left
// as it is and listed, and sum_listed forms it in FP64, as a plain product would.
// Unknowns in different units need that: where one row of B is small in every
// column but those of its own group, the sums in that group's columns are far
// below R (groups 40 binades apart: componentwise backward errors of 1e-8 to 1e-2
// with the slices alone, 7e-16 now and with LAPACK).  Sparse Jacobians too: of the
// star's entries 0.5 % (index notation) to 2.9 % are listed.
//
// One persistent CTA per SM, 128 x 64 tiles:
//   warp 0   TMA loads of operand chunks: k = 32 of all eight slices of A and
//            B (96 KB, 64-byte swizzle), two stages;
//   warp 1   72 MMAs per chunk (M 128, N 64, K 16) into eight accumulators of
//            64 TMEM columns, one per order: all 512 columns;
//   warps 2-17 epilogue: the eight orders of an entry into one integer of 80
//            bits, TMEM released, then C -= its first 62 bits * 2^e (one
//            conversion and one multiply-add on the FP64 pipe) beside the next
//            tile's MMAs, and the list of the entries to sum in FP64.
// Bound: the hand-over of the single set of accumulators and the latency of the
// epilogue behind it, 25,000 cycles a tile of which the tensor pipe works 29 %, the
// FP64 pipe 34 % and the issue slots 37 % (first update of N = 4,000).  128 x 64
// tiles and not 128 x 128: eight orders of 64 columns are all of TMEM, and one pass
// over the operands serves all of them.  (C prefetched into L2: 1 %.)
// Sixteen epilogue warps: with eight, of 32 columns each, their integer work was
// longer than a tile's MMAs (all updates at N = 8,000: 32 against 23 ms).
// All updates of a factorisation, with packing and the listed entries, against the
// library's FP64 GEMM: a dense matrix of N = 8,000 with rows over six decades 23
// against 319 ms, the star's Jacobian at N = 7,819 22 (index notation) and 28
// against 301, at N = 12,331 91 against 1,172.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "kd_gemm_tc.hpp"

namespace kd {

namespace {

constexpr int S_SLICES = 8;
constexpr int S_M = 128, S_N = 64, S_KC = 32;           // tile and k chunk
constexpr int S_MAXK = 128;                              // exact sums: 8 pairs x 128 x 2^14 = 2^24
constexpr int S_A_SLICE = S_M * S_KC * 2;                // bytes of one slice of a chunk
constexpr int S_B_SLICE = S_N * S_KC * 2;
constexpr int S_STAGE = S_SLICES * (S_A_SLICE + S_B_SLICE);
constexpr int S_NST = 2;
constexpr int S_EPI = 16;                                // epilogue warps
constexpr int S_THREADS = 64 + 32 * S_EPI;
constexpr int S_COLS = S_N / (S_EPI / 4);                // columns of an epilogue thread
constexpr size_t S_SMEM = 1024 + static_cast<size_t>(S_NST) * S_STAGE;
constexpr unsigned long long S_WAIT_NS = 2000000000ull;
constexpr int EXP_NONFINITE = 1 << 20;                   // scale of a row or column that holds Inf or NaN
constexpr int EXP_ZERO = -(1 << 20);                     // scale of a zero row or column
constexpr int NEAR = 2;                                  // binades below the scale that count as large
constexpr int NEAR_TERMS = 3;                            // large products that make a sum safe
constexpr int SAFE_BITS = 4;                             // binades below R of a safe sum or result
constexpr int MASK_WORDS = S_MAXK / 32;

// Bit of k in a mask, so that a warp's ballots over two k a lane are its words:
// word 2 (k / 64) + k % 2, bit (k % 64) / 2.  A row or column has two masks: of
// its large entries, then of its nonzero ones.
static_assert(S_MAXK == 128 && MASK_WORDS == 4, "two 64-wide halves, two words each");

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Smallest E with |v| < 2^E; EXP_ZERO for zero, EXP_NONFINITE for Inf and NaN.
__device__ __forceinline__ int exponent_of(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffull;
  const int e = static_cast<int>(b >> 52);
  if (e == 0x7ff) return EXP_NONFINITE;
  if (e != 0) return e - 1022;
  return b ? -1010 - __clzll(static_cast<long long>(b)) : EXP_ZERO;  // subnormal: b 2^-1074
}

// v * 2^(62 - scale) rounded to an integer, for |v| < 2^scale.
__device__ __forceinline__ long long fixed_point(double v, int scale) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  const int e = exponent_of(v);
  if (e == EXP_ZERO || e == EXP_NONFINITE) return 0;
  unsigned long long m = b & 0xfffffffffffffull;
  if (e > -1022) m |= 0x10000000000000ull;
  m <<= __clzll(static_cast<long long>(m)) - 2;  // first bit to place 61
  const int shift = scale - e;
  long long f;
  if (shift <= 0) f = static_cast<long long>(m);  // shift is never negative
  else if (shift > 62) f = 0;
  else f = static_cast<long long>((m + (1ull << (shift - 1))) >> shift);
  return (b >> 63) ? -f : f;
}

// The eight digits of f, most significant first, as bf16.
__device__ __forceinline__ void digits_of(long long f, __nv_bfloat16 (&d)[S_SLICES]) {
  // adding 128 to the lower seven bytes makes each of them its digit + 128
  const long long g = f + 0x0080808080808080ll;
  d[0] = __float2bfloat16_rn(static_cast<float>(static_cast<int>(g >> 56)));
#pragma unroll
  for (int s = 1; s < S_SLICES; s++)
    d[s] = __float2bfloat16_rn(static_cast<float>(static_cast<int>((g >> (8 * (7 - s))) & 255) - 128));
}

// Sums and numbers of the exponents of the nonzero finite entries of B's rows and
// A's columns, stat[quantity][kk]: 0 and 1 of B (k x n, column-major), 2 and 3 of A
// (m x k); stat starts at zero.  The first `nb` CTAs take STAT_COLS columns of B
// each, the others STAT_ROWS rows of one column of A.
constexpr int STAT_THREADS = 128, STAT_COLS = 32, STAT_ROWS = 2048;
__global__ void __launch_bounds__(STAT_THREADS) slice_exponents(const double* __restrict__ A, long long lda, int m,
                                                                const double* __restrict__ B, long long ldb, int k,
                                                                int n, int nb, int* __restrict__ stat) {
  static_assert(STAT_THREADS >= S_MAXK, "a thread a row of B");
  int sum = 0, count = 0;
  auto take = [&](double v) {
    const int e = exponent_of(v);
    if (e == EXP_NONFINITE || e == EXP_ZERO) return;
    sum += e;
    count++;
  };
  if (static_cast<int>(blockIdx.x) < nb) {
    const int kk = threadIdx.x, c0 = blockIdx.x * STAT_COLS, c1 = min(n, c0 + STAT_COLS);
    if (kk >= k) return;
#pragma unroll 8
    for (int c = c0; c < c1; c++) take(B[static_cast<long long>(c) * ldb + kk]);
    if (count) {
      atomicAdd(stat + kk, sum);
      atomicAdd(stat + S_MAXK + kk, count);
    }
    return;
  }
  const int t = blockIdx.x - nb, kk = t % k, r0 = t / k * STAT_ROWS, r1 = min(m, r0 + STAT_ROWS);
  const double* a = A + static_cast<long long>(kk) * lda;
#pragma unroll 8
  for (int r = r0 + threadIdx.x; r < r1; r += STAT_THREADS) take(a[r]);
  sum = __reduce_add_sync(0xffffffffu, sum);
  count = __reduce_add_sync(0xffffffffu, count);
  if ((threadIdx.x & 31) == 0 && count) {
    atomicAdd(stat + 2 * S_MAXK + kk, sum);
    atomicAdd(stat + 3 * S_MAXK + kk, count);
  }
}

// The exponent that row kk of B is divided by and column kk of A multiplied by.
__device__ __forceinline__ int balance(const int* __restrict__ stat, int kk) {
  const int nb = stat[S_MAXK + kk], na = stat[3 * S_MAXK + kk];
  if (nb == 0 || na == 0) return 0;
  return __float2int_rn(0.5f * (static_cast<float>(stat[kk]) / nb - static_cast<float>(stat[2 * S_MAXK + kk]) / na));
}

// Zeros: the statistics and, behind them, the length of the list.
constexpr int STAT_INTS = 4 * S_MAXK + 4;
__global__ void slice_clear(int* __restrict__ v) {
  for (int i = threadIdx.x; i < STAT_INTS; i += blockDim.x) v[i] = 0;
}

// Slices of B: out[s][column][kk] and the columns' scales; one warp a column.
__global__ void slice_pack_b(const double* __restrict__ B, long long ldb, int k, int n, int kpad, int npad,
                             const int* __restrict__ stat, __nv_bfloat16* __restrict__ out, int* __restrict__ scale,
                             uint4* __restrict__ masks) {
  const int col = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (col >= npad) return;
  double v[4];  // kk = 2 lane, 2 lane + 1, then + 64
  int x[4], ex[4], mx = EXP_ZERO;
  bool bad = false;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int kk = 2 * lane + (q & 1) + 64 * (q >> 1);
    v[q] = (col < n && kk < k) ? B[static_cast<long long>(col) * ldb + kk] : 0.0;
    x[q] = kk < k ? balance(stat, kk) : 0;
    ex[q] = exponent_of(v[q]);
    if (ex[q] == EXP_NONFINITE) bad = true;
    else if (ex[q] != EXP_ZERO) mx = max(mx, ex[q] - x[q]);
  }
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  bad = __any_sync(0xffffffffu, bad);
  unsigned large[MASK_WORDS], some[MASK_WORDS];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    some[q] = __ballot_sync(0xffffffffu, ex[q] != EXP_ZERO);
    large[q] = __ballot_sync(0xffffffffu, ex[q] != EXP_ZERO && ex[q] - x[q] >= mx - NEAR);
  }
  if (lane == 0) {
    scale[col] = bad ? EXP_NONFINITE : mx;
    masks[2 * col] = make_uint4(large[0], large[1], large[2], large[3]);
    masks[2 * col + 1] = make_uint4(some[0], some[1], some[2], some[3]);
  }
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const int kk = 2 * lane + 64 * p;
    if (kk >= kpad) continue;
    __nv_bfloat16 d0[S_SLICES], d1[S_SLICES];
    digits_of(fixed_point(v[2 * p], mx + x[2 * p]), d0);
    digits_of(fixed_point(v[2 * p + 1], mx + x[2 * p + 1]), d1);
#pragma unroll
    for (int s = 0; s < S_SLICES; s++)
      *reinterpret_cast<__nv_bfloat162*>(out + (static_cast<long long>(s) * npad + col) * kpad + kk) =
          __nv_bfloat162(d0[s], d1[s]);
  }
}

// Slices of A (m x k, column-major): out[s][row][kk] and the rows' scales; 32
// rows a CTA, staged so that reads run along rows and writes along kk.
constexpr int SA_ROWS = 32;
__global__ void __launch_bounds__(256) slice_pack_a(const double* __restrict__ A, long long lda, int m, int k,
                                                    int kpad, int mpad, const int* __restrict__ stat,
                                                    __nv_bfloat16* __restrict__ out, int* __restrict__ scale,
                                                    unsigned* __restrict__ masks) {
  __shared__ double t[S_MAXK][SA_ROWS + 1];
  __shared__ int x[S_MAXK], part[8][SA_ROWS], sc[SA_ROWS];
  const int r0 = blockIdx.x * SA_ROWS, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < S_MAXK; e += blockDim.x) x[e] = e < k ? balance(stat, e) : 0;
  __syncthreads();
  int mx = EXP_ZERO;
  for (int kk = w; kk < kpad; kk += 8) {
    const double v = (kk < k && r0 + lane < m) ? A[static_cast<long long>(kk) * lda + r0 + lane] : 0.0;
    t[kk][lane] = v;
    const int e = exponent_of(v);
    if (e == EXP_NONFINITE) mx = EXP_NONFINITE;
    else if (e != EXP_ZERO) mx = max(mx, e + x[kk]);
  }
  part[w][lane] = mx;
  __syncthreads();
  if (w == 0) {
    for (int q = 1; q < 8; q++) mx = max(mx, part[q][lane]);
    sc[lane] = mx;
    scale[r0 + lane] = mx;
  }
  __syncthreads();
  {  // warp w: word w % 4 of the large entries (w < 4) or of the nonzero ones
    const int s0 = sc[lane], word = w & (MASK_WORDS - 1);
    unsigned bits = 0;
    for (int i = 0; i < 32; i++) {
      const int kk = 64 * (word >> 1) + 2 * i + (word & 1);
      if (kk >= k) break;
      const int e = exponent_of(t[kk][lane]);
      if (e != EXP_ZERO && (w >= MASK_WORDS || e + x[kk] >= s0 - NEAR)) bits |= 1u << i;
    }
    masks[(2 * static_cast<size_t>(r0 + lane) + (w >= MASK_WORDS ? 1 : 0)) * MASK_WORDS + word] = bits;
  }
  const int pairs = kpad / 2;
  for (int e = threadIdx.x; e < SA_ROWS * pairs; e += blockDim.x) {
    const int r = e / pairs, kk = 2 * (e - r * pairs), s0 = sc[r];
    const bool some = s0 != EXP_NONFINITE && s0 != EXP_ZERO;
    __nv_bfloat16 d0[S_SLICES], d1[S_SLICES];
    digits_of(some ? fixed_point(t[kk][r], s0 - x[kk]) : 0, d0);
    digits_of(some ? fixed_point(t[kk + 1][r], s0 - x[kk + 1]) : 0, d1);
#pragma unroll
    for (int s = 0; s < S_SLICES; s++)
      *reinterpret_cast<__nv_bfloat162*>(out + (static_cast<long long>(s) * mpad + r0 + r) * kpad + kk) =
          __nv_bfloat162(d0[s], d1[s]);
  }
}

// ------------------------------------------------------------- the product --
__device__ __forceinline__ unsigned long long s_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait for phase `parity` of an mbarrier; false when it ran out.
__device__ __forceinline__ bool s_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
  uint32_t done = 0;
  unsigned long long t0 = 0;
  for (int spin = 0;; spin++) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (spin == 0) t0 = s_now();
    else if ((spin & 255) == 0 && s_now() - t0 > S_WAIT_NS) return false;
  }
}

__device__ __forceinline__ void s_load3(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(0), "r"(smem_addr(bar))
      : "memory");
}

// K-major operand, rows of 64 bytes, 64-byte swizzle: 8-row groups 512 bytes
// apart.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(512 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(4) << 61;  // SWIZZLE_64B
  return d;
}

// D = F32, A = B = BF16, both K-major.
__device__ constexpr uint32_t bf16_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_load4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

__global__ void __launch_bounds__(S_THREADS, 1)
    f64_update_sliced(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                      const int* __restrict__ ea, const int* __restrict__ fb, const uint4* __restrict__ ma,
                      const uint4* __restrict__ mb, uint2* __restrict__ list, unsigned* __restrict__ listed,
                      double* __restrict__ C, long long ldc, int m, int n, int nkc, int ntm, int ntiles,
                      int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char s_raw[];
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(s_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t op_full[S_NST], op_empty[S_NST], acc_full, acc_empty, drained;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_flag;
  volatile int* abort_v = &abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < S_NST; i++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&op_full[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&op_empty[i])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&acc_full)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&drained)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&acc_empty)), "n"(S_EPI));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapA)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mapB)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_sh)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_sh;

  if (warp == 0) {
    if (lane == 0) {  // ------------------------------------------- producer
      int g = 0;
      for (int tile = blockIdx.x; tile < ntiles && !*abort_v; tile += gridDim.x) {
        const int tm = tile % ntm, tn = tile / ntm;
        for (int kc = 0; kc < nkc; kc++, g++) {
          const int st = g % S_NST, use = g / S_NST;
          if (use > 0 && !s_wait(&op_empty[st], (use - 1) & 1)) {
            *abort_v = 1;
            break;
          }
          char* sp = base + st * S_STAGE;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&op_full[st])),
                       "r"(S_STAGE)
                       : "memory");
          s_load3(sp, &mapA, kc * S_KC, tm * S_M, &op_full[st]);
          s_load3(sp + S_SLICES * S_A_SLICE, &mapB, kc * S_KC, tn * S_N, &op_full[st]);
        }
      }
      // no copy may be in flight when the CTA leaves
      for (int st = 0; st < S_NST; st++) {
        const int uses = (g + S_NST - 1 - st) / S_NST;
        if (uses > 0 && !s_wait(&op_full[st], (uses - 1) & 1)) *abort_v = 1;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ----------------------------------------- MMA issuer
      const uint32_t idesc = bf16_idesc(S_M, S_N);
      int it = 0, g = 0;
      for (int tile = blockIdx.x; tile < ntiles && !*abort_v; tile += gridDim.x, it++) {
        if (it > 0 && !s_wait(&acc_empty, (it - 1) & 1)) {
          *abort_v = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        bool ok = true;
        for (int kc = 0; kc < nkc; kc++, g++) {
          const int st = g % S_NST;
          if (!s_wait(&op_full[st], (g / S_NST) & 1)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = smem_addr(base + st * S_STAGE), sb = sa + S_SLICES * S_A_SLICE;
          const uint64_t a0 = sw64_desc(sa), b0 = sw64_desc(sb);
          for (int o = 0; o < S_SLICES; o++) {  // order o + 2: slices i and o - i
            const uint32_t d = tmem + static_cast<uint32_t>(o * S_N);
            for (int i = 0; i <= o; i++) {
              const uint64_t ad = a0 + static_cast<uint64_t>((i * S_A_SLICE) >> 4);
              const uint64_t bd = b0 + static_cast<uint64_t>(((o - i) * S_B_SLICE) >> 4);
#pragma unroll
              for (int kk = 0; kk < S_KC / 16; kk++) {
                const uint32_t accum = (kc | i | kk) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
                    "l"(ad + static_cast<uint64_t>(2 * kk)), "l"(bd + static_cast<uint64_t>(2 * kk)), "r"(idesc),
                    "r"(accum));
              }
            }
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           smem_addr(&op_empty[st]))
                       : "memory");
        }
        if (!ok) {
          *abort_v = 1;
          break;
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_addr(&acc_full))
                     : "memory");
      }
      // nor an MMA when the tensor memory is freed
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_addr(&drained))
                   : "memory");
      if (!s_wait(&drained, 0)) *abort_v = 1;
    }
  } else {  // --------------------------------------------- epilogue (2-17)
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    int it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
      const int tm = tile % ntm, tn = tile / ntm;
      if (!s_wait(&acc_full, it & 1) || *abort_v) {
        *abort_v = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // a sum in units of 2^-68 R: v 2^16 + low
      long long v[S_COLS];
      unsigned low[S_COLS / 2];
      const uint32_t t0 = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(part * S_COLS);
#pragma unroll
      for (int c4 = 0; c4 < S_COLS; c4 += 4) {
        uint32_t r[S_SLICES][4];
#pragma unroll
        for (int o = 0; o < S_SLICES; o++) tmem_load4(t0 + static_cast<uint32_t>(o * S_N + c4), r[o]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 4; q++) {
          // orders 2..7 weigh 2^40 .. 1, orders 8 and 9 2^-8 and 2^-16
          long long hi = 0;
#pragma unroll
          for (int o = 0; o < 6; o++) hi = (hi << 8) + __float2int_rn(__uint_as_float(r[o][q]));
          const long long lo = (static_cast<long long>(__float2int_rn(__uint_as_float(r[6][q]))) << 8) +
                               __float2int_rn(__uint_as_float(r[7][q]));
          v[c4 + q] = hi + (lo >> 16);
          const unsigned l = static_cast<unsigned>(lo) & 0xffffu;
          if (q & 1) low[(c4 + q) / 2] |= l << 16;
          else low[(c4 + q) / 2] = l;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&acc_empty)) : "memory");
      // C -= s 2^(ea + fb - 52 - shift), s the first 62 bits of a sum
      const int row = tm * S_M + quarter * 32 + lane;
      const int col0 = tn * S_N + part * S_COLS;
      const int er = ea[row];
      const uint4 near_a = ma[2 * row];  // rows and columns up to a whole tile are packed
      double* cp = C + static_cast<long long>(col0) * ldc + row;
#pragma unroll
      for (int c4 = 0; c4 < S_COLS; c4 += 4) {
        double c[4];
        unsigned exact = 0;  // entries to sum in FP64: left as they are
#pragma unroll
        for (int q = 0; q < 4; q++)
          c[q] = row < m && col0 + c4 + q < n ? cp[static_cast<long long>(c4 + q) * ldc] : 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int ec = fb[col0 + c4 + q];
          if (er == EXP_NONFINITE || ec == EXP_NONFINITE) {
            exact |= 1u << q;
            continue;
          }
          if (er == EXP_ZERO || ec == EXP_ZERO) continue;
          const long long hi = v[c4 + q];
          const unsigned l = (low[(c4 + q) / 2] >> (16 * (q & 1))) & 0xffffu;
          const int shift = min(16, __clzll(hi < 0 ? ~hi : hi) - 2);
          const long long s = (hi << shift) + (l >> (16 - shift));
          if (s != 0) {
            const int e = er + ec - 52 - shift + 1023;
            const double x = static_cast<double>(s);
            if (e > 0 && e < 2047)
              c[q] = fma(-x, __longlong_as_double(static_cast<long long>(e) << 52), c[q]);
            else
              c[q] -= scalbn(x, e - 1023);
          }
          const uint4 near_b = mb[2 * (col0 + c4 + q)];
          const int near = __popc(near_a.x & near_b.x) + __popc(near_a.y & near_b.y) + __popc(near_a.z & near_b.z) +
                           __popc(near_a.w & near_b.w);
          const long long size = s < 0 ? -s : s;
          const int ex = static_cast<int>((__double2hiint(c[q]) >> 20) & 0x7ff) - 1022;
          if (near < NEAR_TERMS && (size >> (52 - SAFE_BITS + shift)) == 0 && ex <= er + ec - SAFE_BITS) exact |= 1u << q;
        }
        if (row >= m) exact = 0;
        if (__any_sync(0xffffffffu, exact != 0u)) {
          unsigned rows = 0;  // lane q: the rows listed of column q
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const unsigned w = __ballot_sync(0xffffffffu, (exact >> q) & 1u);
            if (lane == q && col0 + c4 + q < n) rows = w;
          }
          const unsigned have = __ballot_sync(0xffffffffu, rows != 0u);
          unsigned at = 0;
          if (lane == 0) at = atomicAdd(listed, static_cast<unsigned>(__popc(have)));
          at = __shfl_sync(0xffffffffu, at, 0) + __popc(have & ((1u << lane) - 1u));
          // a place is 32 rows of a column: fewer than 2^32 of them
          if (rows) list[at] = make_uint2(rows, static_cast<unsigned>(tm * (S_M / 32) + quarter) * n + col0 + c4 + lane);
        }
        if (row < m) {
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (col0 + c4 + q < n && !((exact >> q) & 1u)) cp[static_cast<long long>(c4 + q) * ldc] = c[q];
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && *abort_v) atomicExch(err, 1);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// C -= A B in FP64 for the listed entries, a warp a place of the list: the rows of
// a 32-row block (bits) in one column.  Bound: the FP64 pipe where much is listed,
// else latency; every SM full of warps, so that the loads of some (eight k at a
// time) hide behind others.  (The epilogue did this first, and then warps by
// column of the matrix: what is listed comes in clusters, so a few warps had most
// of it, and the updates of the N = 7,819 factorisation took 49 ms, now 22.)
constexpr int SUM_THREADS = 256;
// Rows of a place up to which they go one after the other, 32 lanes a row (3 or 4
// multiply-adds and 5 additions of a warp each), instead of side by side (k
// multiply-adds for all).
constexpr int SUM_FEW = 8;
__global__ void __launch_bounds__(SUM_THREADS) sum_listed(const uint2* __restrict__ list,
                                                         const unsigned* __restrict__ listed, const int* __restrict__ ea,
                                                         const int* __restrict__ fb, const uint4* __restrict__ ma,
                                                         const uint4* __restrict__ mb, const double* __restrict__ A,
                                                         long long lda, const double* __restrict__ B, long long ldb,
                                                         int k, double* __restrict__ C, long long ldc, int m, int n) {
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned count = *listed, step = gridDim.x * (SUM_THREADS / 32);
  for (unsigned at = blockIdx.x * (SUM_THREADS / 32) + (threadIdx.x >> 5); at < count; at += step) {
    const uint2 e = list[at];
    const int col = static_cast<int>(e.y % static_cast<unsigned>(n));
    const int row0 = static_cast<int>(e.y / static_cast<unsigned>(n)) * 32, row = row0 + lane;
    const double* pb = B + static_cast<long long>(col) * ldb;
    if (__popc(e.x) <= SUM_FEW) {  // the lanes share each row's terms
      double v[MASK_WORDS];
#pragma unroll
      for (int q = 0; q < MASK_WORDS; q++) v[q] = lane + 32 * q < k ? pb[lane + 32 * q] : 0.0;
      for (unsigned rows = e.x; rows; rows &= rows - 1) {
        const int r = row0 + __ffs(rows) - 1;
        double u[MASK_WORDS], sum = 0.0;
#pragma unroll
        for (int q = 0; q < MASK_WORDS; q++)
          u[q] = lane + 32 * q < k ? A[static_cast<long long>(lane + 32 * q) * lda + r] : 0.0;
#pragma unroll
        for (int q = 0; q < MASK_WORDS; q++) sum = fma(u[q], v[q], sum);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(ALL, sum, o);
        if (lane == 0) C[static_cast<long long>(col) * ldc + r] -= sum;
      }
      continue;
    }
    const bool mine = row < m && ((e.x >> lane) & 1u);
    const uint4 a = ma[2 * row + 1], b = mb[2 * col + 1];  // (rows up to a whole tile are packed)
    const bool whole = __any_sync(ALL, mine && ea[row] == EXP_NONFINITE) || fb[col] == EXP_NONFINITE;
    // the k that any of the rows needs: of half h, word 2 h holds the even ones, word 2 h + 1 the odd ones
    const unsigned any[MASK_WORDS] = {
        __reduce_or_sync(ALL, mine ? a.x & b.x : 0u), __reduce_or_sync(ALL, mine ? a.y & b.y : 0u),
        __reduce_or_sync(ALL, mine ? a.z & b.z : 0u), __reduce_or_sync(ALL, mine ? a.w & b.w : 0u)};
    const double* pa = A + min(row, m - 1);
    double sum = 0.0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const unsigned even = whole ? ALL : any[2 * h], odd = whole ? ALL : any[2 * h + 1];
      if (!(even | odd)) continue;
      for (int i = 0; i < 32; i += 4) {
        const int k0 = 64 * h + 2 * i;
        const unsigned ev = (even >> i) & 15u, od = (odd >> i) & 15u;
        if (!(ev | od) || k0 >= k) continue;
        double u[8], v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
          const bool in = k0 + q < k;
          u[q] = in ? pa[static_cast<long long>(k0 + q) * lda] : 0.0;
          v[q] = in ? pb[k0 + q] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (((q & 1 ? od : ev) >> (q >> 1)) & 1u) sum = fma(u[q], v[q], sum);
      }
    }
    if (mine) C[static_cast<long long>(col) * ldc + row] -= sum;
  }
}

// 3-D bf16 map of out[slice][row][kk]: boxes of 32 x rows x all slices.
void make_slice_map(CUtensorMap* map, const void* ptr, int kpad, int rows, int box_rows) {
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(kpad), static_cast<cuuint64_t>(rows),
                              static_cast<cuuint64_t>(S_SLICES)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(kpad) * 2, static_cast<cuuint64_t>(kpad) * 2 * rows};
  const cuuint32_t box[3] = {S_KC, static_cast<cuuint32_t>(box_rows), S_SLICES};
  const cuuint32_t estr[3] = {1, 1, 1};
  auto fn = tensor_map_encoder();
  if (!fn) throw KdError(KD_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw KdError(KD_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(r) + ")");
}

}  // namespace

// (k = S_MAXK could fill the 64-bit sum's last bit)
bool f64_sliced_update_possible(int k) { return k > 0 && k < S_MAXK && tensor_map_encoder() != nullptr; }

void f64_sliced_update(Context* ctx, int m, int n, int k, const double* A, long long lda, const double* B,
                       long long ldb, double* C, long long ldc) {
  if (m <= 0 || n <= 0 || k <= 0) return;
  cudaStream_t s = ctx->stream();
  const int kpad = (k + S_KC - 1) / S_KC * S_KC;
  const int mpad = (m + S_M - 1) / S_M * S_M, npad = (n + S_N - 1) / S_N * S_N;
  // slices, then the masks and scales (rows of A, columns of B), then the statistics and the list
  const size_t abytes = static_cast<size_t>(S_SLICES) * mpad * kpad * 2, bbytes = static_cast<size_t>(S_SLICES) * npad * kpad * 2;
  char* wa = static_cast<char*>(ctx->workspace(Context::WS_TC_A, abytes + (2 * sizeof(uint4) + sizeof(int)) * mpad));
  // a place of the list for every 32 rows of every column
  const size_t places = static_cast<size_t>((m + 31) / 32) * n;
  if (places >> 32) throw KdError(KD_ERR_ARG, "sliced FP64 update: matrix too large");
  char* wb = static_cast<char*>(ctx->workspace(
      Context::WS_TC_B,
      bbytes + (2 * sizeof(uint4) + sizeof(int)) * npad + sizeof(int) * STAT_INTS + sizeof(uint2) * places));
  auto* as = reinterpret_cast<__nv_bfloat16*>(wa);
  auto* bs = reinterpret_cast<__nv_bfloat16*>(wb);
  auto* ma = reinterpret_cast<uint4*>(wa + abytes);  // abytes and bbytes are multiples of 4,096
  auto* mb = reinterpret_cast<uint4*>(wb + bbytes);
  int* ea = reinterpret_cast<int*>(ma + 2 * mpad);
  int* fb = reinterpret_cast<int*>(mb + 2 * npad);
  int* stat = fb + npad;
  auto* listed = reinterpret_cast<unsigned*>(stat + 4 * S_MAXK);
  auto* list = reinterpret_cast<uint2*>(stat + STAT_INTS);  // 16-byte aligned: npad is a multiple of 64
  bool fresh = false;
  int* err = static_cast<int*>(ctx->workspace(Context::WS_TC_FLAG, sizeof(int), &fresh));
  if (fresh) cuda_check(cudaMemsetAsync(err, 0, sizeof(int), s), "memset err");
  static std::once_flag attr;
  std::call_once(attr, [] {
    cuda_check(cudaFuncSetAttribute(f64_update_sliced, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(S_SMEM)),
               "cudaFuncSetAttribute(sliced update)");
  });
  slice_clear<<<1, 256, 0, s>>>(stat);
  const int nb = (n + STAT_COLS - 1) / STAT_COLS, na = (m + STAT_ROWS - 1) / STAT_ROWS * k;
  slice_exponents<<<nb + na, STAT_THREADS, 0, s>>>(A, lda, m, B, ldb, k, n, nb, stat);
  slice_pack_b<<<(npad + 7) / 8, 256, 0, s>>>(B, ldb, k, n, kpad, npad, stat, bs, fb, mb);
  slice_pack_a<<<mpad / SA_ROWS, 256, 0, s>>>(A, lda, m, k, kpad, mpad, stat, as, ea, reinterpret_cast<unsigned*>(ma));
  CUtensorMap mA, mB;
  make_slice_map(&mA, as, kpad, mpad, S_M);
  make_slice_map(&mB, bs, kpad, npad, S_N);
  const int ntm = mpad / S_M, ntiles = ntm * (npad / S_N);
  const int grid = ntiles < ctx->sms() ? ntiles : ctx->sms();
  f64_update_sliced<<<grid, S_THREADS, S_SMEM, s>>>(mA, mB, ea, fb, ma, mb, list, listed, C, ldc, m, n, kpad / S_KC, ntm,
                                                   ntiles, err);
  sum_listed<<<8 * ctx->sms(), SUM_THREADS, 0, s>>>(list, listed, ea, fb, ma, mb, A, lda, B, ldb, k, C, ldc, m, n);
  ctx->launches += 6;
  cuda_check(cudaGetLastError(), "sliced FP64 trailing update");
}

}  // namespace kd
