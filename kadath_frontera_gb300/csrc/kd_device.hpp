// Device-side descriptors and kernel launchers (implemented in kd_device.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace kd {

// One output of a line pass: sum_q m[m0 + q mstep] x[x0 + q xstep], q < count,
// stored at y0.  Only the nonzero range of the matrix row is listed; count 0
// stores a zero.  steps = count | mstep << 12 | xstep << 14.
struct KdOut {
  int x0, m0, y0;
  unsigned steps;
};

// One 1-D pass of a separable operator over a 3-D block (r, theta, phi), phi
// fastest, as the list of its outputs (ordered so that the outputs of a warp
// have the same count) and of the mirrored pairs that are replaced by their
// sum and difference in the pass's input (before) and output (after).
struct KdPass {
  int dim;
  int n_in;
  int n_out;
  int nout;            // outputs
  int nbefore, nafter; // pairs
  const KdOut* out;    // null in every pass of an item: no lists, see mat
  const int* pairs;    // first element | second << 16: before, then after
  // The lines' matrices (row-major n_out x n_in) as offsets in doubles into the
  // pool, -1 for a line whose output is zero, for passes without lists and for
  // fields with non-finite values:
  //   dim 0 (r):     mat[j * mat_ld + k]   (basis depends on theta/phi indices)
  //   dim 1 (theta): mat[k]                (basis depends on the phi index)
  //   dim 2 (phi):   mat[0]
  const int* mat;
  int mat_ld;
};

// A run of `batch` fields of identical shape processed by the same pass list.
struct KdItem {
  const double* in;
  double* out;
  long long in_stride;   // elements between consecutive fields of the batch
  long long out_stride;
  int n0, n1, n2;        // input dims
  int npass;
  int stage;             // doubles of the largest stage in shared memory
  int pitch;             // row pitch (phi) of the input staged in shared memory
  int nmats;             // doubles of the matrices staged in shared memory (0: read from the pool)
  double scale;          // applied to the final result
  const double* mats;    // the matrices to stage, 16-byte aligned
  KdPass pass[3];
};

// Up to KD_MAX_ITEMS runs packed in one launch (uneven domains together).
// Passed by value as a kernel parameter so that launches can be captured in
// a CUDA graph without staging descriptors through host memory.
constexpr int KD_MAX_ITEMS = 12;
struct KdItemList {
  int nitems;
  int prefix[KD_MAX_ITEMS + 1];  // prefix sums of batch sizes
  KdItem items[KD_MAX_ITEMS];
};

// The same with one item: a tenth of the parameter bytes of a launch.
struct KdItemList1 {
  int nitems;
  int prefix[2];
  KdItem items[1];
};

// Single-field operations collected by a pass and launched level by level
// (Context::begin_batch): one CTA per operation, up to KD_MAX_OPS of them with
// no dependence on one another in a launch.
constexpr int KD_MAX_OPS = 400;  // 32,008 bytes of the 32,764 that kernel parameters may take
enum KdOpKind : int { KD_OP_LINE = 0, KD_OP_EW = 1, KD_OP_GATHER = 2 };
struct KdOpRec {
  int kind;
  int sub;           // elementwise operation; gather: accumulate
  int n;             // elementwise: points; gather: rows
  int smem;          // line passes: doubles of shared memory
  const void* p[5];  // line: item (its in and out unused), in, out; ew: a, b, out; gather: in, out, rowptr, idx, w
  double alpha, beta;
  long long osr;     // gather: stride of the output rows
};
cudaError_t launch_ops(const KdOpRec* ops, int n, const double* d_pool, cudaStream_t s);

// Launch shape of a line-pass launch: one CTA of `threads` threads per field
// (cluster = 1), or a cluster of `cluster` CTAs (2, 4 or 8) of 128 threads
// per field, each CTA computing every cluster-th block of a pass's outputs.
// Every output value is summed in the same order whatever the shape, so the
// shape changes no result bit.
struct LpShape {
  int cluster = 1;
  int threads = 128;
};
// The rule without a tuning table, from the fields of the launch and the
// doubles of the largest item's stage.  Up to 32 fields are bound by latency:
// clusters of 8 CTAs, or of 4 where the field is small or there are too many
// clusters for each of their CTAs to have an SM of its own (us per launch with
// 8 / 4 CTAs: one (9,5,4) field 6.2 / 6.2, 30 of them 10.2 / 6.2; (21,11,14)
// fields 20.7 / 26.9 up to 12 of them, 28.9 / 26.9 for 32; (33,17,16) 49.5 / 75.7
// for 12, 94.5 / 76.0 for 16).  Beyond that one 256-thread CTA per field (150
// fields of (15,11,12): 26.6 against 42.4 with 128 threads and 39.5 with clusters
// of 4), except that large fields that leave half of the SMs idle keep clusters
// of 4 (60 fields of (21,11,14): 34.0 against 43.0), and that small fields, whose
// passes have fewer outputs than 256 threads, take 128 threads once there are more
// than four of them an SM (3,600 fields: (5,5,4) 23.5 against 29.0, (9,5,4) 35.1
// against 39.9, (11,7,4) 59.8 against 61.9, (13,9,4) 90.2 against 90.3; 300 of
// (9,5,4) 10.5 against 9.7).
LpShape lp_default_shape(int total_fields, int stage);

// Runs the pass lists of all items with the given shape (default rule: the
// overload without one).
cudaError_t launch_line_passes(const KdItemList& list, const double* d_pool, cudaStream_t s, LpShape shape);
cudaError_t launch_line_passes(const KdItemList& list, const double* d_pool, cudaStream_t s);

// Elementwise ops on fields of npts values. a has ba fields, b has bb fields
// (ba, bb in {1, B}); out has max(ba, bb) fields.
enum EwOp : int {
  EW_ADD = 0,    // a + b
  EW_SUB = 1,    // a - b
  EW_MUL = 2,    // a * b
  EW_DIV = 3,    // a / b
  EW_AXPBY = 4,  // alpha*a + beta*b
  EW_SCALE = 5,  // alpha*a
  EW_ADDC = 6,   // a + alpha
  EW_CSUB = 7,   // alpha - a
  EW_CDIV = 8,   // alpha / a
  EW_POWD = 9,   // pow(a, alpha)
  EW_EXP = 10,
  EW_LOG = 11,
  EW_SQRT = 12,
  EW_SIN = 13,
  EW_COS = 14,
  EW_NEG = 15,
  EW_FILL = 16,  // alpha
  EW_COPY = 17,  // a
  EW_POWI = 18,  // pow(a, (int)alpha) for alpha <= 0 (reference uses std::pow)
  EW_ATAN = 19,
  EW_MULC_ADD = 20,  // out = a*b*alpha (product with constant)
  EW_DIVC = 21,      // a / alpha (Val_domain / double divides, it does not scale by 1/alpha)
  EW_COSH = 22,
  EW_SINH = 23,
  EW_ATANH = 24,
};

cudaError_t launch_ew(int op, long long npts, int ba, const double* a, int bb, const double* b,
                      double* out, double alpha, double beta, cudaStream_t s);

// Sparse row gather (CSR): for each field f of the batch and row r,
//   out[f*osf + r*osr] (+)= alpha * sum_{e in [rowptr[r], rowptr[r+1])} w[e] * in[f*in_stride + idx[e]]
// in_stride = 0 broadcasts one input field to every output field.
cudaError_t launch_gather_csr(const double* in, long long in_stride, int batch, int nrows, const int* rowptr,
                              const int* idx, const double* w, double* out, long long osf, long long osr,
                              double alpha, int accumulate, cudaStream_t s);

// Sum over the last axis reduction helpers used by residual norms.
cudaError_t launch_absmax(const double* x, long long n, double* out_scalar, cudaStream_t s);
// Occupies the stream for about ns nanoseconds (profile mode queues the
// launches it times behind it, so that their event pairs see no host gaps).
cudaError_t launch_hold(unsigned long long ns, cudaStream_t s);
// Cold piecewise polytrope (Margherita Cold_PWPoly, include/EOS/standalone/
// cold_pwpoly_implementation.hh), geometrised units, tables derived as in
// Margherita_setup_polytrope (setup_polytrope.cc).
constexpr int KD_EOS_MAX_PIECES = 8;
struct KdEos {
  int npieces;
  double rhomin, rhomax;
  double k[KD_EOS_MAX_PIECES], gamma[KD_EOS_MAX_PIECES], rho[KD_EOS_MAX_PIECES], eps[KD_EOS_MAX_PIECES],
      h[KD_EOS_MAX_PIECES];
};
enum EosVar : int { EOS_EPSILON = 0, EOS_PRESSURE = 1, EOS_DENSITY = 2, EOS_DHDRHO = 3 };
// Value (dh == nullptr): out = var(h) pointwise (EOS::term_by_term).
// Variation: out[b] = d var for the tangent batch dh (B fields) at h
// (EOS::term_by_term_variation, include/EOS/EOS.hh:67-160).
cudaError_t launch_eos(const KdEos& eos, int var, long long npts, const double* h, int B, const double* dh,
                       double* out, cudaStream_t s);

// Deterministic single-CTA reduction: op 0 = sum of squares, 1 = max.
cudaError_t launch_reduce1(const double* x, long long n, int op, double* out_scalar, cudaStream_t s);
// out[i] = ca * (a ? a[i] : as) + cb * (b ? b[i] : bs), i < n: the tangent of
// a linear combination of doubles whose tangents differ from seed to seed.
cudaError_t launch_lincomb2(int n, double ca, const double* a, double as, double cb, const double* b, double bs,
                            double* out, cudaStream_t s);

// The first integral's residual in one domain (Eq_first_integral::export_val /
// export_der, src/Equation/eq_first_integral.cpp:44-120), for B seeds:
//   out[b][p] = (v ? v[b*vs + p] : 0) - (ori ? ori[b*os] : 0),
// and, when inject != 0, the first n0 points (radial index 0) replaced by
// (cst ? cst[b*cs] : cst_scalar).  All arrays at the collocation points.
cudaError_t launch_first_integral(int B, int npts, int n0, const double* v, long long vs, const double* ori,
                                  long long os, int inject, const double* cst, long long cs, double cst_scalar,
                                  double* out, cudaStream_t s);

}  // namespace kd
