#include "kd_spectral.hpp"

#include <algorithm>
#include <cstring>
#include <set>
#include <sstream>

namespace kd {

namespace {

int mat_offset(Context& ctx, int op, int basis, int n_in, int n_out, int* out_basis) {
  int idx = ctx.bank().get(op, basis, n_in, n_out);
  if (idx < 0) {
    std::ostringstream os;
    os << "1-D operator " << op_name(op) << " not defined for basis " << basis_name(basis) << " (n=" << n_in
       << ")";
    throw KdError(KD_ERR_UNSUPPORTED, os.str());
  }
  const Mat1d& m = ctx.bank().at(idx);
  if (out_basis) *out_basis = m.out_basis;
  return static_cast<int>(m.pool_offset);
}

}  // namespace

LinePassSpec ope_1d_spec(Context& ctx, int op, int dim, const Base& base, const int d[3], Base& base_out) {
  if (!base.def) throw KdError(KD_ERR_STATE, "basis not defined in ope_1d");
  LinePassSpec s;
  s.dim = dim;
  s.n_in = d[dim];
  s.n_out = d[dim];
  s.mat_ld = base.n2c;
  if (dim == 0) {
    s.offsets.resize(base.r.size());
    for (int j = 0; j < base.n1c; j++)
      for (int k = 0; k < base.n2c; k++) {
        int ob;
        s.offsets[j * base.n2c + k] = mat_offset(ctx, op, base.rb(j, k), d[0], d[0], &ob);
        base_out.rb(j, k) = ob;
      }
  } else if (dim == 1) {
    s.offsets.resize(base.t.size());
    for (int k = 0; k < base.n2c; k++) {
      int ob;
      s.offsets[k] = mat_offset(ctx, op, base.t[k], d[1], d[1], &ob);
      base_out.t[k] = ob;
    }
  } else {
    int ob;
    s.offsets.assign(1, mat_offset(ctx, op, base.p, d[2], d[2], &ob));
    base_out.p = ob;
  }
  return s;
}

std::vector<LinePassSpec> coef_specs(Context& ctx, const Base& base, const int np[3], const int nc[3]) {
  if (!base.def) throw KdError(KD_ERR_STATE, "Base not defined in Val_domain::coef");
  std::vector<LinePassSpec> v(3);
  // phi first (coef.cpp:98-99 loops d = ndim-1 .. 0)
  v[0].dim = 2;
  v[0].n_in = np[2];
  v[0].n_out = nc[2];
  v[0].mat_ld = 0;
  v[0].offsets = {mat_offset(ctx, OP_COEF, base.p, np[2], nc[2], nullptr)};
  v[1].dim = 1;
  v[1].n_in = np[1];
  v[1].n_out = nc[1];
  v[1].mat_ld = 0;
  // a phi coefficient that the phi transform leaves at zero (sin(0), the sine
  // at the highest frequency) stays zero through the theta and r transforms
  const Mat1d& phi = ctx.bank().at(ctx.bank().get(OP_COEF, base.p, np[2], nc[2]));
  std::vector<char> dead(nc[2]);
  for (int k = 0; k < nc[2]; k++) dead[k] = phi.row_zero(k);
  v[1].dead = v[2].dead = dead;
  v[1].offsets.resize(nc[2]);
  for (int k = 0; k < nc[2]; k++) v[1].offsets[k] = mat_offset(ctx, OP_COEF, base.t[k], np[1], nc[1], nullptr);
  v[2].dim = 0;
  v[2].n_in = np[0];
  v[2].n_out = nc[0];
  v[2].mat_ld = nc[2];
  v[2].offsets.resize(static_cast<size_t>(nc[1]) * nc[2]);
  for (int j = 0; j < nc[1]; j++)
    for (int k = 0; k < nc[2]; k++)
      v[2].offsets[j * nc[2] + k] = mat_offset(ctx, OP_COEF, base.rb(j, k), np[0], nc[0], nullptr);
  return v;
}

std::vector<LinePassSpec> coef_i_specs(Context& ctx, const Base& base, const int np[3], const int nc[3]) {
  if (!base.def) throw KdError(KD_ERR_STATE, "Base not defined in Val_domain::coef_i");
  std::vector<LinePassSpec> v(3);
  // a phi coefficient that contributes to no collocation value (its basis
  // function vanishes there) needs no r and theta transforms
  mat_offset(ctx, OP_COEF_I, base.p, nc[2], np[2], nullptr);
  const int phi_index = ctx.bank().get(OP_COEF_I, base.p, nc[2], np[2]);
  std::vector<char> dead(nc[2]);
  for (int k = 0; k < nc[2]; k++) dead[k] = ctx.bank().at(phi_index).column_zero(k);
  v[0].dim = 0;
  v[0].n_in = nc[0];
  v[0].n_out = np[0];
  v[0].mat_ld = nc[2];
  v[0].offsets.resize(static_cast<size_t>(nc[1]) * nc[2]);
  for (int j = 0; j < nc[1]; j++)
    for (int k = 0; k < nc[2]; k++)
      v[0].offsets[j * nc[2] + k] = mat_offset(ctx, OP_COEF_I, base.rb(j, k), nc[0], np[0], nullptr);
  v[0].dead = v[1].dead = dead;
  v[1].dim = 1;
  v[1].n_in = nc[1];
  v[1].n_out = np[1];
  v[1].mat_ld = 0;
  v[1].offsets.resize(nc[2]);
  for (int k = 0; k < nc[2]; k++) v[1].offsets[k] = mat_offset(ctx, OP_COEF_I, base.t[k], nc[1], np[1], nullptr);
  v[2].dim = 2;
  v[2].n_in = nc[2];
  v[2].n_out = np[2];
  v[2].mat_ld = 0;
  v[2].offsets = {mat_offset(ctx, OP_COEF_I, base.p, nc[2], np[2], nullptr)};
  return v;
}

std::vector<LinePassSpec> resample_specs(Context& ctx, const Base& base, const int nc_old[3], const int np_new[3]) {
  if (!base.def) throw KdError(KD_ERR_STATE, "Base not defined in the resampling");
  std::vector<LinePassSpec> v(3);
  v[0].dim = 0;
  v[0].n_in = nc_old[0];
  v[0].n_out = np_new[0];
  v[0].mat_ld = nc_old[2];
  v[0].offsets.resize(static_cast<size_t>(nc_old[1]) * nc_old[2]);
  for (int j = 0; j < nc_old[1]; j++)
    for (int k = 0; k < nc_old[2]; k++)
      v[0].offsets[j * nc_old[2] + k] = mat_offset(ctx, OP_RESAMPLE, base.rb(j, k), nc_old[0], np_new[0], nullptr);
  v[1].dim = 1;
  v[1].n_in = nc_old[1];
  v[1].n_out = np_new[1];
  v[1].mat_ld = 0;
  v[1].offsets.resize(nc_old[2]);
  for (int k = 0; k < nc_old[2]; k++)
    v[1].offsets[k] = mat_offset(ctx, OP_RESAMPLE, base.t[k], nc_old[1], np_new[1], nullptr);
  v[2].dim = 2;
  v[2].n_in = nc_old[2];
  v[2].n_out = np_new[2];
  v[2].mat_ld = 0;
  v[2].offsets = {mat_offset(ctx, OP_RESAMPLE, base.p, nc_old[2], np_new[2], nullptr)};
  return v;
}

namespace {
// Largest padded stage: two of them stay within an SM's shared memory; larger
// fields keep their rows unpadded.
constexpr int MAX_PADDED_STAGE = 13000;
constexpr long long MAX_SMEM_DOUBLES = 227 * 1024 / 8;
int row_pitch(int n2, bool padded) { return padded ? n2 | 1 : n2; }

struct Line {
  int x, y;  // first input and output element
};

// What a pass's table holds: its outputs, then its mirrored pairs.
struct PassLists {
  std::vector<KdOut> outs;
  std::vector<int> before, after;
};

// Outputs and mirrored pairs of one pass over a block of dims d with row (phi)
// pitches px (input) and py (output).  place(matrix, folded) says where a
// matrix lies among the ones the kernel reads.
template <class Place>
void list_pass(Context& ctx, const LinePassSpec& s, const int d[3], int px, int py, bool fold, Place place,
               PassLists& out) {
  const int xs = s.dim == 0 ? d[1] * px : s.dim == 1 ? px : 1, ys = s.dim == 0 ? d[1] * py : s.dim == 1 ? py : 1;
  // lines grouped by matrix
  std::vector<int> offs;
  std::vector<std::vector<Line>> lines;
  std::vector<KdOut> zeros;
  const int na = s.dim == 0 ? d[1] : d[0], nb = s.dim == 2 ? d[1] : d[2];
  for (int a = 0; a < na; a++)
    for (int b = 0; b < nb; b++) {
      int off;
      Line l;
      if (s.dim == 0) {
        off = s.offsets[static_cast<size_t>(a) * s.mat_ld + b];
        l = {a * px + b, a * py + b};
      } else if (s.dim == 1) {
        off = s.offsets[b];
        l = {a * d[1] * px + b, a * s.n_out * py + b};
      } else {
        off = s.offsets[0];
        l = {(a * d[1] + b) * px, (a * d[1] + b) * py};
      }
      if (s.dim != 2 && !s.dead.empty() && s.dead[b]) off = -1;
      if (off < 0) {
        for (int r = 0; r < s.n_out; r++) zeros.push_back({0, 0, l.y + r * ys, 0});
        continue;
      }
      size_t g = 0;
      while (g < offs.size() && offs[g] != off) g++;
      if (g == offs.size()) {
        offs.push_back(off);
        lines.emplace_back();
      }
      lines[g].push_back(l);
    }
  for (size_t g = 0; g < offs.size(); g++) {
    const Mat1d& m = ctx.bank().at_offset(offs[g]);
    const bool folded = fold && !m.folded.empty();
    const std::vector<double>& v = folded ? m.folded : m.m;
    const int at = place(m, folded);
    for (int r = 0; r < s.n_out; r++) {
      // the row's nonzeros: first to last, every second one when the others
      // are zeros (parity)
      const double* row = &v[static_cast<size_t>(r) * s.n_in];
      int first = -1, last = -1;
      for (int c = 0; c < s.n_in; c++)
        if (row[c] != 0.0) {
          if (first < 0) first = c;
          last = c;
        }
      if (first < 0) {
        for (const Line& l : lines[g]) zeros.push_back({0, 0, l.y + r * ys, 0});
        continue;
      }
      bool parity = true;
      for (int c = first + 1; c <= last; c += 2) parity = parity && row[c] == 0.0;
      const int step = parity ? 2 : 1;
      const unsigned steps = static_cast<unsigned>((last - first) / step + 1) | static_cast<unsigned>(step) << 12 |
                             static_cast<unsigned>(step * xs) << 14;
      for (const Line& l : lines[g])
        out.outs.push_back({l.x + first * xs, at + r * s.n_in + first, l.y + r * ys, steps});
    }
    if (folded) {
      const bool before = m.op == OP_COEF;
      const int n = before ? s.n_in : s.n_out, st = before ? xs : ys, j0 = m.periodic ? 1 : 0, mirror = n - 1 + j0;
      for (int j = j0; j < mirror - j; j++)
        for (const Line& l : lines[g]) {
          const unsigned base = static_cast<unsigned>(before ? l.x : l.y);
          (before ? out.before : out.after)
              .push_back(static_cast<int>((base + j * st) | (base + (mirror - j) * st) << 16));
        }
    }
  }
  // longest sums first: the outputs of a warp have the same count
  std::stable_sort(out.outs.begin(), out.outs.end(),
                   [](const KdOut& a, const KdOut& b) { return (a.steps & 4095u) > (b.steps & 4095u); });
  out.outs.insert(out.outs.end(), zeros.begin(), zeros.end());
}

// The passes of a plan over a field of dims_in, their lists and the matrices to
// stage (none when they do not fit).
void compile_passes(Context& ctx, const std::vector<LinePassSpec>& specs, const int dims_in[3], bool fold,
                    LinePlan& plan, PassLists lists[3], std::vector<double>& mats) {
  if (specs.empty() || specs.size() > 3) throw KdError(KD_ERR_ARG, "one to three passes per item");
  plan.npass = static_cast<int>(specs.size());
  for (int i = 0; i < 3; i++) plan.dims_in[i] = dims_in[i];
  auto stage_of = [&](bool padded) {
    int d[3] = {dims_in[0], dims_in[1], dims_in[2]};
    long long m = static_cast<long long>(d[0]) * d[1] * row_pitch(d[2], padded);
    for (const LinePassSpec& s : specs) {
      d[s.dim] = s.n_out;
      m = std::max(m, static_cast<long long>(d[0]) * d[1] * row_pitch(d[2], padded));
    }
    return m;
  };
  const bool padded = stage_of(true) <= MAX_PADDED_STAGE;
  // an even number: the matrices behind the two stages are 16-byte aligned
  const long long stage_doubles = (stage_of(padded) + 1) & ~1LL;
  if (2 * stage_doubles > MAX_SMEM_DOUBLES)
    throw KdError(KD_ERR_CUDA, "line_passes kernel: a field of this size does not fit in an SM's shared memory");
  plan.stage = static_cast<int>(stage_doubles);
  plan.pitch = row_pitch(dims_in[2], padded);
  // the matrices beside the stages when they fit; otherwise the kernel reads
  // the (unfolded) ones of the pool
  std::map<std::pair<size_t, bool>, int> at;
  long long room = MAX_SMEM_DOUBLES - 2 * stage_doubles;
  std::set<int> seen;
  for (const LinePassSpec& s : specs)
    for (int off : s.offsets)
      if (off >= 0 && seen.insert(off).second) room -= (static_cast<long long>(s.n_in) * s.n_out + 1) & ~1LL;
  const bool stage = room >= 0;
  auto place = [&](const Mat1d& m, bool folded) -> int {
    if (!stage) return static_cast<int>(m.pool_offset);
    auto key = std::make_pair(m.pool_offset, folded);
    auto it = at.find(key);
    if (it != at.end()) return it->second;
    const int here = static_cast<int>(mats.size());
    const std::vector<double>& v = folded ? m.folded : m.m;
    mats.insert(mats.end(), v.begin(), v.end());
    if (mats.size() & 1) mats.push_back(0.0);
    at[key] = here;
    return here;
  };
  int d[3] = {dims_in[0], dims_in[1], dims_in[2]}, px = plan.pitch;
  for (int q = 0; q < plan.npass; q++) {
    const LinePassSpec& s = specs[q];
    const int n2 = s.dim == 2 ? s.n_out : d[2];
    // the last pass writes the field as it lies in memory
    const int py = q == plan.npass - 1 ? n2 : row_pitch(n2, padded);
    list_pass(ctx, s, d, px, py, fold && stage, place, lists[q]);
    KdPass& p = plan.pass[q];
    p.dim = s.dim;
    p.n_in = s.n_in;
    p.n_out = s.n_out;
    p.nout = static_cast<int>(lists[q].outs.size());
    p.nbefore = static_cast<int>(lists[q].before.size());
    p.nafter = static_cast<int>(lists[q].after.size());
    d[s.dim] = s.n_out;
    px = py;
  }
  plan.nmats = static_cast<int>(mats.size());
}

std::vector<int> pass_table(const PassLists& l) {
  std::vector<int> t(l.outs.size() * 4);
  if (!t.empty()) std::memcpy(t.data(), l.outs.data(), t.size() * sizeof(int));
  t.insert(t.end(), l.before.begin(), l.before.end());
  t.insert(t.end(), l.after.begin(), l.after.end());
  return t;
}

void set_pass_table(KdPass& p, const int* table) {
  p.out = reinterpret_cast<const KdOut*>(table);
  p.pairs = table + 4 * static_cast<size_t>(p.nout);
}

void compile_plan(Context& ctx, const std::vector<LinePassSpec>& specs, const int dims_in[3], bool fold,
                  LinePlan& plan) {
  PassLists lists[3];
  std::vector<double> mats;
  compile_passes(ctx, specs, dims_in, fold, plan, lists, mats);
  for (int q = 0; q < plan.npass; q++) {
    set_pass_table(plan.pass[q], ctx.table(pass_table(lists[q])));
    plan.pass[q].mat = ctx.table(specs[q].offsets);
    plan.pass[q].mat_ld = specs[q].mat_ld;
  }
  plan.mats = mats.empty() ? nullptr : ctx.dtable(mats);
}

// What a plan depends on: the operator, the dims and every line's basis.
std::vector<int> plan_key(int op, int dim, const Base& b, const int n_in[3], const int n_out[3]) {
  std::vector<int> k;
  k.reserve(10 + b.t.size() + b.r.size());
  k.insert(k.end(), {op, dim, n_in[0], n_in[1], n_in[2], n_out[0], n_out[1], n_out[2], b.p, b.n2c});
  k.insert(k.end(), b.t.begin(), b.t.end());
  k.insert(k.end(), b.r.begin(), b.r.end());
  return k;
}

}  // namespace

LinePlan plain_plan(const std::vector<LinePassSpec>& specs, const int dims_in[3]) {
  LinePlan plan;
  plan.npass = static_cast<int>(specs.size());
  int d[3] = {dims_in[0], dims_in[1], dims_in[2]};
  long long m = static_cast<long long>(d[0]) * d[1] * d[2];
  for (int q = 0; q < plan.npass; q++) {
    const LinePassSpec& s = specs[q];
    KdPass& p = plan.pass[q];
    p.dim = s.dim;
    p.n_in = s.n_in;
    p.n_out = s.n_out;
    p.mat_ld = s.mat_ld;
    d[s.dim] = s.n_out;
    m = std::max(m, static_cast<long long>(d[0]) * d[1] * d[2]);
  }
  m = (m + 1) & ~1LL;
  if (2 * m > MAX_SMEM_DOUBLES)
    throw KdError(KD_ERR_CUDA, "line_passes kernel: a field of this size does not fit in an SM's shared memory");
  plan.stage = static_cast<int>(m);
  plan.pitch = dims_in[2];
  for (int i = 0; i < 3; i++) plan.dims_in[i] = dims_in[i];
  return plan;
}

const LinePlan& coef_plan(Context& ctx, const Base& base, const int np[3], const int nc[3], bool inverse,
                          long long fields) {
  const bool fold = fields > FOLD_MIN_FIELDS;
  if (!base.def)
    throw KdError(KD_ERR_STATE, inverse ? "Base not defined in Val_domain::coef_i" : "Base not defined in Val_domain::coef");
  std::vector<int> key = plan_key(inverse ? OP_COEF_I : OP_COEF, fold ? -2 : -1, base, np, nc);
  if (const LinePlan* p = ctx.find_plan(key)) return *p;
  LinePlan plan;
  compile_plan(ctx, inverse ? coef_i_specs(ctx, base, np, nc) : coef_specs(ctx, base, np, nc), inverse ? nc : np, fold,
               plan);
  return ctx.add_plan(std::move(key), std::move(plan));
}

const LinePlan& ope_1d_plan(Context& ctx, int op, int dim, const Base& base, const int d[3], Base& base_out) {
  if (!base.def) throw KdError(KD_ERR_STATE, "basis not defined in ope_1d");
  std::vector<int> key = plan_key(op, dim, base, d, d);
  const LinePlan* p = ctx.find_plan(key);
  if (!p) {
    LinePlan plan;
    Base out = base;
    compile_plan(ctx, {ope_1d_spec(ctx, op, dim, base, d, out)}, d, false, plan);
    if (dim == 0) plan.out_base = out.r;
    else if (dim == 1) plan.out_base = out.t;
    else plan.out_base = {out.p};
    p = &ctx.add_plan(std::move(key), std::move(plan));
  }
  if (dim == 0) base_out.r = p->out_base;
  else if (dim == 1) base_out.t = p->out_base;
  else base_out.p = p->out_base[0];
  return *p;
}

KdItem make_item(const LinePlan& plan, const double* in, double* out, const int dims_in[3], long long in_stride,
                 long long out_stride, double scale) {
  KdItem it{};
  it.in = in;
  it.out = out;
  it.in_stride = in_stride;
  it.out_stride = out_stride;
  it.n0 = dims_in[0];
  it.n1 = dims_in[1];
  it.n2 = dims_in[2];
  it.npass = plan.npass;
  it.stage = plan.stage;
  it.pitch = plan.pitch;
  it.nmats = plan.nmats;
  it.mats = plan.mats;
  it.scale = scale;
  for (int q = 0; q < plan.npass; q++) it.pass[q] = plan.pass[q];
  return it;
}

}  // namespace kd
