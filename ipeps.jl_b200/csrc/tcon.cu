// tcon: pairwise tensor contraction with the label convention of the
// reference's ``tcon`` (src/utility/wrapper.jl:15-23, OMEinsum EinCode):
// positive labels are summed over, negative labels -1, -2, ... give the
// output order.  Planned as transpose-transpose-GEMM-transpose on
// column-major tensors:
//   * free labels of each operand are ordered as they appear in the output;
//   * the summed-label order is taken from A or from B, whichever needs fewer
//     permuted elements;
//   * an operand already laid out as [free, summed] or [summed, free] enters
//     the GEMM directly as op N / op T (no copy);
//   * the product is formed as [freeA, freeB] or, when the output lists all
//     of B's labels first, as its transpose [freeB, freeA]; only an
//     interleaved output needs a final permute.
#include "ctx.cuh"

#include <algorithm>
#include <map>

namespace ipeps {
namespace {

// position of each label in a label list
int find(const std::vector<int>& l, int x) {
  for (size_t i = 0; i < l.size(); ++i)
    if (l[i] == x) return int(i);
  return -1;
}

// Is tensor with labels `have` already ordered as concat(first, second)?
bool ordered_as(const std::vector<int>& have, const std::vector<int>& first, const std::vector<int>& second) {
  if (have.size() != first.size() + second.size()) return false;
  for (size_t i = 0; i < first.size(); ++i)
    if (have[i] != first[i]) return false;
  for (size_t i = 0; i < second.size(); ++i)
    if (have[first.size() + i] != second[i]) return false;
  return true;
}

// Unit-extent labels may be placed anywhere; drop them for ordering checks.
std::vector<int> strip_units(const std::vector<int>& labels, const std::map<int, int64_t>& ext) {
  std::vector<int> r;
  for (int l : labels)
    if (ext.at(l) != 1) r.push_back(l);
  return r;
}

int64_t permute_cost(const std::vector<int>& lx, const std::vector<int>& r, const std::vector<int>& col,
                     const std::map<int, int64_t>& ext, int64_t numel) {
  auto sx = strip_units(lx, ext), sr = strip_units(r, ext), sc = strip_units(col, ext);
  if (ordered_as(sx, sr, sc) || ordered_as(sx, sc, sr)) return 0;
  return numel;
}

// How an operand with labels lx becomes a GEMM operand whose logical matrix is [rows, cols].
Contraction::Side plan_side(const std::vector<int>& lx, const std::vector<int>& rows, const std::vector<int>& cols,
                            const std::map<int, int64_t>& ext) {
  int64_t nr = 1, nc = 1;
  for (int l : rows) nr *= ext.at(l);
  for (int l : cols) nc *= ext.at(l);
  auto sx = strip_units(lx, ext), sr = strip_units(rows, ext), scl = strip_units(cols, ext);
  Contraction::Side s;
  if (ordered_as(sx, sr, scl)) {
    s.ld = std::max<int64_t>(nr, 1);
  } else if (ordered_as(sx, scl, sr)) {
    s.op = 'T';
    s.ld = std::max<int64_t>(nc, 1);
  } else {
    for (int l : rows) s.perm.push_back(find(lx, l));
    for (int l : cols) s.perm.push_back(find(lx, l));
    s.ld = std::max<int64_t>(nr, 1);
  }
  return s;
}

// op(A) op(B) of real and complex operands; the result is complex when either is
void gemm_any(Ctx& c, char opA, const Tensor& A, int64_t lda, char opB, const Tensor& B, int64_t ldb, int64_t m,
              int64_t n, int64_t k, double beta, void* C, int64_t ldc) {
  if (A.dt == B.dt)
    gemm(c, A.dt, opA, opB, m, n, k, cplx(1), A.data(), lda, B.data(), ldb, cplx(beta), C, ldc);
  else
    gemm_c128_dmma(c, opA, A.dt, opB, B.dt, m, n, k, cplx(1), A.data(), lda, B.data(), ldb, cplx(beta), C, ldc);
}

}  // namespace

Contraction::Contraction(const Tensor& A, const std::vector<int>& la, const Tensor& B, const std::vector<int>& lb) {
  IPEPS_CHECK(int(la.size()) == A.nd, "tcon: label count != rank of A " + shape_str(A));
  IPEPS_CHECK(int(lb.size()) == B.nd, "tcon: label count != rank of B " + shape_str(B));
  a_shape_ = Shape(A);
  b_shape_ = Shape(B);
  std::map<int, int64_t> ext;
  for (int i = 0; i < A.nd; ++i) ext[la[i]] = A.dims[i];
  for (int i = 0; i < B.nd; ++i) {
    auto it = ext.find(lb[i]);
    if (it != ext.end()) {
      IPEPS_CHECK(lb[i] > 0, "tcon: output label repeated");
      IPEPS_CHECK(it->second == B.dims[i], "tcon: extent mismatch on label " + std::to_string(lb[i]) +
                                               " A" + shape_str(A) + " B" + shape_str(B));
    } else {
      ext[lb[i]] = B.dims[i];
    }
  }
  std::vector<int> fa, fb, kA, kB;
  for (int l : la) (l < 0 ? fa : kA).push_back(l);
  for (int l : lb) (l < 0 ? fb : kB).push_back(l);
  IPEPS_CHECK(kA.size() == kB.size(), "tcon: summed labels must appear in both operands");
  for (int l : kA) IPEPS_CHECK(find(kB, l) >= 0, "tcon: label " + std::to_string(l) + " only in A");
  auto by_out = [](std::vector<int>& v) { std::sort(v.begin(), v.end(), [](int x, int y) { return x > y; }); };
  by_out(fa);
  by_out(fb);
  const int nout = int(fa.size() + fb.size());
  odims_.resize(nout);
  for (int i = 0; i < nout; ++i) {
    auto it = ext.find(-(i + 1));
    IPEPS_CHECK(it != ext.end(), "tcon: output labels must be -1..-n");
    odims_[i] = it->second;
  }
  // output arrangement
  auto pos = [](int l) { return -l - 1; };
  int maxa = -1, mina = 1 << 30, maxb = -1, minb = 1 << 30;
  for (int l : fa) { maxa = std::max(maxa, pos(l)); mina = std::min(mina, pos(l)); }
  for (int l : fb) { maxb = std::max(maxb, pos(l)); minb = std::min(minb, pos(l)); }
  const bool direct = fb.empty() || fa.empty() || maxa < minb;
  swapped_ = !direct && maxb < mina;
  // summed-label order: from A or from B
  int64_t costA = permute_cost(la, fa, kA, ext, A.numel()) + permute_cost(lb, kA, fb, ext, B.numel());
  int64_t costB = permute_cost(la, fa, kB, ext, A.numel()) + permute_cost(lb, kB, fb, ext, B.numel());
  const std::vector<int>& kk = (costB < costA) ? kB : kA;
  for (int l : fa) m_ *= ext[l];
  for (int l : fb) n_ *= ext[l];
  for (int l : kk) k_ *= ext[l];
  if (!swapped_) {
    a_ = plan_side(la, fa, kk, ext);
    b_ = plan_side(lb, kk, fb, ext);
  } else {  // C^T = B^T A^T : rows = fb, cols = fa
    a_ = plan_side(la, kk, fa, ext);
    b_ = plan_side(lb, fb, kk, ext);
  }
  if (!(direct || swapped_)) {
    // the product is [fa..., fb...] -> output order
    std::vector<int> cur(fa);
    cur.insert(cur.end(), fb.begin(), fb.end());
    for (int l : cur) raw_dims_.push_back(ext[l]);
    final_.resize(nout);
    for (int i = 0; i < nout; ++i) final_[i] = find(cur, -(i + 1));
  }
}

Tensor Contraction::prepared(Ctx& c, Side& s, const Tensor& X) {
  if (s.perm.empty()) return X;
  for (const auto& q : s.done)
    if (q.first.buf == X.buf && q.first.offset == X.offset && q.first.dt == X.dt) return q.second;
  Tensor p = permute(c, X, s.perm);
  s.done.emplace_back(X, p);
  return p;
}

void Contraction::add(Ctx& c, Tensor& raw, const Tensor& A, const Tensor& B) {
  // The plan's extents are those of the operands it was made for.  Another component of a
  // nested tensor can differ: set_CT replaces component 0 of an environment alone.
  IPEPS_CHECK(a_shape_.of(A) && b_shape_.of(B),
              "tcon: operands " + shape_str(A) + " " + shape_str(B) + " differ from the sum's other terms");
  const DType dt = (A.dt == DType::C128 || B.dt == DType::C128) ? DType::C128 : DType::F64;
  if (!raw.empty() && raw.dt == DType::F64 && dt == DType::C128) raw = to_complex(c, raw);
  if (!raw.empty() && raw.dt == DType::C128 && dt == DType::F64) {
    Tensor t;
    add(c, t, A, B);
    axpy(c, cplx(1), t, raw);
    return;
  }
  const double beta = raw.empty() ? 0.0 : 1.0;
  if (raw.empty()) raw = c.alloc(dt, final_.empty() ? odims_ : raw_dims_);
  if (k_ == 0 || m_ * n_ == 0) {
    if (beta == 0.0) IPEPS_CUDA(cudaMemsetAsync(raw.data(), 0, raw.bytes(), c.stream));
    return;
  }
  const Tensor a = prepared(c, a_, A), b = prepared(c, b_, B);
  if (!swapped_)
    gemm_any(c, a_.op, a, a_.ld, b_.op, b, b_.ld, m_, n_, k_, beta, raw.data(), m_);
  else
    gemm_any(c, b_.op, b, b_.ld, a_.op, a, a_.ld, n_, m_, k_, beta, raw.data(), n_);
}

Tensor Contraction::finish(Ctx& c, const Tensor& raw) const {
  return final_.empty() ? raw : permute(c, raw, final_);
}

Tensor tcon(Ctx& c, const Tensor& A, const std::vector<int>& la, const Tensor& B,
            const std::vector<int>& lb) {
  Contraction p(A, la, B, lb);
  Tensor raw;
  p.add(c, raw, A, B);
  return p.finish(c, raw);
}

Tensor matmul(Ctx& c, const Tensor& A, char opA, const Tensor& B, char opB) {
  IPEPS_CHECK(A.nd == 2 && B.nd == 2, "matmul: 2-D operands expected");
  int64_t m = (opA == 'N') ? A.dims[0] : A.dims[1];
  int64_t ka = (opA == 'N') ? A.dims[1] : A.dims[0];
  int64_t kb = (opB == 'N') ? B.dims[0] : B.dims[1];
  int64_t n = (opB == 'N') ? B.dims[1] : B.dims[0];
  IPEPS_CHECK(ka == kb, "matmul: inner dimension mismatch " + shape_str(A) + " " + shape_str(B));
  DType dt = (A.dt == DType::C128 || B.dt == DType::C128) ? DType::C128 : DType::F64;
  Tensor C = c.alloc(dt, {m, n});
  gemm_any(c, opA, A, std::max<int64_t>(A.dims[0], 1), opB, B, std::max<int64_t>(B.dims[0], 1), m, n, ka, 0.0,
           C.data(), std::max<int64_t>(m, 1));
  return C;
}

// Which products of the mixed form run as 3xTF32.  Measured per product on B200
// (splits and split-K sums included): splitting both operands and the pipeline's
// start cost 20-30 us whatever the size, and the split moves 24 bytes per operand
// element, so the FP64 kernel is the faster one below ~0.9 GFLOP (1450 x 118 x
// 1450, 0.50 GFLOP: 29 us against 34; 2250 x 2250 x 90, 0.91 GFLOP: 48 against 47;
// 2500 x 160 x 2500, 2 GFLOP: 84 against 58) and, at any size, for short inner
// dimensions (250000 x 50 x 25: 62 us against 88).  planes_kept: the large operand's
// split is shared by all products of a projector (0.4 GFLOP: about the split of
// 1150 x 1150, 10 us, less).
bool tf32x3_pays(int64_t m, int64_t n, int64_t k, bool planes_kept) {
  return k >= 64 && 2.0 * double(m) * double(n) * double(k) >= (planes_kept ? 4e8 : 9e8);
}

void gemm(Ctx& c, DType dt, char opA, char opB, int64_t m, int64_t n, int64_t k,
          cuDoubleComplex alpha, const void* A, int64_t lda, const void* B, int64_t ldb,
          cuDoubleComplex beta, void* C, int64_t ldc, bool force_fp64) {
  if (dt == DType::F64 && c.precision == kPrecMixed && !force_fp64 && alpha.y == 0 && beta.y == 0 &&
      opA != 'C' && opB != 'C' && tf32x3_pays(m, n, k)) {
    gemm_tf32x3(c, opA, opB, m, n, k, alpha.x, static_cast<const double*>(A), lda,
                static_cast<const double*>(B), ldb, beta.x, static_cast<double*>(C), ldc);
    return;
  }
  gemm_f64(c, dt, opA, opB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

}  // namespace ipeps
