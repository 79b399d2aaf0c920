// Projector of the directional CTMRG move (real and complex enlarged corners).
//
// The reference forms M = R1*R2 (N x N, N = chi*D^2) and takes its full LAPACK
// SVD (ctmrg.jl:254-265, wrapper.jl:25-55).  Here M is never formed: a
// randomized range finder with power iterations works on R1 (R2 X) and
// R2^T (R1^T X) (all GEMMs), the sketches are orthonormalised by shifted
// CholeskyQR in FP64, and the projected k x k matrix is diagonalised by a
// one-sided Jacobi SVD in FP64 (k = n+1 plus oversampling).  Accuracy is
// checked a posteriori: the residual ||M v_i - s_i u_i|| of every kept
// triplet (the part of M v_i outside the sketch) must be below
// resid_tol * s_1, otherwise one more power iteration runs, warm-started from
// the current vectors.  The resolved right vectors of the last call of the
// same direction seed the next sketch, which near the CTMRG fixed point makes
// one pass sufficient.  Sorting, the relative cutoff 1e-12 and the
// degenerate-pair rule follow cutoff_matrix exactly.
#include "linalg.cuh"
#include "projector.cuh"

#include <algorithm>
#include <cmath>

namespace ipeps {

namespace {

// TF32 hi/lo planes of an enlarged-corner matrix Rt (r0 x c0, column-major)
// for the mixed form, split once per projector call and shared by all its
// products: `row` holds Rt itself as the A operand (rows r0, K = c0), `col`
// holds Rt^T (rows c0, K = r0), which is also Rt as a B operand.
const Planes& planes_row(Ctx& c, const Tensor& Rt, PlaneCache* pc) {
  if (pc->row.empty()) pc->row = split_kmajor(c, Rt.f64(), Rt.dims[0], false, Rt.dims[0], Rt.dims[1]);
  return pc->row;
}
const Planes& planes_col(Ctx& c, const Tensor& Rt, PlaneCache* pc) {
  if (pc->col.empty()) pc->col = split_kmajor(c, Rt.f64(), Rt.dims[0], true, Rt.dims[1], Rt.dims[0]);
  return pc->col;
}

bool use_planes(const Ctx& c, const MatRef& R, const PlaneCache* pc, int64_t cols) {
  return pc && c.precision == kPrecMixed && R.t.dt == DType::F64 && tf32x3_pays(R.rows(), cols, R.cols(), true) &&
         tf32x3_pays(R.cols(), cols, R.rows(), true);
}

}  // namespace

Tensor apply(Ctx& c, const MatRef& R, char op, const Tensor& X, PlaneCache* pc) {
  if (use_planes(c, R, pc, X.nd > 1 ? X.dims[1] : 1)) {
    const bool t = (op == 'T') != R.trans;
    const int64_t m = (op == 'N') ? R.rows() : R.cols();
    const int64_t kk = (op == 'N') ? R.cols() : R.rows();
    IPEPS_CHECK(X.dims[0] == kk, "apply: shape mismatch");
    const int64_t n = X.nd > 1 ? X.dims[1] : 1;
    Tensor Y = c.alloc(DType::F64, {m, n});
    const Planes& PA = t ? planes_col(c, R.t, pc) : planes_row(c, R.t, pc);
    const Planes PB = split_kmajor(c, X.f64(), X.dims[0], true, n, kk);
    gemm_tf32x3_planes(c, PA, PB, m, n, kk, 1.0, 0.0, Y.f64(), m);
    return Y;
  }
  return apply(c, R, op, X);
}

Tensor apply_left_T(Ctx& c, const Tensor& X, const MatRef& R, char op, PlaneCache* pc) {
  if (use_planes(c, R, pc, X.dims[1])) {
    const bool t = (op == 'T') != R.trans;
    const int64_t kk = (op == 'N') ? R.rows() : R.cols();
    const int64_t n = (op == 'N') ? R.cols() : R.rows();
    IPEPS_CHECK(X.dims[0] == kk, "apply_left_T: shape mismatch");
    const int64_t m = X.dims[1];
    Tensor Y = c.alloc(DType::F64, {m, n});
    const Planes PA = split_kmajor(c, X.f64(), X.dims[0], true, m, kk);
    const Planes& PB = t ? planes_row(c, R.t, pc) : planes_col(c, R.t, pc);
    gemm_tf32x3_planes(c, PA, PB, m, n, kk, 1.0, 0.0, Y.f64(), m);
    return Y;
  }
  return apply_left_T(c, X, R, op);
}

Tensor apply(Ctx& c, const MatRef& R, char op, const Tensor& X) {
  // op(R) * X
  bool t = (op == 'T') != R.trans;
  int64_t m = (op == 'N') ? R.rows() : R.cols();
  int64_t kk = (op == 'N') ? R.cols() : R.rows();
  IPEPS_CHECK(X.dims[0] == kk, "apply: shape mismatch");
  int64_t n = X.nd > 1 ? X.dims[1] : 1;
  Tensor Y = c.alloc(DType::F64, {m, n});
  gemm(c, DType::F64, t ? 'T' : 'N', 'N', m, n, kk, cplx(1), R.t.data(), R.t.dims[0], X.data(), X.dims[0],
       cplx(0), Y.data(), m);
  return Y;
}

Tensor apply_left_T(Ctx& c, const Tensor& X, const MatRef& R, char op) {
  // X^T * op(R): X is (kk x m) -> result (m x ncols)
  bool t = (op == 'T') != R.trans;
  int64_t kk = (op == 'N') ? R.rows() : R.cols();
  int64_t n = (op == 'N') ? R.cols() : R.rows();
  IPEPS_CHECK(X.dims[0] == kk, "apply_left_T: shape mismatch");
  int64_t m = X.dims[1];
  Tensor Y = c.alloc(DType::F64, {m, n});
  gemm(c, DType::F64, 'T', t ? 'T' : 'N', m, n, kk, cplx(1), X.data(), X.dims[0], R.t.data(), R.t.dims[0],
       cplx(0), Y.data(), m);
  return Y;
}

Tensor orth(Ctx& c, const Tensor& Y0, int passes, Tensor* Rout, std::vector<Tensor>* factors) {
  const int64_t N = Y0.dims[0];
  const int k = int(Y0.dims[1]);
  const double u = 1.1102230246251565e-16;
  // shifted CholeskyQR: the first pass adds 11 (N k + k (k+1)) u trace(G) to the diagonal
  const double sf0 = 11.0 * (double(N) * k + double(k) * (k + 1)) * u;
  if (!Rout && orth_fits(N, k)) {
    const int64_t np = cholqr_packed(k);
    Tensor R = factors ? c.alloc(DType::F64, {np * passes}) : Tensor();
    Tensor Q = c.alloc(DType::F64, {N, k});
    orth_small(c, Y0.f64(), N, k, passes, sf0, factors ? R.f64() : nullptr, Q.f64());
    for (int p = 0; factors && p < passes; ++p) {
      Tensor v = R;
      v.offset += size_t(p) * np * 8;
      v.dims[0] = np;
      factors->push_back(v);
    }
    return Q;
  }
  Tensor Y = Y0;
  Tensor G = c.alloc(DType::F64, {k, k});
  Tensor Ri = c.alloc(DType::F64, {k, k});
  Tensor Racc;
  double* d_tr = reinterpret_cast<double*>(c.scal->p) + 8;
  const bool packed = cholqr_fits(k), blocked = !packed && chol_fits(k) && trsm_fits(k);
  Tensor Rrow = packed    ? c.alloc(DType::F64, {cholqr_packed(k)})
                : blocked ? c.alloc(DType::F64, {int64_t(k) * (k + 1) / 2})
                          : Tensor();
  for (int pass = 0; pass < passes; ++pass) {
    // G = Y^T Y  (FP64 always: the Gram matrix is where precision is lost), its upper triangle: all
    // that the Cholesky kernels read
    gemm_f64_dmma(c, 'T', 'N', k, k, N, 1.0, Y.f64(), N, Y.f64(), N, 0.0, G.f64(), k, true);
    const double sf = (pass == 0) ? sf0 : 0.0;
    Tensor Yn = c.alloc(DType::F64, {N, k});
    if (packed) {
      if (factors && pass > 0) Rrow = c.alloc(DType::F64, {cholqr_packed(k)});
      chol_packed(c, G.f64(), k, k, sf, Rrow.f64(), Rout != nullptr);
      if (factors) factors->push_back(Rrow);
      trsm_packed(c, Y.f64(), N, N, k, Rrow.f64(), Yn.f64(), N);
    } else if (blocked) {
      chol_blocked(c, G.f64(), k, k, sf, Rrow.f64());
      trsm_right_upper(c, Y.f64(), N, N, k, G.f64(), k, Yn.f64(), N, Rrow.f64());
    } else {
      if (pass == 0) {
        trace(c, G.f64(), k, k, d_tr);
        chol_upper(c, G.f64(), k, k, d_tr, sf);
      } else {
        chol_upper(c, G.f64(), k, k, nullptr, 0.0);
      }
      triinv_upper(c, G.f64(), k, k, Ri.f64(), k);
      gemm(c, DType::F64, 'N', 'N', N, k, k, cplx(1), Y.data(), N, Ri.data(), k, cplx(0), Yn.data(), N, true);
    }
    Y = Yn;
    if (Rout) {
      if (pass == 0) {
        Racc = clone(c, G);
      } else {
        Tensor Rn = c.alloc(DType::F64, {k, k});
        gemm(c, DType::F64, 'N', 'N', k, k, k, cplx(1), G.data(), k, Racc.data(), k, cplx(0), Rn.data(), k, true);
        Racc = Rn;
      }
    }
  }
  if (Rout) *Rout = Racc;
  return Y;
}

namespace {

// out[j] = ||X[:, j]|| for j < nc (FP64, one warp per column)
__global__ void colnorms_kernel(const double* X, int64_t m, int nc, double* out) {
  pdl_wait();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= nc) return;
  double s = 0;
  for (int64_t i = lane; i < m; i += 32) s = fma(X[i + warp * m], X[i + warp * m], s);
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[warp] = sqrt(s);
}

// max over columns j < nc of ||X[:, j]|| (FP64, one warp per column)
__global__ void colnorm_max_kernel(const double* X, int64_t m, int nc, unsigned long long* out) {
  pdl_wait();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= nc) return;
  double s = 0;
  for (int64_t i = lane; i < m; i += 32) s = fma(X[i + warp * m], X[i + warp * m], s);
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) atomicMax(out, static_cast<unsigned long long>(__double_as_longlong(sqrt(s))));
}

// y -= f norm^2 x
__global__ void sub_shift_kernel(double f, const double* norm, const double* x, double* y, int64_t n) {
  pdl_wait();
  const double a = -f * norm[0] * norm[0];
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    y[i] = fma(a, x[i], y[i]);
}

// ------------------------------------------------------------------ backends
// The projector logic below is written once over two backends: real (FP64)
// and complex (complex128) enlarged corners.  M = R1 R2 is N1 x N2 with
// R1 (N1 x K1), R2 (K1 x N2); it is rectangular while the corner dimensions of
// an environment still differ (first iterations from init_ctm1).  words is the
// number of doubles per element, so that the gathers and column scalings can
// treat a complex column as a real column of twice the height.

struct RealOps {
  Ctx& c;
  const MatRef& R1;
  const MatRef& R2;
  PlaneCache pc1, pc2;  // mixed form: TF32 planes of R1, R2
  static constexpr DType dt = DType::F64;
  static constexpr int words = 1;
  int64_t N1() const { return R1.rows(); }
  int64_t K1() const { return R1.cols(); }
  int64_t N2() const { return R2.cols(); }
  Tensor M(const Tensor& X) { return apply(c, R1, 'N', apply(c, R2, 'N', X, &pc2), &pc1); }   // M X
  Tensor MH(const Tensor& X) { return apply(c, R2, 'T', apply(c, R1, 'T', X, &pc1), &pc2); }  // M^T X
  Tensor orth_(const Tensor& Y, int passes) { return orth(c, Y, passes, nullptr); }
  // shifted power iterations: real sketches within the packed CholeskyQR
  static bool can_shift(int k) { return cholqr_fits(k); }
  // orth(M^T Q - sigma Z R^-1) with Q R = Y = M Z, sigma = f |M z_1|^2 with *norm =
  // |M z_1|: an orthonormal basis of (M^T M - sigma) Z, without forming M^T M Z
  // (whose columns span s_k^2 .. s_1^2)
  Tensor shifted(const Tensor& Y, const Tensor& Z, double f, const double* norm, int inter) {
    std::vector<Tensor> R;
    Tensor W = MH(orth(c, Y, inter, nullptr, &R));
    Tensor T = Z;
    for (const Tensor& f : R) {
      Tensor Tn = c.alloc(dt, Z.shape());
      trsm_packed(c, T.f64(), N2(), N2(), int(Z.dims[1]), f.f64(), Tn.f64(), N2());
      T = Tn;
    }
    const int64_t n = W.numel();
    const unsigned grid = unsigned(std::min<int64_t>((n + 255) / 256, int64_t(c.sm_count) * 8));
    launch(c.stream, sub_shift_kernel, grid, 256, 0, f, norm, T.f64(), W.f64(), n);
    IPEPS_LAUNCH_CHECK();
    c.count(KFam::Elementwise, 0, 24.0 * n);
    return orth_(W, inter);
  }
  // X = Bh^H Q2 (k x k) for Bh = M^H Q (N2 x k)
  Tensor small(const Tensor& Bh, const Tensor& Q2, int k) {
    Tensor X = c.alloc(dt, {k, k});
    gemm(c, dt, 'T', 'N', k, k, N2(), cplx(1), Bh.data(), N2(), Q2.data(), N2(), cplx(0), X.data(), k, true);
    return X;
  }
  void jacobi(Tensor& X, Tensor& J, Tensor& S, int k, const SvdParams& sp, int* d_sweeps) {
    const double tol = (c.precision == kPrecMixed) ? std::max(sp.jacobi_tol, sp.jacobi_tol_mixed) : sp.jacobi_tol;
    jacobi_svd_auto(c, X.f64(), k, k, k, J.f64(), k, S.f64(), sp.jacobi_max_sweeps, tol, d_sweeps);
  }
  // sketch width: 128 columns when that still oversamples by want/2, else at most 160: every
  // column lengthens the serial steps (Cholesky, Jacobi) and shortens the iterations.
  // Gradient at D = 4, chi = 64: 128 columns 112.7 ms, the 130 asked for 121.2; at D = 5,
  // chi = 100: 151 columns 497 ms, 160 482, 192 479
  int width(int want, int kw, const SvdParams& sp) const {
    if (kw > 128 && want + std::max(sp.min_oversample, want / 2) <= 128) return 128;
    if (kw > 160 && want + sp.min_oversample <= 160) return 160;
    return kw;
  }
  Tensor P1(const Tensor& V) { return apply(c, R2, 'N', V, &pc2); }          // R2 V      (K1 x n)
  Tensor P2(const Tensor& U) { return apply_left_T(c, U, R1, 'N', &pc1); }   // U^T R1    (n x K1)
};

Tensor cmm(Ctx& c, char oa, char ob, int64_t m, int64_t n, int64_t k, const Tensor& A, int64_t lda, const Tensor& B,
           int64_t ldb) {
  Tensor Y = c.alloc(DType::C128, {m, n});
  gemm(c, DType::C128, oa, ob, m, n, k, cplx(1), A.data(), lda, B.data(), ldb, cplx(0), Y.data(), m, true);
  return Y;
}

Tensor orth_c(Ctx& c, const Tensor& Y0, int passes) {
  const int64_t N = Y0.dims[0];
  const int k = int(Y0.dims[1]);
  const double u = 1.1102230246251565e-16;
  const double sf0 = 11.0 * (double(N) * k + double(k) * (k + 1)) * u;
  if (orth_fits_c(N, k)) {
    Tensor Q = c.alloc(DType::C128, {N, k});
    orth_small_c(c, Y0.data(), N, k, passes, sf0, Q.data());
    return Q;
  }
  Tensor Y = Y0;
  Tensor G = c.alloc(DType::C128, {k, k});
  const bool packed = cholqr_fits(2 * k);
  Tensor Rpk = packed ? c.alloc(DType::F64, {cholqr_packed(2 * k)}) : Tensor();
  for (int pass = 0; pass < passes; ++pass) {
    gemm(c, DType::C128, 'C', 'N', k, k, N, cplx(1), Y.data(), N, Y.data(), N, cplx(0), G.data(), k, true);
    const double sf = (pass == 0) ? sf0 : 0.0;
    Tensor Yn = c.alloc(DType::C128, {N, k});
    if (packed) {
      chol_packed_c(c, G.data(), k, k, sf, Rpk.f64());
      trsm_packed_c(c, Y.data(), N, N, k, Rpk.f64(), Yn.data(), N);
    } else {
      chol_c(c, G.data(), k, k, sf);
      trsm_c(c, Y.data(), N, N, k, G.data(), k, Yn.data(), N);
    }
    Y = Yn;
  }
  return Y;
}

struct ComplexOps {
  Ctx& c;
  Tensor R1, R2;  // materialised (untransposed) complex128
  static constexpr DType dt = DType::C128;
  static constexpr int words = 2;
  ComplexOps(Ctx& cc, const MatRef& a, const MatRef& b)
      : c(cc),
        R1(to_complex(cc, a.trans ? permute(cc, a.t, {1, 0}) : a.t)),
        R2(to_complex(cc, b.trans ? permute(cc, b.t, {1, 0}) : b.t)) {}
  int64_t N1() const { return R1.dims[0]; }
  int64_t K1() const { return R1.dims[1]; }
  int64_t N2() const { return R2.dims[1]; }
  Tensor M(const Tensor& X) {
    const int64_t n = X.dims[1];
    return cmm(c, 'N', 'N', N1(), n, K1(), R1, N1(), cmm(c, 'N', 'N', K1(), n, N2(), R2, K1(), X, N2()), K1());
  }
  Tensor MH(const Tensor& X) {
    const int64_t n = X.dims[1];
    return cmm(c, 'C', 'N', N2(), n, K1(), R2, K1(), cmm(c, 'C', 'N', K1(), n, N1(), R1, N1(), X, N1()), K1());
  }
  Tensor orth_(const Tensor& Y, int passes) { return orth_c(c, Y, passes); }
  static bool can_shift(int) { return false; }
  Tensor shifted(const Tensor& Y, const Tensor&, double, const double*, int inter) { return orth_(MH(orth_(Y, inter)), inter); }
  Tensor small(const Tensor& Bh, const Tensor& Q2, int k) { return cmm(c, 'C', 'N', k, k, N2(), Bh, N2(), Q2, N2()); }
  void jacobi(Tensor& X, Tensor& J, Tensor& S, int k, const SvdParams& sp, int* d_sweeps) {
    jacobi_c_svd(c, X.data(), k, k, k, J.data(), k, S.f64(), sp.jacobi_max_sweeps, sp.jacobi_tol, d_sweeps);
  }
  int width(int want, int kw, const SvdParams& sp) const {
    while (kw > want + sp.min_oversample && !complex_small_fits(kw, kw)) --kw;
    IPEPS_CHECK(complex_small_fits(kw, kw), "get_projector: complex sketch too wide for the shared-memory kernels");
    return kw;
  }
  Tensor P1(const Tensor& V) { return cmm(c, 'N', 'N', K1(), V.dims[1], N2(), R2, K1(), V, N2()); }
  Tensor P2(const Tensor& U) { return cmm(c, 'C', 'N', U.dims[1], K1(), N1(), U, N1(), R1, N1()); }
};

// One sketch pass: range finder with q power iterations from Omega, Rayleigh-Ritz, Jacobi.
struct Sketch {
  Tensor Q, Q2, X, J, Ss;  // Q: N1 x k, Q2: N2 x k; X = W (k x k); J (k x k); Ss sorted S (k)
  Tensor perm;             // int[k] stored in a double buffer
  int sweeps = 0;
};

// inter: CholeskyQR passes of the intermediate sketches.  One shifted pass
// suppresses directions below ~sqrt(shift) ~ 1e-6 s_1, which over the power
// iterations then decay away; three passes (sCholQR3) keep them, as needed
// when the truncation reaches down to the 1e-12 relative cutoff.
// b > 0: the power iterations are shifted, Z <- orth((M^T M - sigma_j) Z) with the
// sigma_j at the Chebyshev nodes of [0, b s_1^2]: the product over the iterations is
// the Chebyshev polynomial of degree q on that interval.  With b = (s_k / s_1)^2 the
// directions outside the sketch shrink against s_n by exp(-q acosh(2 s_n^2 / s_k^2 - 1))
// instead of (s_k / s_n)^2q: at D=5 chi=100 (s_n / s_k = 1.6) by ~5 per iteration
// instead of ~1.8.  s_1 is |M z_1| of the first column (the leading seed), a lower
// bound: the scale of M changes from call to call.
template <class Ops>
Sketch sketch_pass(Ctx& c, Ops& o, const Tensor& Om, int q, const SvdParams& sp, int inter, double b) {
  const int k = int(Om.dims[1]);
  Sketch s;
  Tensor Z = Om, Y = o.M(Om);
  double* norm = reinterpret_cast<double*>(c.scal->p) + 56;
  if (b > 0 && q > 0) {
    launch(c.stream, colnorms_kernel, 1, 32, 0, Y.f64(), o.N1(), 1, norm);
    IPEPS_LAUNCH_CHECK();
  }
  for (int it = 0; it < q; ++it) {
    if (b > 0)
      Z = o.shifted(Y, Z, 0.5 * b * (1.0 + std::cos((2 * it + 1) * 3.14159265358979323846 / (2.0 * q))), norm, inter);
    else
      Z = o.orth_(o.MH(o.orth_(Y, inter)), inter);
    Y = o.M(Z);
  }
  s.Q = o.orth_(Y, 3);
  // B^H = M^H Q (N2 x k), Q2 = orth(B^H).  The Rayleigh-Ritz matrix is formed
  // explicitly, X = B = (M^H Q)^H Q2, rather than taken as R^H from B^H = Q2 R:
  // when M is numerically rank deficient the shifted first CholeskyQR pass
  // leaves sqrt(shift)-sized entries in R for the null directions, which the
  // later passes cannot normalise, and R^H would show them as spurious
  // singular values far above the 1e-12 cutoff.
  Tensor Bh = o.MH(s.Q);
  s.Q2 = o.orth_(Bh, 3);
  s.X = o.small(Bh, s.Q2, k);
  // one-sided Jacobi: X J = W = Ux S  =>  U = Q Ux, V = Q2 J
  s.J = c.alloc(Ops::dt, {k, k});
  Tensor S = c.alloc(DType::F64, {k});
  int* d_sweeps = reinterpret_cast<int*>(static_cast<char*>(c.scal->p) + 3900);
  o.jacobi(s.X, s.J, S, k, sp, d_sweeps);
  s.Ss = c.alloc(DType::F64, {k});
  s.perm = c.alloc(DType::F64, {(k + 1) / 2});
  sort_desc(c, S.f64(), k, s.Ss.f64(), static_cast<int*>(s.perm.data()));
  IPEPS_CUDA(cudaMemcpyAsync(&s.sweeps, d_sweeps, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  return s;
}

void copy_cols(Ctx& c, Tensor& dst, const Tensor& src, int64_t rows, int ncols, int words) {
  IPEPS_CUDA(cudaMemcpyAsync(dst.data(), src.data(), size_t(rows) * ncols * 8 * words, cudaMemcpyDeviceToDevice,
                             c.stream));
}

// Whether one shifted CholeskyQR pass keeps the directions of the first n triplets of
// a sketch with singular values s: its shift, 11 (N k + k (k + 1)) u times the trace
// of the Gram matrix (<= the sum of s_i^2 for a product of M with an orthonormal
// basis), damps a direction by s_i / sqrt(s_i^2 + shift) per pass.
bool one_pass_keeps(const std::vector<double>& s, int64_t N, int k, int n) {
  double tr = 0;
  for (double v : s) tr += v * v;
  const double shift = 11.0 * (double(N) * k + double(k) * (k + 1)) * 1.1102230246251565e-16 * tr;
  return s[size_t(n - 1)] * s[size_t(n - 1)] >= 10.0 * shift;
}

template <class Ops>
ProjResult projector_impl(Ctx& c, Ops& o, int chi, const SvdParams& sp, ProjCache* cache, bool keep_factors) {
  constexpr DType dt = Ops::dt;
  constexpr int w = Ops::words;
  const int64_t N1 = o.N1(), K1 = o.K1(), N2 = o.N2(), Nmin = std::min(N1, N2);
  const int new_chi = int(std::min<int64_t>(chi, K1));
  const int want = int(std::min<int64_t>(Nmin, new_chi + 1));
  const int over = std::max(sp.min_oversample, want * sp.oversample_num / std::max(sp.oversample_den, 1));
  const int k = o.width(want, int(std::min<int64_t>(Nmin, int64_t(want) + over)), sp);

  // Sketch Omega (N2 x k): resolved right vectors of an earlier call first,
  // then Gaussian columns.  No seeds when k = min(N1, N2): a Gaussian Omega
  // then spans the domain and one pass is exact, which seed vectors (possibly
  // confined to a few symmetry sectors of M) would not guarantee.  After a
  // cutoff-limited truncation at least min_oversample columns stay Gaussian,
  // so that directions absent from the seeds can enter; in the chi-limited
  // regime the seeds may fill the sketch.
  Tensor Om = c.alloc(dt, {N2, k});
  randn(c, Om);
  bool warm = false;
  const bool room = !cache || cache->cutoff_limited;
  const int seed_cap = room ? std::max(0, k - std::max(sp.min_oversample, 1)) : k;
  if (k < Nmin && seed_cap > 0 && sp.warm_start && cache && !cache->seed(sp.seed_older).empty() &&
      cache->seed(sp.seed_older).dims[0] == N2 && cache->seed(sp.seed_older).dt == dt) {
    const Tensor& Vs = cache->seed(sp.seed_older);
    copy_cols(c, Om, Vs, N2, int(std::min<int64_t>(Vs.dims[1], seed_cap)), w);
    warm = true;
  }
  int q = (k == Nmin) ? 0 : (warm ? sp.power_iters_warm : sp.power_iters);
  int inter = sp.inter_passes;
  if (!warm || !cache || cache->cutoff_limited) inter = std::max(inter, 3);
  // power iterations this direction's recent calls needed beyond q (each
  // extra pass below costs a Rayleigh-Ritz step, two sCholQR3 and a Jacobi SVD
  // on top of its power iteration; doing the iterations up front is cheaper).
  // Only with sCholQR3 intermediates: a single shifted pass drops directions
  // below ~sqrt(shift) s_1 at every iteration, so more iterations would lose them.
  // residual tolerance of this call (the mixed form's 3xTF32 iterations settle
  // for the FP32-level floor of their products)
  const double rtol = (c.precision == kPrecMixed && dt == DType::F64) ? std::max(sp.resid_tol, sp.resid_tol_mixed)
                                                                       : sp.resid_tol;
  // seeds resolved to a looser tolerance than this call's (the first FP64
  // iterations after the mixed form's 3xTF32 ones, the adjoint's checkpoint
  // iterations at 1e-12): one power iteration per factor ~7 of the residual,
  // done up front with sCholQR3 intermediates, instead of as extra passes
  if (warm && q > 0 && cache->seed_tol(sp.seed_older) > 10.0 * rtol) {
    inter = std::max(inter, 3);
    q += std::min(6, int(std::ceil(std::log(cache->seed_tol(sp.seed_older) / rtol) / std::log(7.0))));
  }
  // Shifted iterations (see sketch_pass) where the seeds' spectrum is known and not
  // cutoff-limited: as many as this direction's last call needed, corrected for
  // another tolerance, at the rate of the Chebyshev polynomial (a quarter off: s_k of
  // the sketch is a lower bound of the first value outside it).  Done up front an
  // iteration costs two products with M and two CholeskyQR passes; as an extra pass
  // it costs a Rayleigh-Ritz step (two sCholQR3, a Jacobi SVD) besides.
  // The target is a thirtieth of the tolerance, as an extra pass overshoots it (a
  // residual just below the tolerance leaves the errors of a whole trajectory larger).
  const auto rate_of = [](double sn2, double b) { return 0.75 * std::acosh(2.0 * sn2 / b - 1.0); };
  constexpr double kAim = 1.0 / 30.0;
  constexpr int kMaxShifted = 8;
  double b = 0;
  const bool shift = warm && q > 0 && Ops::can_shift(k) && !cache->cutoff_limited &&
                     cache->seed_spec(sp.seed_older).k == k;
  if (shift) {
    const auto& spec = cache->seed_spec(sp.seed_older);
    b = std::min(spec.sk2, 0.9 * spec.sn2);
    double need = cache->need;
    if (cache->rtol > 0) need += std::log(cache->rtol / rtol) / rate_of(spec.sn2, b);
    q = std::max(sp.power_iters_warm, std::min(kMaxShifted, int(std::ceil(need))));
    inter = std::max(sp.inter_passes, spec.one_pass ? 1 : 3);
  }
  const bool adapt = q > 0 && cache && inter >= 3 && !shift;
  if (adapt) q += cache->qbonus;
  int iters = q;  // power iterations behind the accepted sketch
  int extra = 0;
  double res_final = 1.0;

  ProjResult r;
  r.k = k;
  Sketch sk;
  std::vector<double> all(k);
  int n = 0, n_above_last = 0;
  Tensor Ux, Vk;
  int* d_perm = nullptr;
  double* d_res = reinterpret_cast<double*>(c.scal->p) + 48;
  double prev_res = 1e300;
  for (int attempt = 0;; ++attempt) {
    sk = sketch_pass(c, o, Om, q, sp, inter, b);
    d_perm = static_cast<int*>(sk.perm.data());
    IPEPS_CUDA(cudaMemcpyAsync(all.data(), sk.Ss.data(), size_t(k) * 8, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    c.jacobi_sweeps += uint64_t(sk.sweeps);
    // cutoff_matrix (wrapper.jl:37-55)
    const double smax = all[0];
    int n_above = 0;
    for (int i = 0; i < k; ++i)
      if (smax > 0 && all[i] / smax > 1e-12) n_above++;
    n_above_last = n_above;
    if (n_above < new_chi && inter < 3 && q > 0) {
      // cutoff-limited after cheap intermediates: small directions may be missing; redo cold with sCholQR3
      inter = 3;
      Om = c.alloc(dt, {N2, k});
      randn(c, Om);
      q = sp.power_iters;
      b = 0;
      iters = q;  // the abandoned sketch says nothing about the next call
      --attempt;
      continue;
    }
    n = std::min(new_chi, n_above);
    IPEPS_CHECK(n >= 1, "get_projector: no singular value above the cutoff (zero enlarged corner?)");
    // the reference's s has length min(N1, N2) (full SVD); ours is the top-k part
    if (Nmin > n && k > n) {
      if (std::fabs(all[n] - all[n - 1]) < 1e-10) n = n + 1;
    }
    IPEPS_CHECK(n <= k, "get_projector: truncation beyond the sketch");
    // Ux[:, j] = W[:, perm[j]] / S_sorted[j] (kept + one), Vk = Q2 J[:, perm]
    const int nc = std::min(n + 1, k);
    Ux = c.alloc(dt, {k, nc});
    gather_cols(c, sk.X.f64(), w * k, w * k, d_perm, nc, sk.Ss.f64(), 2, Ux.f64(), w * k);
    Tensor Js = c.alloc(dt, {k, k});
    gather_cols(c, sk.J.f64(), w * k, w * k, d_perm, k, nullptr, 0, Js.f64(), w * k);
    Vk = c.alloc(dt, {N2, k});
    gemm(c, dt, 'N', 'N', N2, k, k, cplx(1), sk.Q2.data(), N2, Js.data(), k, cplx(0), Vk.data(), N2, true);
    if (q == 0 && k == Nmin) {  // the sketch spans a whole side of M: exact
      res_final = 0.0;
      break;
    }
    // residual of the kept triplets and the next one: ||M v_i - s_i u_i|| <= resid_tol * s_1.
    // For the adjoint (keep_factors) also the tail down to 0.8 s_n: the adjoint
    // sums those triplets exactly, and the interval of its expansion of the
    // rest of the spectrum, and with it the number of terms, is set by the
    // first triplet it does not resolve.
    int nr = nc;
    if (keep_factors)
      while (nr < k && all[nr] >= 0.8 * all[n - 1]) ++nr;
    Tensor Vc = c.alloc(dt, {N2, nr});
    copy_cols(c, Vc, Vk, N2, nr, w);
    Tensor Res = o.M(Vc);
    Tensor Us = c.alloc(dt, {k, nr});
    gather_cols(c, sk.X.f64(), w * k, w * k, d_perm, nr, nullptr, 0, Us.f64(), w * k);  // W = Ux S
    gemm(c, dt, 'N', 'N', N1, nr, k, cplx(-1), sk.Q.data(), N1, Us.data(), k, cplx(1), Res.data(), N1, true);
    IPEPS_CUDA(cudaMemsetAsync(d_res, 0, 8, c.stream));
    launch(c.stream, colnorm_max_kernel, (nr * 32 + 255) / 256, 256, 0, Res.f64(), w * N1, nr,
           reinterpret_cast<unsigned long long*>(d_res));
    IPEPS_LAUNCH_CHECK();
    double res = 0;
    IPEPS_CUDA(cudaMemcpyAsync(&res, d_res, 8, cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    // done when below tolerance, or when it stopped decreasing (the FP64 floor of
    // R1 (R2 v), ~eps ||R1|| ||R2||, can sit above resid_tol * s_1)
    res_final = smax > 0 ? res / smax : 1.0;
    if (res <= rtol * smax) break;
    if (res > 0.5 * prev_res || attempt >= sp.max_extra_passes) {
      c.resid_misses++;
      break;
    }
    prev_res = res;
    // not converged: more power iterations from the current right vectors
    Om = Vk;
    q = 1;
    if (Ops::can_shift(k) && n_above >= new_chi && all[n - 1] > 0) {
      const double sn2 = std::pow(all[n - 1] / smax, 2);
      b = std::min(std::pow(all[k - 1] / smax, 2), 0.9 * sn2);
      q = std::max(1, std::min(kMaxShifted, int(std::ceil(std::log(res_final / (kAim * rtol)) / rate_of(sn2, b))) - 1));
      if (!one_pass_keeps(all, N1, k, n)) inter = std::max(inter, 3);
    }
    iters += q + 1;
    c.projector_extra_passes++;
    ++extra;
  }
  r.sweeps = sk.sweeps;
  c.projector_calls++;
  r.n = n;
  r.s_host.assign(all.begin(), all.begin() + n);

  Tensor U = c.alloc(dt, {N1, n});
  gemm(c, dt, 'N', 'N', N1, n, k, cplx(1), sk.Q.data(), N1, Ux.data(), k, cplx(0), U.data(), N1, true);
  Tensor V = c.alloc(dt, {N2, n});
  copy_cols(c, V, Vk, N2, n, w);
  // resolved part of the sketch: s_a > 1e-13 s_1 (W/s is accurate there)
  int rr = 0;
  while (rr < k && all[rr] > 1e-13 * all[0]) ++rr;
  rr = std::max(rr, n);
  if (cache) {
    // seed for the next call of this direction: the resolved right vectors only
    // (near-null directions of this M say nothing about the next one)
    Tensor Vc = c.alloc(dt, {N2, rr});
    copy_cols(c, Vc, Vk, N2, rr, w);
    cache->Vold = cache->V;
    cache->V = Vc;
    cache->tol_old = cache->tol;
    cache->tol = std::max(res_final, 1e-15);  // the residual these vectors reached
    cache->cutoff_limited = n_above_last < new_chi;
    cache->spec_old = cache->spec;
    cache->spec = {};
    if (n_above_last >= new_chi && all[n - 1] > 0) {
      cache->spec = {k, std::pow(all[n - 1] / all[0], 2), std::pow(all[k - 1] / all[0], 2),
                     one_pass_keeps(all, N1, k, n)};
      const double r = rate_of(cache->spec.sn2, std::min(cache->spec.sk2, 0.9 * cache->spec.sn2));
      cache->need = std::min(iters, kMaxShifted) + std::log(std::max(res_final, 1e-16) / (kAim * rtol)) / r;
      // without an extra pass at least one less: the mixed form's residuals stay at
      // the floor of its products whatever the iterations
      if (extra == 0) cache->need = std::min(cache->need, double(iters - 1));
      cache->rtol = rtol;
    }
    if (adapt)
      cache->qbonus = extra > 0 ? std::min(cache->qbonus + extra, sp.max_extra_passes) : std::max(cache->qbonus - 1, 0);
  }
  if (keep_factors) {
    IPEPS_CHECK(dt == DType::F64, "get_projector: the projector adjoint is real-only");
    // The adjoint sums the resolved triplets exactly and expands the rest of the
    // spectrum on their complement, which is exact only if the resolved vectors
    // span an invariant subspace: keep just the leading triplets whose residual
    // ||M v_a - s_a u_a|| is at most 1e-10 s_1 (the sketch's oversampled tail is
    // less accurate and goes to the expansion instead).
    if (rr > n) {
      Tensor Vall = c.alloc(dt, {N2, rr});
      copy_cols(c, Vall, Vk, N2, rr, w);
      Tensor Res = o.M(Vall);
      Tensor Wall = c.alloc(dt, {k, rr});
      gather_cols(c, sk.X.f64(), k, k, d_perm, rr, nullptr, 0, Wall.f64(), k);
      gemm(c, dt, 'N', 'N', N1, rr, k, cplx(-1), sk.Q.data(), N1, Wall.data(), k, cplx(1), Res.data(), N1, true);
      Tensor rn = c.alloc(DType::F64, {rr});
      launch(c.stream, colnorms_kernel, (rr * 32 + 255) / 256, 256, 0, Res.f64(), N1, rr, rn.f64());
      IPEPS_LAUNCH_CHECK();
      std::vector<double> rh(rr);
      IPEPS_CUDA(cudaMemcpyAsync(rh.data(), rn.data(), size_t(rr) * 8, cudaMemcpyDeviceToHost, c.stream));
      c.sync();
      int acc = n;
      while (acc < rr && rh[acc] <= 1e-10 * all[0]) ++acc;
      rr = acc;
    }
    r.r = rr;
    r.sr_host.assign(all.begin(), all.begin() + rr);
    r.s_next = (rr < k) ? all[rr] : all[k - 1];
    Tensor Uxr = c.alloc(dt, {k, rr});
    gather_cols(c, sk.X.f64(), k, k, d_perm, rr, sk.Ss.f64(), 2, Uxr.f64(), k);
    r.Ur = c.alloc(dt, {N1, rr});
    gemm(c, dt, 'N', 'N', N1, rr, k, cplx(1), sk.Q.data(), N1, Uxr.data(), k, cplx(0), r.Ur.data(), N1, true);
    r.Vr = c.alloc(dt, {N2, rr});
    copy_cols(c, r.Vr, Vk, N2, rr, w);
    r.Sr = c.alloc(DType::F64, {rr});
    IPEPS_CUDA(cudaMemcpyAsync(r.Sr.data(), sk.Ss.data(), size_t(rr) * 8, cudaMemcpyDeviceToDevice, c.stream));
  }

  r.S = c.alloc(DType::F64, {n});
  IPEPS_CUDA(cudaMemcpyAsync(r.S.data(), sk.Ss.data(), size_t(n) * 8, cudaMemcpyDeviceToDevice, c.stream));
  // P1 = R2 V S^-1/2 ; P2 = S^-1/2 U^H R1
  scale_cols(c, V.f64(), w * N2, w * N2, n, r.S.f64(), 1);
  scale_cols(c, U.f64(), w * N1, w * N1, n, r.S.f64(), 1);
  r.P1 = o.P1(V);
  r.P2 = o.P2(U);
  return r;
}

}  // namespace

ProjResult get_projector(Ctx& c, const MatRef& R1, const MatRef& R2, int chi, const SvdParams& sp,
                         ProjCache* cache, bool keep_factors) {
  IPEPS_CHECK(R1.cols() == R2.rows(), "get_projector: inner dimensions of R1*R2 differ");
  if (R1.t.dt == DType::C128 || R2.t.dt == DType::C128) {
    ComplexOps o(c, R1, R2);
    return projector_impl(c, o, chi, sp, cache, keep_factors);
  }
  RealOps o{c, R1, R2, {}, {}};
  return projector_impl(c, o, chi, sp, cache, keep_factors);
}

}  // namespace ipeps
