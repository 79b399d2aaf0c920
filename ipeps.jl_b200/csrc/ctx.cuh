// Engine context: one CUDA stream per context, a stream-ordered memory pool,
// per-kernel-family launch/flop counters and the small helpers every
// contraction uses.
#pragma once

#include "common.cuh"

#include <algorithm>
#include <array>
#include <atomic>
#include <map>
#include <tuple>

namespace ipeps {

enum class KFam : int {
  Permute = 0,
  GemmF64,
  GemmTF32x3,
  Reduce,
  Elementwise,
  SmallLinalg,
  Jacobi,
  Count
};

struct KStat {
  uint64_t launches = 0;
  double flops = 0;   // algorithmic flops credited (2*M*N*K per real GEMM, 8*M*N*K complex)
  double bytes = 0;   // algorithmic bytes moved (permutes, reductions)
};

enum Precision : int { kPrecFP64 = 0, kPrecMixed = 1 };

struct Ctx {
  int device = 0;
  std::shared_ptr<StreamHolder> sh;
  cudaStream_t stream = nullptr;
  int sm_count = 148;
  int precision = kPrecFP64;
  uint64_t rng_seed = 0x1234abcdULL;
  uint64_t rng_counter = 0;
  std::string last_error;
  std::array<KStat, int(KFam::Count)> stats{};
  uint64_t jacobi_sweeps = 0;
  uint64_t projector_calls = 0;
  uint64_t projector_extra_passes = 0;
  // projector adjoints whose resolvent expansion stopped at its term cap before
  // reaching its tolerance (the gradient may be inexact)
  uint64_t series_cap_hits = 0;
  // Chebyshev terms summed over all projector adjoints, and expansions redone
  // over a wider interval after the resolvent check failed
  uint64_t series_terms = 0;
  uint64_t series_retries = 0;
  // projectors whose kept triplets ended above the residual tolerance (the
  // extra passes stopped converging or ran out)
  uint64_t resid_misses = 0;
  // split-K partial sums live here (grown on demand, stream ordered)
  std::shared_ptr<DBuf> ws;
  // small device scalars (max-abs, traces, status words)
  std::shared_ptr<DBuf> scal;
  int* d_status = nullptr;
  // tile configuration and K split of the FP64 GEMMs by (m, n, k, kind: 0 real, 1 to 3
  // complex with both, the first, the second operand complex, 4 real upper triangle):
  // chosen from an estimate over all of them, so kept (bounded: emptied at 4096 shapes)
  struct GemmPlan {
    int config = 0, S = 1, cs = 1;
  };
  std::map<std::tuple<int64_t, int64_t, int64_t, int>, GemmPlan> gemm_plans;
  // per-kernel-family CUDA-event timing (enabled by ipeps_prof_enable)
  bool prof = false;
  // with prof: wall ms of the E+grad pullback's phases (checkpoint iterations,
  // energy tape, recorded recomputation of the iterations, their backward,
  // and the projector adjoints inside that backward), stream-synchronised
  std::array<double, 5> ad_phase_ms{};
  std::array<KStat, int(KFam::Count)> prof_stats{};
  std::vector<std::tuple<int, cudaEvent_t, cudaEvent_t>> prof_rec;
  std::vector<cudaEvent_t> ev_pool;
  cudaEvent_t take_event();
  // returns ms per family and clears the records
  std::array<double, int(KFam::Count)> prof_collect();

  explicit Ctx(int dev);
  ~Ctx();

  Tensor alloc(DType dt, const std::vector<int64_t>& dims);
  Tensor zeros(DType dt, const std::vector<int64_t>& dims);
  void* workspace(size_t bytes);
  void sync() { IPEPS_CUDA(cudaStreamSynchronize(stream)); }
  void count(KFam f, double flops = 0, double bytes = 0) {
    auto& s = stats[int(f)];
    s.launches++;
    s.flops += flops;
    s.bytes += bytes;
    if (prof) {
      auto& p = prof_stats[int(f)];
      p.launches++;
      p.flops += flops;
      p.bytes += bytes;
    }
  }
};

// Brackets the launches of one kernel family with CUDA events on the
// context stream while profiling is enabled.
// FP64 contractions for the lifetime of the scope, whatever the context's
// precision: the observables (energies, norms, density matrices) are
// evaluated in FP64 in both forms.
struct Fp64Scope {
  Ctx& c;
  int prev;
  explicit Fp64Scope(Ctx& cc) : c(cc), prev(cc.precision) { c.precision = kPrecFP64; }
  ~Fp64Scope() { c.precision = prev; }
  Fp64Scope(const Fp64Scope&) = delete;
  Fp64Scope& operator=(const Fp64Scope&) = delete;
};

// Programmatic dependent launch: a kernel started by launch() is handed to the device
// while its predecessor on the stream still runs, and waits (pdl_wait, the first
// statement of each such kernel, in all threads) until that one is complete and its
// writes are visible, so all memory accesses keep the stream's order.  Kernels without
// pdl_wait are started with <<< >>>.  A chain of small kernels, per kernel: 3.0 -> 1.9 us.
// No kernel signals its successor early (griddepcontrol.launch_dependents): with a
// signal at the start or at the end of the long kernels the cases differ by under 1%,
// and from GEMMs at their start D = 5, chi = 100 is 6% slower (the waiting CTAs hold SMs
// that the other stream's kernels could use).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// kern<<<grid, block, smem, stream>>>(args...) with programmatic dependent launch, in
// clusters of `cluster` CTAs when that is not 1 x 1 x 1
template <class... P, class... A>
void launch_clusters(cudaStream_t stream, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, dim3 cluster,
                     A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2]{};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster.x;
  at[1].val.clusterDim.y = cluster.y;
  at[1].val.clusterDim.z = cluster.z;
  cfg.attrs = at;
  cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
  IPEPS_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
}
template <class... P, class... A>
void launch(cudaStream_t stream, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
  launch_clusters(stream, kern, grid, block, smem, dim3(1), std::forward<A>(args)...);
}

// The dynamic shared-memory limit of a kernel is a per-function, per-device
// attribute: set it once on every device the kernel is launched on.
struct SmemAttrOnce {
  static constexpr int kMaxDevices = 64;
  std::atomic<bool> done[kMaxDevices] = {};
  template <class K>
  void ensure(K kern, int bytes) {
    int dev = 0;
    IPEPS_CUDA(cudaGetDevice(&dev));
    if (dev < kMaxDevices && done[dev].load()) return;
    IPEPS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    if (dev < kMaxDevices) done[dev].store(true);
  }
};

struct ProfScope {
  Ctx& c;
  int fam;
  cudaEvent_t a = nullptr;
  ProfScope(Ctx& cc, KFam f) : c(cc), fam(int(f)) {
    if (c.prof) {
      a = c.take_event();
      cudaEventRecord(a, c.stream);
    }
  }
  ~ProfScope() {
    if (a) {
      cudaEvent_t b = c.take_event();
      cudaEventRecord(b, c.stream);
      c.prof_rec.emplace_back(fam, a, b);
    }
  }
};

// ---------------------------------------------------------------- kernels
// permute: out = permutedims(in, perm) (0-based perm, Julia semantics:
// size(out,i) = size(in, perm[i])).
Tensor permute(Ctx& c, const Tensor& in, const std::vector<int>& perm);
// out = in (copy) into a fresh contiguous tensor
Tensor clone(Ctx& c, const Tensor& in);

// C = alpha*op(A)*op(B) + beta*C, column-major, op in {'N','T','C'}.
// Dispatches on c.precision and the size for real operands (FP64 DMMA or 3xTF32 tcgen05).
void gemm(Ctx& c, DType dt, char opA, char opB, int64_t m, int64_t n, int64_t k,
          cuDoubleComplex alpha, const void* A, int64_t lda, const void* B, int64_t ldb,
          cuDoubleComplex beta, void* C, int64_t ldc, bool force_fp64 = false);
// FP64 GEMM on the DMMA path: real, or complex128
void gemm_f64(Ctx& c, DType dt, char opA, char opB, int64_t m, int64_t n, int64_t k,
              cuDoubleComplex alpha, const void* A, int64_t lda, const void* B, int64_t ldb,
              cuDoubleComplex beta, void* C, int64_t ldc);
// real FP64 GEMM on the DMMA (FP64 tensor-core) path, op in {N, T}; upper: C is symmetric and only its
// upper triangle is needed (entries below the diagonal are left undefined)
void gemm_f64_dmma(Ctx& c, char opA, char opB, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                   int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc,
                   bool upper = false);
// complex128 GEMM on the DMMA path, op in {N, T, C}; one operand may be real (dtA or dtB F64)
void gemm_c128_dmma(Ctx& c, char opA, DType dtA, char opB, DType dtB, int64_t m, int64_t n, int64_t k,
                    cuDoubleComplex alpha, const void* A, int64_t lda, const void* B, int64_t ldb, cuDoubleComplex beta,
                    void* C, int64_t ldc);
// 3xTF32 tcgen05 GEMM for real operands (FP32-accumulated split products)
// BF16 operands (rounded from FP32 while staged), FP32 accumulation and result; op in {N, T}
void gemm_bf16(Ctx& c, char opA, char opB, int64_t m, int64_t n, int64_t k, float alpha, const float* A, int64_t lda,
               const float* B, int64_t ldb, float beta, float* C, int64_t ldc);
// An FP64 operand split once into TF32 hi/lo planes for the 3xTF32 GEMM:
// rows x Kp FP32 each, K contiguous (K-major), Kp = K rounded up to 32 with
// zero padding, the lo plane stacked after the hi plane.
struct Planes {
  Tensor buf;
  int64_t rows = 0, K = 0, Kp = 0;
  bool empty() const { return buf.empty(); }
};
// X(r, k) = kcontig ? X[k + r*ld] : X[r + k*ld], r < rows, k < K
Planes split_kmajor(Ctx& c, const double* X, int64_t ld, bool kcontig, int64_t rows, int64_t K);
// C = alpha * A B + beta * C with A given as m x k planes and B as n x k planes (B^T rows)
void gemm_tf32x3_planes(Ctx& c, const Planes& A, const Planes& B, int64_t m, int64_t n, int64_t k, double alpha,
                        double beta, double* C, int64_t ldc);
void gemm_tf32x3(Ctx& c, char opA, char opB, int64_t m, int64_t n, int64_t k, double alpha,
                 const double* A, int64_t lda, const double* B, int64_t ldb, double beta, double* C,
                 int64_t ldc);

// whether the mixed form runs an m x n x k product as 3xTF32 (else in FP64); planes_kept:
// its large operand is split already
bool tf32x3_pays(int64_t m, int64_t n, int64_t k, bool planes_kept = false);

inline cuDoubleComplex cplx(double r, double i = 0) { return make_cuDoubleComplex(r, i); }

// Matrix product helpers on 2-D tensors: returns op(A)*op(B)
Tensor matmul(Ctx& c, const Tensor& A, char opA, const Tensor& B, char opB);

// tcon: contraction with the reference's label convention (positive labels
// are summed, negative labels -1,-2,... give the output order).
Tensor tcon(Ctx& c, const Tensor& A, const std::vector<int>& la, const Tensor& B,
            const std::vector<int>& lb);
// The plan of one tcon for operands of given shapes and labels, for sums of products
// of the same contraction (the components of nested tensors): each operand is
// permuted once however many products it enters, the products are added by the GEMM
// in the layout it writes, and the sum is permuted once at the end.
class Contraction {
 public:
  Contraction(const Tensor& A, const std::vector<int>& la, const Tensor& B, const std::vector<int>& lb);
  // raw += A B (raw is allocated by the first product); both of the shapes the plan was made for
  void add(Ctx& c, Tensor& raw, const Tensor& A, const Tensor& B);
  // the sum in output order
  Tensor finish(Ctx& c, const Tensor& raw) const;

  struct Side {
    std::vector<int> perm;  // empty: used as it stands
    char op = 'N';
    int64_t ld = 1;
    std::vector<std::pair<Tensor, Tensor>> done;  // operands permuted so far (kept alive by the plan)
  };

 private:
  static Tensor prepared(Ctx& c, Side& s, const Tensor& X);
  Side a_, b_;
  bool swapped_ = false;
  int64_t m_ = 1, n_ = 1, k_ = 1;
  struct Shape {  // (no allocation: a plan is made for every product)
    int nd = 0;
    int64_t dims[kMaxDims] = {0};
    Shape() = default;
    explicit Shape(const Tensor& t) : nd(t.nd) { std::copy(t.dims, t.dims + t.nd, dims); }
    bool of(const Tensor& t) const { return t.nd == nd && std::equal(dims, dims + nd, t.dims); }
  } a_shape_, b_shape_;
  std::vector<int64_t> odims_, raw_dims_;
  std::vector<int> final_;  // permutation of the product to output order; empty: none
};

// ------------------------------------------------------------ reductions
// d_out[0] = max |x| (device scalar)
void maxabs(Ctx& c, const Tensor& x, double* d_out);
// x *= 1/d_s[0] (x real or complex), in place
void scale_inv(Ctx& c, Tensor& x, const double* d_s);
// x *= s (complex scalar), in place
void scale(Ctx& c, Tensor& x, cuDoubleComplex s);
// y += a*x
void axpy(Ctx& c, cuDoubleComplex a, const Tensor& x, Tensor& y);
// conj copy (returns new tensor; real input -> plain copy)
Tensor conj(Ctx& c, const Tensor& x);
// convert real tensor to complex128
Tensor to_complex(Ctx& c, const Tensor& x);
// ORs `bits` into the status word on the context stream (host-detected
// conditions that the caller reads with the device-side ones)
void flag_status(Ctx& c, int bits);
// nonfinite scan: sets bit in c.d_status
void check_finite(Ctx& c, const Tensor& x);
// fill with N(0,1) (counter-based hash RNG, reproducible)
void randn(Ctx& c, Tensor& x);

}  // namespace ipeps
