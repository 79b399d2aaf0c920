// Dispatch of the FP64 GEMMs (real: gemm_dmma.cu, complex128: gemm_zmma.cu), and the
// real register-tiled FMA kernel of the allocation-free entry point: 64x64x16 tiles,
// 4x4 outputs per thread, operands staged through shared memory with one register
// prefetch stage, deterministic split-K for skinny problems (few output tiles, long
// K): partial products go to a fixed scratch array and are summed in a fixed order.
#include "ctx.cuh"

#include <algorithm>

namespace ipeps {
namespace {

// op codes: 0 = N, 1 = T
template <int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
    gemm_kernel(int opA, int opB, int64_t M, int64_t N, int64_t K, int64_t kchunk,
                double alpha, const double* __restrict__ A, int64_t lda,
                const double* __restrict__ B, int64_t ldb, double beta, double* __restrict__ C,
                int64_t ldc, double* __restrict__ partial) {
  constexpr int NT = (BM / TM) * (BN / TN);
  constexpr int TX = BM / TM;  // threads along m
  constexpr int A_PER = BM * BK / NT;
  constexpr int B_PER = BN * BK / NT;
  static_assert(A_PER >= 1 && B_PER >= 1, "tile too small");
  __shared__ double As[2][BK][BM + 1];
  __shared__ double Bs[2][BK][BN + 1];

  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const int64_t m0 = int64_t(blockIdx.x) * BM;
  const int64_t n0 = int64_t(blockIdx.y) * BN;
  const int64_t kb = int64_t(blockIdx.z) * kchunk;
  const int64_t ke = min(K, kb + kchunk);

  double acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0;

  double ra[A_PER], rb[B_PER];

  auto load_a = [&](int64_t k0) {
#pragma unroll
    for (int r = 0; r < A_PER; ++r) {
      int e = tid + r * NT;
      int mi, ki;
      if (opA == 0) { mi = e % BM; ki = e / BM; }
      else { ki = e % BK; mi = e / BK; }
      int64_t gm = m0 + mi, gk = k0 + ki;
      double v = 0.0;
      if (gm < M && gk < ke) {
        v = (opA == 0) ? A[gm + gk * lda] : A[gk + gm * lda];
      }
      ra[r] = v;
    }
  };
  auto load_b = [&](int64_t k0) {
#pragma unroll
    for (int r = 0; r < B_PER; ++r) {
      int e = tid + r * NT;
      int ni, ki;
      if (opB == 0) { ki = e % BK; ni = e / BK; }
      else { ni = e % BN; ki = e / BN; }
      int64_t gn = n0 + ni, gk = k0 + ki;
      double v = 0.0;
      if (gn < N && gk < ke) {
        v = (opB == 0) ? B[gk + gn * ldb] : B[gn + gk * ldb];
      }
      rb[r] = v;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int r = 0; r < A_PER; ++r) {
      int e = tid + r * NT;
      int mi, ki;
      if (opA == 0) { mi = e % BM; ki = e / BM; }
      else { ki = e % BK; mi = e / BK; }
      As[buf][ki][mi] = ra[r];
    }
#pragma unroll
    for (int r = 0; r < B_PER; ++r) {
      int e = tid + r * NT;
      int ni, ki;
      if (opB == 0) { ki = e % BK; ni = e / BK; }
      else { ni = e % BN; ki = e / BN; }
      Bs[buf][ki][ni] = rb[r];
    }
  };

  int buf = 0;
  if (kb < ke) {
    load_a(kb);
    load_b(kb);
    store(0);
  }
  __syncthreads();
  for (int64_t k0 = kb; k0 < ke; k0 += BK) {
    const bool more = k0 + BK < ke;
    if (more) {
      load_a(k0 + BK);
      load_b(k0 + BK);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      double a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[buf][kk][tx + i * TX];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[buf][kk][ty + j * (BN / TN)];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    if (more) {
      store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }

  // epilogue
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int64_t gm = m0 + tx + i * TX;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int64_t gn = n0 + ty + j * (BN / TN);
      if (gn >= N) continue;
      if (partial) {
        partial[int64_t(blockIdx.z) * M * N + gm + gn * M] = acc[i][j];
      } else {
        double v = acc[i][j] * alpha;
        if (beta != 0.0) v += C[gm + gn * ldc] * beta;
        C[gm + gn * ldc] = v;
      }
    }
  }
}

__global__ void splitk_reduce(int64_t M, int64_t N, int S, const double* __restrict__ partial,
                              double alpha, double beta, double* __restrict__ C,
                              int64_t ldc) {
  int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= M * N) return;
  int64_t gm = idx % M, gn = idx / M;
  double s = partial[idx];
  for (int z = 1; z < S; ++z) s += partial[int64_t(z) * M * N + idx];
  double v = s * alpha;
  if (beta != 0.0) v += C[gm + gn * ldc] * beta;
  C[gm + gn * ldc] = v;
}

int opcode(char o) {
  switch (o) {
    case 'N': case 'n': return 0;
    case 'T': case 't': return 1;
    case 'C': case 'c': return 2;
  }
  throw Error(kEInval, "gemm: bad op");
}

}  // namespace

void gemm_f64(Ctx& c, DType dt, char opA, char opB, int64_t m, int64_t n, int64_t k,
              cuDoubleComplex alpha, const void* A, int64_t lda, const void* B, int64_t ldb,
              cuDoubleComplex beta, void* C, int64_t ldc) {
  if (m <= 0 || n <= 0) return;
  int oa = opcode(opA), ob = opcode(opB);
  IPEPS_CHECK(k > 0, "gemm: k == 0 is not supported");
  if (dt == DType::F64) {
    IPEPS_CHECK(oa != 2 && ob != 2, "gemm: conjugate op on real data");
    gemm_f64_dmma(c, opA, opB, m, n, k, alpha.x, static_cast<const double*>(A), lda, static_cast<const double*>(B),
                  ldb, beta.x, static_cast<double*>(C), ldc);
  } else {
    gemm_c128_dmma(c, opA, dt, opB, dt, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
  }
}

}  // namespace ipeps

// ---------------------------------------------------------------------------
// Allocation-free variant of the split-K FP64 GEMM.
//
// Some callers cannot call cudaMalloc: a host framework that owns every byte
// of device memory through its own pool (a Julia CUDA.jl session, a plugin
// host with a fixed budget), or a latency-critical section where
// cudaMalloc/cudaFree, which may synchronise the device, are not allowed.
// For them the split-K partial sums live in this fixed device array
// (4 MiB = 524288 doubles; every GPU that loads the library holds it until
// the process exits).  The caller passes device pointers for A, B and C and a
// stream.  The split factor S is capped so that S*m*n partial sums fit in the
// array; an output of more than 262144 elements therefore runs unsplit and
// touches no scratch at all.  Requests the kernel grid cannot cover
// (ceil(n/64) > 65535) are rejected with IPEPS_EINVAL and a message on stderr.
//
// The first call on a device looks up the array's device address with
// cudaGetSymbolAddress (with that device current); make that first call
// before any stream capture.  Every call shares the array: calls that overlap
// on the GPU (different streams, or threads without ordering) race on it.
// Each call overwrites all the partial sums it reads, so nothing needs
// clearing between calls.
// ---------------------------------------------------------------------------
#include <mutex>

#include "../../include/ipeps_b200.h"

namespace ipeps {
namespace {

constexpr int64_t kNoAllocScratchDoubles = int64_t(1) << 19;  // 4 MiB of FP64 partial sums
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) double g_noalloc_splitk_scratch[kNoAllocScratchDoubles];

std::mutex g_noalloc_mu;
double* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device (set-up once per device).
cudaError_t noalloc_scratch(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_splitk_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

}  // namespace
}  // namespace ipeps

extern "C" int ipeps_gemm_f64_noalloc(char opA, char opB, int64_t m, int64_t n, int64_t k, double alpha,
                                      const double* A, int64_t lda, const double* B, int64_t ldb, double beta,
                                      double* C, int64_t ldc, void* stream) {
  using namespace ipeps;
  if (!A || !B || !C || m <= 0 || n <= 0 || k <= 0) return IPEPS_EINVAL;
  int oa, ob;
  try {
    oa = opcode(opA);
    ob = opcode(opB);
  } catch (...) {
    return IPEPS_EINVAL;
  }
  if (oa == 2 || ob == 2) return IPEPS_EINVAL;  // real data: 'C' is not meaningful
  if (lda < ((oa == 0) ? m : k) || ldb < ((ob == 0) ? k : n) || ldc < m) return IPEPS_EINVAL;
  constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, NT = (BM / TM) * (BN / TN);
  const int64_t gx = (m + BM - 1) / BM, gy = (n + BN - 1) / BN;
  if (gy > 65535 || gx > int64_t(0x7fffffff)) {
    std::fprintf(stderr, "ipeps_gemm_f64_noalloc: m = %lld, n = %lld exceed the kernel grid (n <= %lld)\n",
                 static_cast<long long>(m), static_cast<long long>(n), 65535LL * BN);
    return IPEPS_EINVAL;
  }
  double* scratch = nullptr;
  if (noalloc_scratch(&scratch) != cudaSuccess) return IPEPS_ECUDA;
  int sms = 148;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // same split heuristic as the allocating path, capped by the scratch size
  const int64_t tiles = gx * gy, target = 2LL * sms;
  int64_t S = 1;
  if (tiles < target && k >= 8 * BK * 2) S = std::min<int64_t>(std::min<int64_t>((target + tiles - 1) / tiles, k / (8 * BK)), 64);
  // cap by the scratch: S * m * n partial sums at most (S = 1 uses none)
  S = std::max<int64_t>(1, std::min<int64_t>(S, kNoAllocScratchDoubles / (m * n)));
  int64_t kchunk = (k + S - 1) / S;
  kchunk = ((kchunk + BK - 1) / BK) * BK;
  S = (k + kchunk - 1) / kchunk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  dim3 grid{unsigned(gx), unsigned(gy), unsigned(S)};
  gemm_kernel<BM, BN, BK, TM, TN><<<grid, NT, 0, st>>>(oa, ob, m, n, k, kchunk, alpha, A, lda, B, ldb, beta, C, ldc,
                                                                S > 1 ? scratch : nullptr);
  if (cudaGetLastError() != cudaSuccess) return IPEPS_ECUDA;
  if (S > 1) {
    const int64_t tot = m * n;
    splitk_reduce<<<unsigned((tot + 255) / 256), 256, 0, st>>>(m, n, int(S), scratch, alpha, beta, C, ldc);
    if (cudaGetLastError() != cudaSuccess) return IPEPS_ECUDA;
  }
  return IPEPS_OK;
}
