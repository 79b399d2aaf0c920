// Real FP64 GEMM on the FP64 tensor-core path (DMMA, mma.sync m8n8k4 .f64).
//
// tcgen05 has no FP64 kind, so FP64 matrix products on sm_100a go through the
// warp-level DMMA instruction.  Its point over a DFMA kernel is operand reuse:
// one m8n8k4 takes one A and one B value per lane and does 256 FMAs per warp,
// so a warp tile of 64x32 (or 32x32) reads shared memory at a quarter of the
// rate a register-tiled DFMA kernel needs for the same FMAs; the DFMA kernel
// was bound by shared-memory bandwidth (16 doubles per SM cycle for 64 FMAs).
//
//   C = alpha op(A) op(B) + beta C, column-major, op in {N, T}
//
// Tiles BM x BN x 16, staged by cp.async (16-byte chunks when the operand is
// 16-byte aligned with an even leading dimension, else 8-byte) through a
// three-stage shared-memory ring.  Each operand keeps its global contiguity in
// shared memory: k-contiguous operands as [mn][16 + 4], mn-contiguous ones as
// [16][BMN + 4]; both paddings make the fragment loads of a warp (8 rows x 4
// columns of doubles) conflict-free.  Out-of-range elements are zero-filled by
// the copy (src-size 0 or 8), so tiles at the edges need no special path.
// What bounds it: at 4096^3 the FP64 pipe (64 x 64 tiles, 33.9 TFLOP/s; a DMMA takes
// a scheduler's pipe 16 cycles, 37.2 TFLOP/s in all), at the engine's sizes the
// number of SMs that get a tile and the K steps they run one after another.  So K
// is split: the CTAs of a cluster add their tiles through distributed shared
// memory (no workspace, no second launch), and only where one cluster per tile
// leaves SMs idle do several go to a workspace, summed in split order by a second
// kernel.  Tile and split come from an estimate over all of them (plan).
// Back-to-back launches, before -> now: 120 x 62 x 120 9.5 -> 6.3 us, 333 x 76 x
// 333 14.5 -> 8.3, Gram 160 x 160 x 2500 26 -> 12.4 (upper triangle), 1024 x 128 x
// 1024 25 -> 17, 2500 x 160 x 2500 113 -> 80, 2500 x 200 x 2500 140 -> 101.
#include "ctx.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <iterator>
#include <mutex>

#include <cooperative_groups.h>

namespace ipeps {
namespace {

constexpr int kBK = 16;
constexpr int kStages = 3;
constexpr int kPad = 4;

__device__ __forceinline__ unsigned su32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ int64_t imin(int64_t a, int64_t b) { return a < b ? a : b; }
__device__ __forceinline__ int64_t imax(int64_t a, int64_t b) { return a > b ? a : b; }

template <int VEC>
__device__ __forceinline__ void cp_async(double* dst, const double* src, int bytes) {
  if constexpr (VEC == 2) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(su32(dst)), "l"(src), "r"(bytes));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(su32(dst)), "l"(src), "r"(bytes));
  }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Shared-memory geometry of one operand tile (BMN rows of the m or n index).
template <int BMN, bool KMAJ>
struct Tile {
  static constexpr int ld = KMAJ ? (kBK + kPad) : (BMN + kPad);  // doubles per stored row
  static constexpr int size = KMAJ ? BMN * ld : kBK * ld;         // doubles per stage
  // element (mn, k) of the tile
  static __device__ __forceinline__ int at(int mn, int k) { return KMAJ ? mn * ld + k : k * ld + mn; }
};

// Copy the operand tile [mn0, mn0 + BMN) x [k0, k0 + 16) into shared memory.
// Global layout: KMAJ: element (mn, k) at P[k + mn * ld]; else at P[mn + k * ld].
template <int BMN, bool KMAJ, int VEC, int NT>
__device__ __forceinline__ void load_tile(double* s, const double* __restrict__ P, int64_t ldp, int64_t MN,
                                          int64_t mn0, int64_t k0, int64_t ke, int tid) {
  using T = Tile<BMN, KMAJ>;
  constexpr int inner = KMAJ ? kBK : BMN;  // contiguous extent
  constexpr int outer = KMAJ ? BMN : kBK;
  constexpr int chunks = inner / VEC * outer;
#pragma unroll
  for (int r = 0; r < (chunks + NT - 1) / NT; ++r) {
    const int e = tid + r * NT;
    if (chunks % NT != 0 && e >= chunks) break;
    const int i = (e % (inner / VEC)) * VEC, o = e / (inner / VEC);
    const int mn = KMAJ ? o : i, k = KMAJ ? i : o;
    const int64_t gmn = mn0 + mn, gk = k0 + k;
    int64_t valid;
    const double* src;
    if (KMAJ) {
      valid = (gmn < MN) ? imin(VEC, imax(0, ke - gk)) : 0;
      src = P + gk + gmn * ldp;
    } else {
      valid = (gk < ke) ? imin(VEC, imax(0, MN - gmn)) : 0;
      src = P + gmn + gk * ldp;
    }
    if (valid == 0) src = P;  // any valid address; nothing is read
    cp_async<VEC>(s + T::at(mn, k), src, int(valid) * 8);
  }
}

// The same for a thread's chunks of successive tiles along k: one pointer that
// moves with k, the chunks a fixed number of rows apart (the address arithmetic of
// load_tile, per chunk and tile, cost the issue slots of ~10% of the products).
template <int BMN, bool KMAJ, int VEC, int NT>
struct Loader {
  using T = Tile<BMN, KMAJ>;
  static constexpr int inner = (KMAJ ? kBK : BMN) / VEC, outer = KMAJ ? BMN : kBK;
  static constexpr bool regular = NT % inner == 0;
  static constexpr int step = regular ? NT / inner : 1;  // rows between a thread's chunks
  const double* P;
  const double* p;
  int64_t ldp, MN, mn0;
  int i, o, mn_left;
  __device__ __forceinline__ Loader(const double* P_, int64_t ld, int64_t MN_, int64_t mn0_, int64_t k0, int tid)
      : P(P_), ldp(ld), MN(MN_), mn0(mn0_) {
    i = (tid % inner) * VEC;
    o = tid / inner;
    mn_left = int(imin(MN - mn0, BMN));
    p = KMAJ ? P + (k0 + i) + (mn0 + o) * ldp : P + (mn0 + i) + (k0 + o) * ldp;
  }
  // tile at k0 (its k's below ke) into s; then on to the next 16 k
  __device__ __forceinline__ void next(double* s, int64_t k0, int64_t ke, int tid) {
    if constexpr (!regular) {
      load_tile<BMN, KMAJ, VEC, NT>(s, P, ldp, MN, mn0, k0, ke, tid);
    } else {
      const int k_left = int(imin(ke - k0, kBK));
      const int in_left = (KMAJ ? k_left : mn_left) - i, out_left = KMAJ ? mn_left : k_left;
      const int bytes = 8 * max(0, min(VEC, in_left));
      double* d = s + (KMAJ ? T::at(o, i) : T::at(i, o));
#pragma unroll
      for (int r = 0; r < (outer + step - 1) / step; ++r) {
        const int row = o + r * step;
        if (outer % step != 0 && row >= outer) break;
        const int n = row < out_left ? bytes : 0;
        cp_async<VEC>(d + r * step * T::ld, n ? p + int64_t(r * step) * ldp : P, n);
      }
      p += KMAJ ? int64_t(kBK) : kBK * ldp;
    }
  }
};

// Warps: WGM x WGN over the tile, times KW over the 16 k of a stage (each of the
// KW sums 16 / KW of them; the sums meet in shared memory at the end).
template <int BM, int BN, int WGM, int WGN, int KW, bool AK, bool BK_>
struct Geo {
  static constexpr int NT = WGM * WGN * KW * 32;
  static constexpr int ring = kStages * (Tile<BM, AK>::size + Tile<BN, BK_>::size);  // doubles
  static constexpr int sums = (KW > 1 ? KW - 1 : 1) * BM * BN;  // KW sums, then the tile for the cluster's sum
  static constexpr size_t smem = size_t(ring > sums ? ring : sums) * sizeof(double);
};

// One tile of C per cluster of `cs` CTAs along z, each over its K chunk; the
// CTAs of a cluster add their tiles through distributed shared memory, each
// CTA a slice of the rows-by-columns of all of them, in rank order (so the
// result does not depend on timing).  More than one cluster per tile (cz > 1):
// the clusters' sums go to `partial` for dmma_splitk_reduce.  upper: only tiles
// that reach the upper triangle are formed (C symmetric).
template <int BM, int BN, int WGM, int WGN, int KW, int MINB, bool AK, bool BK_, int VEC>
__global__ void __launch_bounds__(WGM * WGN * KW * 32, MINB)
    dmma_gemm_kernel(int64_t M, int64_t N, int64_t K, int64_t kchunk, double alpha, const double* __restrict__ A,
                     int64_t lda, const double* __restrict__ B, int64_t ldb, double beta, double* __restrict__ C,
                     int64_t ldc, double* __restrict__ partial, int cs, int upper) {
  using GE = Geo<BM, BN, WGM, WGN, KW, AK, BK_>;
  constexpr int NT = GE::NT;
  constexpr int WM = BM / WGM, WN = BN / WGN;  // warp tile
  constexpr int TI = WM / 8, TJ = WN / 8;      // 8x8 DMMA tiles per warp
  using TA = Tile<BM, AK>;
  using TB = Tile<BN, BK_>;
  extern __shared__ __align__(16) double smem[];
  double* sA = smem;
  double* sB = smem + kStages * TA::size;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int kw = warp / (WGM * WGN), wmn = warp % (WGM * WGN);
  const int wm0 = (wmn % WGM) * WM, wn0 = (wmn / WGM) * WN;
  const int64_t m0 = int64_t(blockIdx.x) * BM, n0 = int64_t(blockIdx.y) * BN;
  if (upper && n0 + BN <= m0) return;  // the whole cluster: its CTAs share the tile
  const int64_t kb = int64_t(blockIdx.z) * kchunk;
  const int64_t ke = imin(K, kb + kchunk);
  const int nk = ke > kb ? int((ke - kb + kBK - 1) / kBK) : 0;

  double acc[TI][TJ][2];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < TJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  // B is consumed as (k, n): its "mn" index is n and it is k-contiguous when op(B) = N
  Loader<BM, AK, VEC, NT> la(A, lda, M, m0, kb, tid);
  Loader<BN, BK_, VEC, NT> lb(B, ldb, N, n0, kb, tid);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nk) {
      la.next(sA + s * TA::size, kb + s * kBK, ke, tid);
      lb.next(sB + s * TB::size, kb + s * kBK, ke, tid);
    }
    cp_commit();
  }
  int cur = 0, fill = kStages - 1;  // stages read and filled in this step
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<kStages - 2>();
    __syncthreads();
    const int pf = kt + kStages - 1;
    if (pf < nk) {
      la.next(sA + fill * TA::size, kb + int64_t(pf) * kBK, ke, tid);
      lb.next(sB + fill * TB::size, kb + int64_t(pf) * kBK, ke, tid);
    }
    cp_commit();
    const double* a_s = sA + cur * TA::size;
    const double* b_s = sB + cur * TB::size;
    cur = cur + 1 == kStages ? 0 : cur + 1;
    fill = fill + 1 == kStages ? 0 : fill + 1;
#pragma unroll
    for (int k4 = 0; k4 < kBK / KW; k4 += 4) {
      const int kk = kw * (kBK / KW) + k4;
      double a[TI], b[TJ];
#pragma unroll
      for (int i = 0; i < TI; ++i) a[i] = a_s[TA::at(wm0 + i * 8 + g, kk + t)];
#pragma unroll
      for (int j = 0; j < TJ; ++j) b[j] = b_s[TB::at(wn0 + j * 8 + g, kk + t)];
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
  }
  cp_wait<0>();

  // lane holds rows g, columns 2t and 2t+1 of each 8x8 tile
  if constexpr (KW > 1) {
    __syncthreads();
    if (kw > 0) {
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j)
          *reinterpret_cast<double2*>(smem + ((kw - 1) * WGM * WGN + wmn) * (WM * WN) + (i * TJ + j) * 64 + 2 * lane) =
              make_double2(acc[i][j][0], acc[i][j][1]);
    }
    __syncthreads();
    if (kw == 0) {
#pragma unroll
      for (int q = 0; q < KW - 1; ++q)
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
          for (int j = 0; j < TJ; ++j) {
            const double2 v = *reinterpret_cast<const double2*>(smem + (q * WGM * WGN + wmn) * (WM * WN) +
                                                                (i * TJ + j) * 64 + 2 * lane);
            acc[i][j][0] += v.x;
            acc[i][j][1] += v.y;
          }
    }
  }
  if (cs > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();  // the ring (and the KW sums) are read
    if (kw == 0) {
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) smem[wm0 + i * 8 + g + (wn0 + j * 8 + 2 * t + e) * BM] = acc[i][j][e];
    }
    cluster.sync();
    const int rank = int(cluster.block_rank());
    constexpr int pairs = BM * BN / 2;  // two rows at a time
    const int per = (pairs + cs - 1) / cs, last = min(pairs, (rank + 1) * per);
    double* P = partial ? partial + int64_t(blockIdx.z / unsigned(cs)) * M * N : nullptr;
    for (int p = rank * per + tid; p < last; p += NT) {
      const int r = (2 * p) % BM, col = (2 * p) / BM;
      const int64_t gm = m0 + r, gn = n0 + col;
      if (gm >= M || gn >= N) continue;
      double2 v = *reinterpret_cast<const double2*>(cluster.map_shared_rank(smem, 0) + 2 * p);
#pragma unroll 7
      for (int q = 1; q < cs; ++q) {
        const double2 w = *reinterpret_cast<const double2*>(cluster.map_shared_rank(smem, q) + 2 * p);
        v.x += w.x;
        v.y += w.y;
      }
      if (P) {
        P[gm + gn * M] = v.x;
        if (gm + 1 < M) P[gm + 1 + gn * M] = v.y;
      } else {
        double* c = C + gm + gn * ldc;
        c[0] = beta != 0.0 ? fma(beta, c[0], alpha * v.x) : alpha * v.x;
        if (gm + 1 < M) c[1] = beta != 0.0 ? fma(beta, c[1], alpha * v.y) : alpha * v.y;
      }
    }
    cluster.sync();  // no CTA leaves while another still reads its tile
    return;
  }
  if (kw > 0) return;
#pragma unroll
  for (int i = 0; i < TI; ++i) {
    const int64_t gm = m0 + wm0 + i * 8 + g;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TJ; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t gn = n0 + wn0 + j * 8 + 2 * t + e;
        if (gn >= N) continue;
        if (partial) {
          partial[int64_t(blockIdx.z) * M * N + gm + gn * M] = acc[i][j][e];
        } else {
          double v = alpha * acc[i][j][e];
          if (beta != 0.0) v = fma(beta, C[gm + gn * ldc], v);
          C[gm + gn * ldc] = v;
        }
      }
    }
  }
}

// Sum of the S split-K partial products (in split order, so the result does
// not depend on the launch).  Contiguous C (ldc == M) takes two elements per
// thread with 16-byte loads; the general case one element per thread.
__global__ void dmma_splitk_reduce(int64_t M, int64_t N, int S, const double* __restrict__ partial, double alpha,
                                   double beta, double* __restrict__ C, int64_t ldc) {
  const int64_t tot = M * N;
  if (ldc == M && (tot & 1) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0) {
    const int64_t i2 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, idx = 2 * i2;
    if (idx >= tot) return;
    double2 acc = *reinterpret_cast<const double2*>(partial + idx);
    for (int z = 1; z < S; ++z) {
      const double2 p = *reinterpret_cast<const double2*>(partial + int64_t(z) * tot + idx);
      acc.x += p.x;
      acc.y += p.y;
    }
    double2 v = make_double2(alpha * acc.x, alpha * acc.y);
    if (beta != 0.0) {
      const double2 c = *reinterpret_cast<const double2*>(C + idx);
      v.x = fma(beta, c.x, v.x);
      v.y = fma(beta, c.y, v.y);
    }
    *reinterpret_cast<double2*>(C + idx) = v;
    return;
  }
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= tot) return;
  const int64_t gn = idx / M, gm = idx - gn * M;
  double s = partial[idx];
  for (int z = 1; z < S; ++z) s += partial[int64_t(z) * tot + idx];
  double v = alpha * s;
  if (beta != 0.0) v = fma(beta, C[gm + gn * ldc], v);
  C[gm + gn * ldc] = v;
}

struct Args {
  bool ta, tb, vec, upper;
  int64_t m, n, k;
  double alpha;
  const double* A;
  int64_t lda;
  const double* B;
  int64_t ldb;
  double beta;
  double* C;
  int64_t ldc;
};

// S K chunks per tile: clusters of cs CTAs, S / cs clusters
struct Split {
  int S = 1, cs = 1;
};

// CTAs of one kernel that run at the same time in clusters of cs, asked of the
// driver once per kernel, cluster size and device: clusters need their SMs in one
// GPC, so the larger ones leave some idle (128 x 80 tiles in clusters of 7: 40
// clusters did not run at once on 148 SMs x 2, 117 us instead of 81).
template <class K>
int resident(K kern, int threads, size_t smem, int cs) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1, 1, unsigned(cs));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = unsigned(cs);
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  IPEPS_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
  return n * cs;
}

template <int BM, int BN, int WGM, int WGN, int KW, int MINB, bool AK, bool BK_, int VEC>
void launch_cfg(Ctx& c, const Args& a, Split sp) {
  using GE = Geo<BM, BN, WGM, WGN, KW, AK, BK_>;
  auto kern = dmma_gemm_kernel<BM, BN, WGM, WGN, KW, MINB, AK, BK_, VEC>;
  static SmemAttrOnce attr;
  attr.ensure(kern, int(GE::smem));
  const int64_t gx = (a.m + BM - 1) / BM, gy = (a.n + BN - 1) / BN;
  IPEPS_CHECK(gy <= 65535, "gemm: n too large for grid");
  int64_t kchunk = (a.k + sp.S - 1) / sp.S;
  kchunk = ((kchunk + kBK - 1) / kBK) * kBK;
  const int cz = sp.S / sp.cs;
  double* partial = nullptr;
  if (cz > 1) partial = static_cast<double*>(c.workspace(size_t(cz) * a.m * a.n * sizeof(double)));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(gx), unsigned(gy), unsigned(sp.S));
  cfg.blockDim = dim3(GE::NT);
  cfg.dynamicSmemBytes = GE::smem;
  cfg.stream = c.stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = unsigned(sp.cs);
  cfg.attrs = &at;
  cfg.numAttrs = sp.cs > 1 ? 1 : 0;
  IPEPS_CUDA(cudaLaunchKernelEx(&cfg, kern, a.m, a.n, a.k, kchunk, a.alpha, a.A, a.lda, a.B, a.ldb, a.beta, a.C, a.ldc,
                                partial, sp.cs, int(a.upper)));
  if (cz > 1) {
    const int64_t tot = a.m * a.n;
    const bool pairs = a.ldc == a.m && (tot & 1) == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0;
    const int64_t threads = pairs ? tot / 2 : tot;
    dmma_splitk_reduce<<<unsigned((threads + 255) / 256), 256, 0, c.stream>>>(a.m, a.n, cz, partial, a.alpha, a.beta,
                                                                              a.C, a.ldc);
    IPEPS_LAUNCH_CHECK();
    c.count(KFam::Reduce, 0, double(cz + 2) * tot * sizeof(double));
  }
}

template <int BM, int BN, int WGM, int WGN, int KW, int MINB>
void launch_ops(Ctx& c, const Args& a, Split sp) {
  // A is k-contiguous when op(A) = T; B is k-contiguous when op(B) = N
#define IPEPS_DMMA_CASE(AK, BKM)                                                                   \
  a.vec ? launch_cfg<BM, BN, WGM, WGN, KW, MINB, AK, BKM, 2>(c, a, sp)                              \
        : launch_cfg<BM, BN, WGM, WGN, KW, MINB, AK, BKM, 1>(c, a, sp)
  if (a.ta && !a.tb) IPEPS_DMMA_CASE(true, true);
  else if (a.ta && a.tb) IPEPS_DMMA_CASE(true, false);
  else if (!a.ta && !a.tb) IPEPS_DMMA_CASE(false, true);
  else IPEPS_DMMA_CASE(false, false);
#undef IPEPS_DMMA_CASE
}

constexpr int kMaxCluster = 8;

template <int BM, int BN, int WGM, int WGN, int KW, int MINB>
int resident_cfg(int cs) {
  using GE = Geo<BM, BN, WGM, WGN, KW, true, true>;
  auto kern = dmma_gemm_kernel<BM, BN, WGM, WGN, KW, MINB, true, true, 2>;
  static SmemAttrOnce attr;
  attr.ensure(kern, int(GE::smem));
  return resident(kern, GE::NT, GE::smem, cs);
}

// Tile configurations.  32 x 32 tiles reach the most SMs with the fewest K steps
// and win for small outputs (62 x 62 x 120: 6.3 us, 10.4 with 64 x 64; 128 x 128 x
// 1024: 8.3 and 12.4), 64 x 32 for the sketches (2500 x 160 x 2500: 80 us, 64 x 64:
// 90), 64 x 64 for large ones (4096^3: 4.06 ms, 128 x 80: 4.23), the 128-row tiles
// for narrow outputs (a leg of D^2 d = 50: 128 x 64, 59.5 us at 250000 x 50 x 25,
// 64 x 32: 81).  pipe: share of the FP64 pipe's rate that a full SM reaches, step:
// cycles that one CTA alone needs per K step (see estimate).
struct Config {
  int bm, bn;
  double pipe, step;
  void (*launch)(Ctx&, const Args&, Split);
  int (*resident)(int);
};
const Config kConfigs[] = {
    {32, 32, 0.80, 520, launch_ops<32, 32, 1, 1, 4, 4>, resident_cfg<32, 32, 1, 1, 4, 4>},
    {64, 32, 0.86, 830, launch_ops<64, 32, 2, 1, 2, 4>, resident_cfg<64, 32, 2, 1, 2, 4>},
    {64, 64, 0.89, 1500, launch_ops<64, 64, 2, 2, 1, 3>, resident_cfg<64, 64, 2, 2, 1, 3>},
    {128, 48, 0.80, 1900, launch_ops<128, 48, 8, 1, 1, 2>, resident_cfg<128, 48, 8, 1, 1, 2>},
    {128, 64, 0.81, 2500, launch_ops<128, 64, 8, 1, 1, 2>, resident_cfg<128, 64, 8, 1, 1, 2>},
    {128, 80, 0.81, 3150, launch_ops<128, 80, 8, 1, 1, 2>, resident_cfg<128, 80, 8, 1, 1, 2>},
};
constexpr int kNumConfigs = int(std::size(kConfigs));

// resident CTAs per configuration and cluster size, per device
struct Residency {
  std::once_flag once;
  int n[kNumConfigs][kMaxCluster + 1] = {};
};
const Residency& residency(int device) {
  static Residency r[SmemAttrOnce::kMaxDevices];
  Residency& q = r[device % SmemAttrOnce::kMaxDevices];
  std::call_once(q.once, [&] {
    for (int f = 0; f < kNumConfigs; ++f)
      for (int cs = 1; cs <= kMaxCluster; ++cs) q.n[f][cs] = std::max(1, kConfigs[f].resident(cs));
  });
  return q;
}

// Estimated cycles of a configuration with S K chunks in clusters of cs: waves of
// CTAs, each as long as its steps take on the fullest SM.  The constants are fitted
// to a sweep of all configurations and splits over 151 shapes (D = 2 to 5, chi = 9 to
// 100): the choice is 2.3% slower than the best of the sweep on average.
double estimate(const Config& f, const Args& a, int sms, int slots, int S, int cs) {
  const double gx = double((a.m + f.bm - 1) / f.bm), gy = double((a.n + f.bn - 1) / f.bn);
  const double tiles = a.upper ? 0.5 * gx * gy + 0.5 * std::max(gx, gy) : gx * gy;
  const double steps = std::ceil(std::ceil(double(a.k) / kBK) / S), ctas = tiles * S;
  const double tile = f.bm * f.bn / (4.0 * f.pipe);  // one step of one CTA on the FP64 pipe of its SM
  const double waves = std::floor(ctas / slots), rest = ctas - waves * slots;
  const double full = std::max(1.0, double(slots) / sms);
  // a cluster's CTAs share SMs sooner than the same number of single ones
  const double part = std::min(full, std::ceil(rest / sms) * (cs > 1 ? 1.0 + 0.025 * (cs - 1) : 1.0));
  double t = waves * (steps * std::max(full * tile, f.step) + 4100.0);
  if (rest > 0) t += steps * std::max(part * tile, f.step) + 4100.0;
  if (cs > 1) t = t * (cs > 2 && waves >= 1 ? 1.04 : 1.0) + (waves + 1) * (1300.0 + 0.43 * f.bm * f.bn);
  if (S > cs) t += 7000.0 + (S / cs) * (106.0 + double(a.m) * double(a.n) * 16.0 / 9400.0);
  return t;
}

Ctx::GemmPlan plan(Ctx& c, const Args& a) {
  const auto key = std::make_tuple(a.m, a.n, a.k, a.upper);
  const auto it = c.gemm_plans.find(key);
  if (it != c.gemm_plans.end()) return it->second;
  const Residency& res = residency(c.device);
  Ctx::GemmPlan best;
  double t = -1.0;
  for (int f = 0; f < kNumConfigs; ++f)
    for (int S = 1; S <= 1024; S = S < 8 ? S + 1 : 2 * S) {
      if (S > 1 && int64_t(S) * 2 * kBK > a.k) break;
      for (int cs : {std::min(S, kMaxCluster), 1}) {
        if ((cs & (cs - 1)) != 0) continue;  // clusters of 3, 5, 6, 7 measured behind those of 2, 4, 8
        if (cs == 1 && S > 1 && double(S) * double(a.m) * double(a.n) > 5e7) break;  // at most 400 MB of partial sums
        const double e = estimate(kConfigs[f], a, c.sm_count, res.n[f][cs], S, cs);
        if (t < 0 || e < t) {
          best = {f, S, cs};
          t = e;
        }
      }
    }
  if (c.gemm_plans.size() >= 4096) c.gemm_plans.clear();
  c.gemm_plans[key] = best;
  return best;
}

}  // namespace

void gemm_f64_dmma(Ctx& c, char opA, char opB, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                   int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc, bool upper) {
  if (m <= 0 || n <= 0) return;
  IPEPS_CHECK(k > 0, "gemm: k == 0 is not supported");
  const bool ta = (opA == 'T' || opA == 't'), tb = (opB == 'T' || opB == 't');
  IPEPS_CHECK(ta || opA == 'N' || opA == 'n', "gemm: bad op");
  IPEPS_CHECK(tb || opB == 'N' || opB == 'n', "gemm: bad op");
  ProfScope ps(c, KFam::GemmF64);
  const bool vec = (reinterpret_cast<uintptr_t>(A) % 16 == 0) && (reinterpret_cast<uintptr_t>(B) % 16 == 0) &&
                   lda % 2 == 0 && ldb % 2 == 0;
  const Args a{ta, tb, vec, upper, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc};
  const Ctx::GemmPlan p = plan(c, a);
  kConfigs[p.config].launch(c, a, {p.S, p.cs});
  c.count(KFam::GemmF64, 2.0 * double(m) * double(n) * double(k));
}

}  // namespace ipeps
