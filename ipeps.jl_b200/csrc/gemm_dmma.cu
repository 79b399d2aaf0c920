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
#include "dmma.cuh"

#include <atomic>
#include <iterator>
#include <mutex>

#include <cooperative_groups.h>

namespace ipeps {
namespace {

// Warps: WGM x WGN over the tile, times KW over the 16 k of a stage (each of the
// KW sums 16 / KW of them; the sums meet in shared memory at the end).
template <int BM, int BN, int WGM, int WGN, int KW, bool AK, bool BK_>
struct Geo {
  static constexpr int NT = WGM * WGN * KW * 32;
  static constexpr int ring = kStages * (Tile<double, BM, AK>::size + Tile<double, BN, BK_>::size);  // doubles
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
  pdl_wait();
  using GE = Geo<BM, BN, WGM, WGN, KW, AK, BK_>;
  constexpr int NT = GE::NT;
  constexpr int WM = BM / WGM, WN = BN / WGN;  // warp tile
  constexpr int TI = WM / 8, TJ = WN / 8;      // 8x8 DMMA tiles per warp
  using TA = Tile<double, BM, AK>;
  using TB = Tile<double, BN, BK_>;
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
  Loader<double, BM, AK, VEC, NT> la(A, lda, M, m0, kb, tid);
  Loader<double, BN, BK_, VEC, NT> lb(B, ldb, N, n0, kb, tid);
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
  pdl_wait();
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

template <int BM, int BN, int WGM, int WGN, int KW, int MINB, bool AK, bool BK_, int VEC>
void launch_cfg(Ctx& c, const Args& a, Split sp) {
  using GE = Geo<BM, BN, WGM, WGN, KW, AK, BK_>;
  auto kern = dmma_gemm_kernel<BM, BN, WGM, WGN, KW, MINB, AK, BK_, VEC>;
  static SmemAttrOnce attr;
  attr.ensure(kern, int(GE::smem));
  const int64_t gx = (a.m + BM - 1) / BM, gy = (a.n + BN - 1) / BN;
  IPEPS_CHECK(gy <= kMaxGridY, "gemm: n too large for grid");
  int64_t kchunk = (a.k + sp.S - 1) / sp.S;
  kchunk = ((kchunk + kBK - 1) / kBK) * kBK;
  const int cz = sp.S / sp.cs;
  double* partial = nullptr;
  if (cz > 1) partial = static_cast<double*>(c.workspace(size_t(cz) * a.m * a.n * sizeof(double)));
  launch_clusters(c.stream, kern, dim3(unsigned(gx), unsigned(gy), unsigned(sp.S)), GE::NT, GE::smem,
                  dim3(1, 1, unsigned(sp.cs)), a.m, a.n, a.k, kchunk, a.alpha, a.A, a.lda, a.B, a.ldb, a.beta, a.C,
                  a.ldc, partial, sp.cs, int(a.upper));
  if (cz > 1) {
    const int64_t tot = a.m * a.n;
    const bool pairs = a.ldc == a.m && (tot & 1) == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0;
    const int64_t threads = pairs ? tot / 2 : tot;
    launch(c.stream, dmma_splitk_reduce, unsigned((threads + 255) / 256), 256, 0, a.m, a.n, cz, partial, a.alpha,
           a.beta, a.C, a.ldc);
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
// 64 x 32: 81).  pipe, step: cycles of one K step (see split_cost; the
// pipe at the share of its rate that a full SM reaches).
struct Config {
  int bm, bn;
  double pipe, step;
  void (*launch)(Ctx&, const Args&, Split);
  int (*resident)(int);
};
const Config kConfigs[] = {
    {32, 32, 1024 / (4 * 0.80), 520, launch_ops<32, 32, 1, 1, 4, 4>, resident_cfg<32, 32, 1, 1, 4, 4>},
    {64, 32, 2048 / (4 * 0.86), 830, launch_ops<64, 32, 2, 1, 2, 4>, resident_cfg<64, 32, 2, 1, 2, 4>},
    {64, 64, 4096 / (4 * 0.89), 1500, launch_ops<64, 64, 2, 2, 1, 3>, resident_cfg<64, 64, 2, 2, 1, 3>},
    {128, 48, 6144 / (4 * 0.80), 1900, launch_ops<128, 48, 8, 1, 1, 2>, resident_cfg<128, 48, 8, 1, 1, 2>},
    {128, 64, 8192 / (4 * 0.81), 2500, launch_ops<128, 64, 8, 1, 1, 2>, resident_cfg<128, 64, 8, 1, 1, 2>},
    {128, 80, 10240 / (4 * 0.81), 3150, launch_ops<128, 80, 8, 1, 1, 2>, resident_cfg<128, 80, 8, 1, 1, 2>},
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

Ctx::GemmPlan plan(Ctx& c, const Args& a) {
  const auto key = std::make_tuple(a.m, a.n, a.k, a.upper ? 4 : 0);
  const auto it = c.gemm_plans.find(key);
  if (it != c.gemm_plans.end()) return it->second;
  const Residency& res = residency(c.device);
  const Ctx::GemmPlan best = best_split(kConfigs, kNumConfigs, [&](int f, int cs) { return res.n[f][cs]; }, c.sm_count,
                                        a.m, a.n, a.k, 8, a.upper);
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
  if (n > kMaxColumns) {  // (upper: square outputs are never this wide)
    for (int64_t j = 0; j < n; j += kMaxColumns)
      gemm_f64_dmma(c, opA, opB, m, std::min(kMaxColumns, n - j), k, alpha, A, lda, B + (tb ? j : j * ldb), ldb, beta,
                    C + j * ldc, ldc);
    return;
  }
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
