// complex128 GEMM on the FP64 tensor cores: C = alpha op(A) op(B) + beta C, column-
// major, op in {N, T, C}; either operand may be real (FP64) as it stands.
//
// A complex product of 8 x 8 x 4 is four DMMAs (re += ar br - ai bi, im += ar bi +
// ai br), with a real operand two; the SIMT kernel this one replaces needed both
// operands complex (a conversion launch and four times the products for a real one)
// and ran on 64 x 64 tiles only, one or two CTAs at the engine's sizes.  Bound there by
// the K steps one after another, so the split of K inside clusters and the choice
// of tile are those of the real kernel (dmma.cuh).  Per product, before -> now:
// 66 x 66 x 128 39 -> 6.6 us (with a real operand 6.5), 48 x 432 x 48 17 -> 6.4 (5.3),
// 288 x 288 x 1296 110 -> 41 (25).
#include "dmma.cuh"

#include <cooperative_groups.h>
#include <iterator>
#include <mutex>
#include <type_traits>

namespace ipeps {
namespace {

template <int BM, int BN, int WGM, int WGN, int KW, class EA, class EB, bool AK, bool BK_>
struct Geo {
  static constexpr int NT = WGM * WGN * KW * 32;
  static constexpr size_t stageA = size_t(Tile<EA, BM, AK>::size) * sizeof(EA);
  static constexpr size_t stageB = size_t(Tile<EB, BN, BK_>::size) * sizeof(EB);
  static constexpr size_t ring = kStages * (stageA + stageB);
  static constexpr size_t sums = size_t(KW > 1 ? KW - 1 : 1) * BM * BN * 16;
  static constexpr size_t smem = ring > sums ? ring : sums;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ void store_c(double2* c, double2 v, double2 alpha, double2 beta) {
  double2 r = cmul(alpha, v);
  if (beta.x != 0.0 || beta.y != 0.0) {
    const double2 o = cmul(beta, *c);
    r.x += o.x;
    r.y += o.y;
  }
  *c = r;
}

// Tiles, splits and sums as dmma_gemm_kernel (gemm_dmma.cu); sa, sb: -1 conjugates
// the operand.
template <int BM, int BN, int WGM, int WGN, int KW, class EA, class EB, bool AK, bool BK_>
__global__ void __launch_bounds__(WGM * WGN * KW * 32)
    zmma_gemm_kernel(int64_t M, int64_t N, int64_t K, int64_t kchunk, double2 alpha, const EA* __restrict__ A,
                     int64_t lda, double sa, const EB* __restrict__ B, int64_t ldb, double sb, double2 beta,
                     double2* __restrict__ C, int64_t ldc, double2* __restrict__ partial, int cs) {
  pdl_wait();
  using GE = Geo<BM, BN, WGM, WGN, KW, EA, EB, AK, BK_>;
  constexpr bool CA = std::is_same_v<EA, double2>, CB = std::is_same_v<EB, double2>;
  constexpr int NT = GE::NT;
  constexpr int WM = BM / WGM, WN = BN / WGN, TI = WM / 8, TJ = WN / 8;
  using TA = Tile<EA, BM, AK>;
  using TB = Tile<EB, BN, BK_>;
  extern __shared__ __align__(16) char smem[];
  EA* sA = reinterpret_cast<EA*>(smem);
  EB* sB = reinterpret_cast<EB*>(smem + kStages * GE::stageA);
  double2* sums = reinterpret_cast<double2*>(smem);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int kw = warp / (WGM * WGN), wmn = warp % (WGM * WGN);
  const int wm0 = (wmn % WGM) * WM, wn0 = (wmn / WGM) * WN;
  const int64_t m0 = int64_t(blockIdx.x) * BM, n0 = int64_t(blockIdx.y) * BN;
  const int64_t kb = int64_t(blockIdx.z) * kchunk;
  const int64_t ke = imin(K, kb + kchunk);
  const int nk = ke > kb ? int((ke - kb + kBK - 1) / kBK) : 0;

  double re[TI][TJ][2], im[TI][TJ][2];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < TJ; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;

  Loader<EA, BM, AK, 1, NT> la(A, lda, M, m0, kb, tid);
  Loader<EB, BN, BK_, 1, NT> lb(B, ldb, N, n0, kb, tid);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nk) {
      la.next(sA + s * TA::size, kb + s * kBK, ke, tid);
      lb.next(sB + s * TB::size, kb + s * kBK, ke, tid);
    }
    cp_commit();
  }
  int cur = 0, fill = kStages - 1;
  for (int kt = 0; kt < nk; ++kt) {
    cp_wait<kStages - 2>();
    __syncthreads();
    const int pf = kt + kStages - 1;
    if (pf < nk) {
      la.next(sA + fill * TA::size, kb + int64_t(pf) * kBK, ke, tid);
      lb.next(sB + fill * TB::size, kb + int64_t(pf) * kBK, ke, tid);
    }
    cp_commit();
    const EA* a_s = sA + cur * TA::size;
    const EB* b_s = sB + cur * TB::size;
    cur = cur + 1 == kStages ? 0 : cur + 1;
    fill = fill + 1 == kStages ? 0 : fill + 1;
#pragma unroll
    for (int k4 = 0; k4 < kBK / KW; k4 += 4) {
      const int kk = kw * (kBK / KW) + k4;
      EA a[TI];
      EB b[TJ];
#pragma unroll
      for (int i = 0; i < TI; ++i) {
        a[i] = a_s[TA::at(wm0 + i * 8 + g, kk + t)];
        if constexpr (CA) a[i].y *= sa;
      }
#pragma unroll
      for (int j = 0; j < TJ; ++j) {
        b[j] = b_s[TB::at(wn0 + j * 8 + g, kk + t)];
        if constexpr (CB) b[j].y *= sb;
      }
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) {
          if constexpr (CA && CB) {
            dmma(re[i][j][0], re[i][j][1], a[i].x, b[j].x);
            dmma(im[i][j][0], im[i][j][1], a[i].x, b[j].y);
            dmma(re[i][j][0], re[i][j][1], -a[i].y, b[j].y);
            dmma(im[i][j][0], im[i][j][1], a[i].y, b[j].x);
          } else if constexpr (CA) {
            dmma(re[i][j][0], re[i][j][1], a[i].x, b[j]);
            dmma(im[i][j][0], im[i][j][1], a[i].y, b[j]);
          } else {
            dmma(re[i][j][0], re[i][j][1], a[i], b[j].x);
            dmma(im[i][j][0], im[i][j][1], a[i], b[j].y);
          }
        }
    }
  }
  cp_wait<0>();

  if constexpr (KW > 1) {
    __syncthreads();
    if (kw > 0) {
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            sums[((kw - 1) * WGM * WGN + wmn) * (WM * WN) + (i * TJ + j) * 64 + e * 32 + lane] =
                make_double2(re[i][j][e], im[i][j][e]);
    }
    __syncthreads();
    if (kw == 0) {
#pragma unroll
      for (int q = 0; q < KW - 1; ++q)
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
          for (int j = 0; j < TJ; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const double2 v = sums[(q * WGM * WGN + wmn) * (WM * WN) + (i * TJ + j) * 64 + e * 32 + lane];
              re[i][j][e] += v.x;
              im[i][j][e] += v.y;
            }
    }
  }
  if (cs > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();
    if (kw == 0) {
#pragma unroll
      for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            sums[wm0 + i * 8 + g + (wn0 + j * 8 + 2 * t + e) * BM] = make_double2(re[i][j][e], im[i][j][e]);
    }
    cluster.sync();
    const int rank = int(cluster.block_rank());
    const int per = (BM * BN + cs - 1) / cs, last = min(BM * BN, (rank + 1) * per);
    double2* P = partial ? partial + int64_t(blockIdx.z / unsigned(cs)) * M * N : nullptr;
    for (int p = rank * per + tid; p < last; p += NT) {
      const int64_t gm = m0 + p % BM, gn = n0 + p / BM;
      if (gm >= M || gn >= N) continue;
      double2 v = cluster.map_shared_rank(sums, 0)[p];
#pragma unroll 7
      for (int q = 1; q < cs; ++q) {
        const double2 w = cluster.map_shared_rank(sums, q)[p];
        v.x += w.x;
        v.y += w.y;
      }
      if (P) P[gm + gn * M] = v;
      else store_c(C + gm + gn * ldc, v, alpha, beta);
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
    for (int j = 0; j < TJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t gn = n0 + wn0 + j * 8 + 2 * t + e;
        if (gn >= N) continue;
        const double2 v = make_double2(re[i][j][e], im[i][j][e]);
        if (partial) partial[int64_t(blockIdx.z) * M * N + gm + gn * M] = v;
        else store_c(C + gm + gn * ldc, v, alpha, beta);
      }
  }
}

// sum of the clusters' partial products, in split order
__global__ void zmma_splitk_reduce(int64_t M, int64_t N, int S, const double2* __restrict__ partial, double2 alpha,
                                   double2 beta, double2* __restrict__ C, int64_t ldc) {
  pdl_wait();
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, tot = M * N;
  if (idx >= tot) return;
  double2 v = partial[idx];
  for (int z = 1; z < S; ++z) {
    const double2 p = partial[int64_t(z) * tot + idx];
    v.x += p.x;
    v.y += p.y;
  }
  const int64_t gn = idx / M, gm = idx - gn * M;
  store_c(C + gm + gn * ldc, v, alpha, beta);
}

struct Args {
  bool ka, kb;       // k-contiguous operands
  double sa, sb;     // -1: conjugated
  int64_t m, n, k;
  double2 alpha, beta;
  const void* A;
  int64_t lda;
  const void* B;
  int64_t ldb;
  double2* C;
  int64_t ldc;
};

template <int BM, int BN, int WGM, int WGN, int KW, class EA, class EB, bool AK, bool BK_>
void launch_cfg(Ctx& c, const Args& a, int S, int cs) {
  using GE = Geo<BM, BN, WGM, WGN, KW, EA, EB, AK, BK_>;
  auto kern = zmma_gemm_kernel<BM, BN, WGM, WGN, KW, EA, EB, AK, BK_>;
  static SmemAttrOnce attr;
  attr.ensure(kern, int(GE::smem));
  const int64_t gx = (a.m + BM - 1) / BM, gy = (a.n + BN - 1) / BN;
  IPEPS_CHECK(gy <= kMaxGridY, "gemm: n too large for grid");
  int64_t kchunk = (a.k + S - 1) / S;
  kchunk = ((kchunk + kBK - 1) / kBK) * kBK;
  const int cz = S / cs;
  double2* partial = nullptr;
  if (cz > 1) partial = static_cast<double2*>(c.workspace(size_t(cz) * a.m * a.n * sizeof(double2)));
  launch_clusters(c.stream, kern, dim3(unsigned(gx), unsigned(gy), unsigned(S)), GE::NT, GE::smem,
                  dim3(1, 1, unsigned(cs)), a.m, a.n, a.k, kchunk, a.alpha, static_cast<const EA*>(a.A), a.lda, a.sa,
                  static_cast<const EB*>(a.B), a.ldb, a.sb, a.beta, a.C, a.ldc, partial, cs);
  if (cz > 1) {
    const int64_t tot = a.m * a.n;
    launch(c.stream, zmma_splitk_reduce, unsigned((tot + 255) / 256), 256, 0, a.m, a.n, cz, partial, a.alpha, a.beta,
           a.C, a.ldc);
    IPEPS_LAUNCH_CHECK();
    c.count(KFam::Reduce, 0, double(cz + 2) * tot * sizeof(double2));
  }
}

template <int BM, int BN, int WGM, int WGN, int KW, class EA, class EB>
void launch_ops(Ctx& c, const Args& a, int S, int cs) {
  if (a.ka && a.kb) launch_cfg<BM, BN, WGM, WGN, KW, EA, EB, true, true>(c, a, S, cs);
  else if (a.ka) launch_cfg<BM, BN, WGM, WGN, KW, EA, EB, true, false>(c, a, S, cs);
  else if (a.kb) launch_cfg<BM, BN, WGM, WGN, KW, EA, EB, false, true>(c, a, S, cs);
  else launch_cfg<BM, BN, WGM, WGN, KW, EA, EB, false, false>(c, a, S, cs);
}

template <int BM, int BN, int WGM, int WGN, int KW, class EA, class EB>
int resident_cfg(int cs) {
  using GE = Geo<BM, BN, WGM, WGN, KW, EA, EB, true, true>;
  auto kern = zmma_gemm_kernel<BM, BN, WGM, WGN, KW, EA, EB, true, true>;
  static SmemAttrOnce attr;
  attr.ensure(kern, int(GE::smem));
  return resident(kern, GE::NT, GE::smem, cs);
}

// Per pair of operand types: 16 x 32 tiles (one warp per 4 of the 16 k) for small outputs
// (66 x 66 x 128: 6.6 us, 32 x 32: 8.5) and 32 x 32 (20736 x 18 x 9: 9.5 us, 16 x 32:
// 12.5); 64 x 64 was behind at every size of the engine (1600 x 80 x 1600: 101 us, 77
// with 32 x 32).  pipe and step as in gemm_dmma.cu, times the DMMAs per product (4, with a
// real operand 2).
struct Config {
  int bm, bn;
  double pipe, step;
  void (*launch)(Ctx&, const Args&, int, int);
  int (*resident)(int);
};
#define IPEPS_ZMMA_CONFIGS(EA, EB, W)                                                                                \
  {                                                                                                                  \
    {16, 32, 512 * W / (4 * .75), 350 + 130 * W, launch_ops<16, 32, 1, 1, 4, EA, EB>,                                 \
     resident_cfg<16, 32, 1, 1, 4, EA, EB>},                                                                         \
        {32, 32, 1024 * W / (4 * .80), 350 + 260 * W, launch_ops<32, 32, 2, 1, 2, EA, EB>,                            \
         resident_cfg<32, 32, 2, 1, 2, EA, EB>},                                                                     \
  }
constexpr int kNumConfigs = 2;
const Config kConfigs[3][kNumConfigs] = {IPEPS_ZMMA_CONFIGS(double2, double2, 4), IPEPS_ZMMA_CONFIGS(double2, double, 2),
                                         IPEPS_ZMMA_CONFIGS(double, double2, 2)};
#undef IPEPS_ZMMA_CONFIGS

struct Residency {
  std::once_flag once;
  int n[3][kNumConfigs][kMaxCluster + 1] = {};
};
const Residency& residency(int device) {
  static Residency r[SmemAttrOnce::kMaxDevices];
  Residency& q = r[device % SmemAttrOnce::kMaxDevices];
  std::call_once(q.once, [&] {
    for (int t = 0; t < 3; ++t)
      for (int f = 0; f < kNumConfigs; ++f)
        for (int cs = 1; cs <= kMaxCluster; ++cs) q.n[t][f][cs] = std::max(1, kConfigs[t][f].resident(cs));
  });
  return q;
}

}  // namespace

void gemm_c128_dmma(Ctx& c, char opA, DType dtA, char opB, DType dtB, int64_t m, int64_t n, int64_t k,
                    cuDoubleComplex alpha, const void* A, int64_t lda, const void* B, int64_t ldb, cuDoubleComplex beta,
                    void* C, int64_t ldc) {
  if (m <= 0 || n <= 0) return;
  IPEPS_CHECK(k > 0, "gemm: k == 0 is not supported");
  auto op = [](char o) {
    if (o == 'N' || o == 'n') return 0;
    if (o == 'T' || o == 't') return 1;
    if (o == 'C' || o == 'c') return 2;
    throw Error(kEInval, "gemm: bad op");
  };
  const int oa = op(opA), ob = op(opB);
  if (n > kMaxColumns) {
    for (int64_t j = 0; j < n; j += kMaxColumns)
      gemm_c128_dmma(c, opA, dtA, opB, dtB, m, std::min(kMaxColumns, n - j), k, alpha, A, lda,
                     static_cast<const char*>(B) + (ob ? j : j * ldb) * int64_t(dtype_size(dtB)), ldb, beta,
                     static_cast<double2*>(C) + j * ldc, ldc);
    return;
  }
  const int type = dtA == DType::F64 ? 2 : dtB == DType::F64 ? 1 : 0;
  IPEPS_CHECK(dtA == DType::C128 || dtB == DType::C128, "gemm: a complex operand is needed");
  ProfScope ps(c, KFam::GemmF64);
  Args a{oa != 0, ob == 0, oa == 2 ? -1.0 : 1.0, ob == 2 ? -1.0 : 1.0, m, n, k, alpha, beta, A, lda, B, ldb,
         static_cast<double2*>(C), ldc};
  const auto key = std::make_tuple(m, n, k, 1 + type);
  auto it = c.gemm_plans.find(key);
  if (it == c.gemm_plans.end()) {
    const Residency& res = residency(c.device);
    const Ctx::GemmPlan p = best_split(kConfigs[type], kNumConfigs, [&](int f, int cs) { return res.n[type][f][cs]; },
                                       c.sm_count, m, n, k, 16, false);
    if (c.gemm_plans.size() >= 4096) c.gemm_plans.clear();
    it = c.gemm_plans.emplace(key, p).first;
  }
  kConfigs[type][it->second.config].launch(c, a, it->second.S, it->second.cs);
  c.count(KFam::GemmF64, (type == 0 ? 8.0 : 4.0) * double(m) * double(n) * double(k));
}

}  // namespace ipeps
