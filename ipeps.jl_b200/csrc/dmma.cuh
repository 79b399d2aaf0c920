// Shared-memory tiles, their asynchronous copies and the split-K cost model of the
// FP64 tensor-core GEMMs (gemm_dmma.cu: real, gemm_zmma.cu: complex128).
#pragma once
#include "ctx.cuh"

#include <algorithm>
#include <cmath>

namespace ipeps {

constexpr int kBK = 16;
constexpr int kStages = 3;

__device__ __forceinline__ int64_t imin(int64_t a, int64_t b) { return a < b ? a : b; }
__device__ __forceinline__ int64_t imax(int64_t a, int64_t b) { return a > b ? a : b; }

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src, int bytes) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if constexpr (BYTES == 16) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes));
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

// Shared-memory geometry of one operand tile of E = double or double2 (BMN rows of
// the m or n index).  Each operand keeps its global contiguity: k-contiguous ones as
// [mn][16 + 4], mn-contiguous ones as [16][BMN + pad]; the paddings make a warp's
// fragment loads (8 rows x 4 columns) conflict-free.
template <class E, int BMN, bool KMAJ>
struct Tile {
  static constexpr int ld = KMAJ ? kBK + 4 : BMN + (sizeof(E) == 8 ? 4 : 2);  // elements per stored row
  static constexpr int size = KMAJ ? BMN * ld : kBK * ld;                     // elements per stage
  // element (mn, k) of the tile
  static __device__ __forceinline__ int at(int mn, int k) { return KMAJ ? mn * ld + k : k * ld + mn; }
};

// Copies operand tiles [mn0, mn0 + BMN) x [k0, k0 + 16) of successive k0 into shared
// memory, VEC elements per copy, zero-filled out of range.  Global layout: KMAJ:
// element (mn, k) at P[k + mn * ld]; else at P[mn + k * ld].  A thread's copies of a
// tile lie a fixed number of rows apart and move with k by one pointer (their
// addresses formed one by one cost the issue slots of ~10% of the large products);
// where the rows do not divide evenly over the threads they are formed one by one.
template <class E, int BMN, bool KMAJ, int VEC, int NT>
struct Loader {
  using T = Tile<E, BMN, KMAJ>;
  static constexpr int inner = (KMAJ ? kBK : BMN) / VEC, outer = KMAJ ? BMN : kBK;
  static constexpr bool regular = NT % inner == 0;
  static constexpr int step = regular ? NT / inner : 1;  // rows between a thread's copies
  const E* P;
  const E* p;
  int64_t ldp, MN, mn0;
  int i, o, mn_left;
  __device__ __forceinline__ Loader(const E* P_, int64_t ld, int64_t MN_, int64_t mn0_, int64_t k0, int tid)
      : P(P_), ldp(ld), MN(MN_), mn0(mn0_) {
    i = (tid % inner) * VEC;
    o = tid / inner;
    mn_left = int(imin(MN - mn0, BMN));
    p = KMAJ ? P + (k0 + i) + (mn0 + o) * ldp : P + (mn0 + i) + (k0 + o) * ldp;
  }
  // tile at k0 (its k's below ke) into s; then on to the next 16 k
  __device__ __forceinline__ void next(E* s, int64_t k0, int64_t ke, int tid) {
    constexpr int B = VEC * int(sizeof(E));
    if constexpr (!regular) {
      constexpr int chunks = inner * outer;
#pragma unroll
      for (int r = 0; r < (chunks + NT - 1) / NT; ++r) {
        const int e = tid + r * NT;
        if (chunks % NT != 0 && e >= chunks) break;
        const int ii = (e % inner) * VEC, oo = e / inner;
        const int mn = KMAJ ? oo : ii, k = KMAJ ? ii : oo;
        const int64_t gmn = mn0 + mn, gk = k0 + k;
        const int64_t valid = KMAJ ? (gmn < MN ? imin(VEC, imax(0, ke - gk)) : 0)
                                   : (gk < ke ? imin(VEC, imax(0, MN - gmn)) : 0);
        const E* src = KMAJ ? P + gk + gmn * ldp : P + gmn + gk * ldp;
        cp_async<B>(s + T::at(mn, k), valid ? src : P, int(valid) * int(sizeof(E)));
      }
    } else {
      const int k_left = int(imin(ke - k0, kBK));
      const int in_left = (KMAJ ? k_left : mn_left) - i, out_left = KMAJ ? mn_left : k_left;
      const int bytes = int(sizeof(E)) * max(0, min(VEC, in_left));
      E* d = s + (KMAJ ? T::at(o, i) : T::at(i, o));
#pragma unroll
      for (int r = 0; r < (outer + step - 1) / step; ++r) {
        const int row = o + r * step;
        if (outer % step != 0 && row >= outer) break;
        const int n = row < out_left ? bytes : 0;
        cp_async<B>(d + r * step * T::ld, n ? p + int64_t(r * step) * ldp : P, n);
      }
      p += KMAJ ? int64_t(kBK) : kBK * ldp;
    }
  }
};

// Tiles that the grid's y side (the columns) holds, and the columns of one launch: wider
// outputs are formed in panels of as many (2.1 million at the narrowest tiles, and a
// multiple of 32, so that operands keep their alignment).  The alternative, the column tiles
// along x in such cases, costs every launch of many small tiles (8 x 1000000 x 4:
// 106.4 -> 108.5 us).
constexpr int64_t kMaxGridY = 65535;
constexpr int64_t kMaxColumns = 32 * kMaxGridY;

constexpr int kMaxCluster = 8;

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

// Estimated cycles of a product on tiles of bm x bn with S K chunks in clusters of
// cs: waves of CTAs, each as long as its steps take on the fullest SM.  pipe: cycles
// of a K step of one CTA on the FP64 pipe of its SM, step: cycles one CTA alone
// needs for it, slots: resident CTAs.  The constants are fitted to a sweep of all real
// configurations and splits over 151 shapes (D = 2 to 5, chi = 9 to 100): the choice
// is 2.3% slower than the best of the sweep on average.
inline double split_cost(int bm, int bn, double pipe, double step, int64_t m, int64_t n, int64_t k, int elem_bytes,
                         bool upper, int sms, int slots, int S, int cs) {
  const double gx = double((m + bm - 1) / bm), gy = double((n + bn - 1) / bn);
  const double tiles = upper ? 0.5 * gx * gy + 0.5 * std::max(gx, gy) : gx * gy;
  const double steps = std::ceil(std::ceil(double(k) / kBK) / S), ctas = tiles * S;
  const double waves = std::floor(ctas / slots), rest = ctas - waves * slots;
  const double full = std::max(1.0, double(slots) / sms);
  // a cluster's CTAs share SMs sooner than the same number of single ones
  const double part = std::min(full, std::ceil(rest / sms) * (cs > 1 ? 1.0 + 0.025 * (cs - 1) : 1.0));
  const double w = elem_bytes / 8.0;
  double t = waves * (steps * std::max(full * pipe, step) + 4100.0);
  if (rest > 0) t += steps * std::max(part * pipe, step) + 4100.0;
  if (cs > 1) t = t * (cs > 2 && waves >= 1 ? 1.04 : 1.0) + (waves + 1) * (1300.0 + 0.43 * w * bm * bn);
  if (S > cs) t += 7000.0 + (S / cs) * (106.0 + w * double(m) * double(n) * 16.0 / 9400.0);
  return t;
}

// Best (configuration, S, cs) over the configurations cfg[i] (fields bm, bn, pipe,
// step), slots(i, cs) CTAs resident; clusters of 3, 5, 6, 7 measured behind those of
// 2, 4, 8, and at most 400 MB of partial sums.
template <class Cfg, class Slots>
Ctx::GemmPlan best_split(const Cfg* cfg, int n_cfg, const Slots& slots, int sms, int64_t m, int64_t n, int64_t k,
                         int elem_bytes, bool upper) {
  Ctx::GemmPlan best;
  double t = -1.0;
  for (int f = 0; f < n_cfg; ++f)
    for (int S = 1; S <= 1024; S = S < 8 ? S + 1 : 2 * S) {
      if (S > 1 && int64_t(S) * 2 * kBK > k) break;
      for (int cs : {std::min(S, kMaxCluster), 1}) {
        if ((cs & (cs - 1)) != 0) continue;
        if (cs == 1 && S > 1 && double(S) * double(m) * double(n) * elem_bytes > 4e8) break;
        const double e = split_cost(cfg[f].bm, cfg[f].bn, cfg[f].pipe, cfg[f].step, m, n, k, elem_bytes, upper, sms,
                                    slots(f, cs), S, cs);
        if (t < 0 || e < t) {
          best = {f, S, cs};
          t = e;
        }
      }
    }
  return best;
}

}  // namespace ipeps
