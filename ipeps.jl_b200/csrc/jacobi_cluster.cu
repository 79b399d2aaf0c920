// One-sided Jacobi SVD of the projector's k x k Rayleigh-Ritz matrix on a
// thread-block cluster of 8 CTAs (8 SMs) instead of one CTA.
//
// The columns of [X; J] (J starts as the identity and accumulates the
// rotations, so no separate pass forms it) are cut into 16 blocks of b
// columns; each CTA holds two blocks in shared memory.  A sweep is the
// block round robin of 15 rounds (the circle method over 16 block
// positions): in round 0 each CTA also orthogonalises the column pairs
// inside its two blocks, and in every round all b x b pairs between its two
// blocks, b disjoint pairs at a time (one warp per pair; the first block's
// column stays in the warp's registers for the whole round).  Between rounds
// every CTA writes its two blocks into the shared memory of the CTAs that
// hold those block positions next (distributed shared memory, double
// buffered), and the cluster barrier orders the exchange.  Every pair of
// columns meets exactly once per sweep, as in the cyclic Jacobi method.  The
// sweep loop ends when no CTA rotated (an all-to-all flag exchange) or at
// max_sweeps (status bit 4).  The rotation (angle from rsqrt only, as the
// single-CTA kernel) and the threshold |x_p.x_q| > tol |x_p| |x_q| are those
// of the single-CTA kernel, so the result is the same SVD up to rounding.
#include "linalg.cuh"

#include <cooperative_groups.h>

namespace ipeps {
namespace {

namespace cg = cooperative_groups;

constexpr int kJP = 8;                 // CTAs per cluster (portable cluster size; 16: 508 us instead of 556 at k = 160,
                                       // slower below k = 128)
constexpr int kJBlocks = 2 * kJP;      // column blocks
constexpr int kJWarps = 16;            // warps per CTA (>= b)
constexpr int kJMaxRowsPerLane = 16;   // height of [X; J] <= 512
constexpr size_t kJSmemMax = 200 * 1024;

struct JcArgs {
  const void* X;
  int64_t ldx;
  int m, k, b;  // rows of X, columns, block width
  int max_sweeps;
  double tol2;
  void* Xout;
  void* J;
  int64_t ldj;
  double* S;
  int* status;
  int* sweeps_out;
};

// circle-method pair w of round t among n (even) players
__device__ __forceinline__ void circle_pair(int w, int t, int n, int& p, int& q) {
  const int n1 = n - 1;
  int a = w - 1 + t;
  a %= n1;
  int c = n - 2 - w + t;
  c %= n1;
  p = (w == 0) ? 0 : 1 + a;
  q = 1 + c;
}

// position p of the block round robin -> (cluster rank, slot)
__device__ __forceinline__ void pos_owner(int p, int& rank, int& slot) {
  if (p < kJP) {
    rank = p;
    slot = 0;
  } else {
    rank = kJBlocks - 1 - p;
    slot = 1;
  }
}

// 1 / sqrt(h) of h > 0, subnormal ones too: the columns of a rank-deficient X shrink
// by the rounding level with every sweep, until their squared norms underflow.
__device__ __forceinline__ double rsqrt_pos(double h) { return h >= 1e-300 ? rsqrt_normal(h) : rsqrt(h); }

// Rotates column u (registers, squared norm nu) against the shared column y
// (squared norm *ny); true when it rotated.  The dot product runs over the rows of
// X only (nx of the NR rows per lane), the rotation over those of [X; J].
template <int NR>
__device__ __forceinline__ bool rotate_pair(double (&u)[NR], double& nu, double* y, double* ny, int m, int nx, int H,
                                            int lane, double tol2) {
  double v[NR];
  double c0 = 0, c1 = 0;
  const double nv = *ny;
#pragma unroll
  for (int j = 0; j < NR; ++j) v[j] = y[lane + 32 * j];
#pragma unroll
  for (int j = 0; j < NR; ++j)
    if (j < nx) {
      const double w = lane + 32 * j < m ? v[j] : 0.0;
      if (j & 1) c1 = fma(u[j], w, c1);
      else c0 = fma(u[j], w, c0);
    }
  double c = c0 + c1;
#pragma unroll
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (!(c != 0.0 && nu > 0.0 && nv > 0.0 && c * c > tol2 * (nu * nv))) return false;
  const double d = nv - nu;
  const double rho = rsqrt_pos(fma(d, d, 4.0 * c * c));
  const double c2 = fabs(d) * rho, s2 = copysign(1.0, d) * (2.0 * c * rho);
  const double uu = 0.5 * (1.0 + c2);
  const double ru = rsqrt_normal(uu);
  const double cs = uu * ru, sn = 0.5 * s2 * ru;
#pragma unroll
  for (int j = 0; j < NR; ++j) {
    const double up = cs * u[j] - sn * v[j], vq = sn * u[j] + cs * v[j];
    u[j] = up;
    y[lane + 32 * j] = vq;
  }
  const double tc = 0.5 * s2 * c * (ru * ru);  // tan(t) * c
  nu -= tc;
  if (lane == 0) *ny = nv + tc;
  return true;
}

// The complex pair: c = u^H y = |c| e^{i phi} is rotated as the real pair (u,
// e^{-i phi} y); the transform of the columns is unitary.
template <int NR>
__device__ __forceinline__ bool rotate_pair(double2 (&u)[NR], double& nu, double2* y, double* ny, int m, int nx, int H,
                                            int lane, double tol2) {
  double2 v[NR];
  double cr = 0, ci = 0;
  const double nv = *ny;
#pragma unroll
  for (int j = 0; j < NR; ++j) v[j] = y[lane + 32 * j];
#pragma unroll
  for (int j = 0; j < NR; ++j)
    if (j < nx) {
      const double2 w = lane + 32 * j < m ? v[j] : make_double2(0.0, 0.0);
      cr = fma(u[j].x, w.x, fma(u[j].y, w.y, cr));
      ci = fma(u[j].x, w.y, fma(-u[j].y, w.x, ci));
    }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    cr += __shfl_xor_sync(0xffffffffu, cr, o);
    ci += __shfl_xor_sync(0xffffffffu, ci, o);
  }
  const double mag2 = fma(cr, cr, ci * ci);
  // (an underflowing |c|^2 has no usable phase: null columns of a rank-deficient X are left as they are; X is
  // scaled, so the threshold is relative to its largest entry)
  if (!(mag2 >= 1e-300 && nu > 0.0 && nv > 0.0 && mag2 > tol2 * (nu * nv))) return false;
  const double im = rsqrt_normal(mag2), mag = mag2 * im;
  const double ex = cr * im, ey = -ci * im;        // e^{-i phi}
  const double d = nv - nu;
  const double rho = rsqrt_normal(fma(d, d, 4.0 * mag2));  // >= 4 |c|^2
  const double c2 = fabs(d) * rho, s2 = copysign(1.0, d) * (2.0 * mag * rho);
  const double uu = 0.5 * (1.0 + c2);
  const double ru = rsqrt_normal(uu);
  const double cs = uu * ru, sn = 0.5 * s2 * ru;
#pragma unroll
  for (int j = 0; j < NR; ++j) {
    const double2 w = make_double2(ex * v[j].x - ey * v[j].y, ex * v[j].y + ey * v[j].x);
    const double2 p = u[j];
    u[j] = make_double2(cs * p.x - sn * w.x, cs * p.y - sn * w.y);
    y[lane + 32 * j] = make_double2(sn * p.x + cs * w.x, sn * p.y + cs * w.y);
  }
  const double tc = 0.5 * s2 * mag * (ru * ru);
  nu -= tc;
  if (lane == 0) *ny = nv + tc;
  return true;
}

__device__ __forceinline__ double norm2_of(double x) { return x * x; }
__device__ __forceinline__ double norm2_of(double2 x) { return fma(x.x, x.x, x.y * x.y); }
__device__ __forceinline__ void set_real(double& x, double r) { x = r; }
__device__ __forceinline__ void set_real(double2& x, double r) { x = make_double2(r, 0.0); }
// x 2^e (real columns are not scaled)
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ double scaled(double x, int) { return x; }
__device__ __forceinline__ double2 scaled(double2 x, int e) { return make_double2(x.x * pow2(e), x.y * pow2(e)); }

template <class T, int NR>
__device__ __forceinline__ void load_col(T (&u)[NR], const T* x, int lane) {
#pragma unroll
  for (int j = 0; j < NR; ++j) u[j] = x[lane + 32 * j];
}

template <class T, int NR>
__device__ __forceinline__ void store_col(const T (&u)[NR], T* x, int lane) {
#pragma unroll
  for (int j = 0; j < NR; ++j) x[lane + 32 * j] = u[j];
}

// Exponent by which a complex X is scaled down while it is rotated: that of its largest
// component (`mx`, this CTA's, of all CTAs through `all` in their shared memory), where
// that lies beyond 2^+-100 = 1e+-30: the rotations work with fourth powers of the
// entries, and columns of 1e-13 of the largest are resolved to rounding.  A power of
// two, so nothing is rounded.  All CTAs of the cluster must have started.
constexpr int kJScaleExp = 100;
__device__ int scale_exponent(double mx, double* all, double* red) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  if (threadIdx.x < kJP) {
    for (int w = 0; w < kJWarps; ++w) mx = fmax(mx, red[w]);
    *cluster.map_shared_rank(all + cluster.block_rank(), threadIdx.x) = mx;
  }
  cluster.sync();
  mx = 0.0;
  for (int r = 0; r < kJP; ++r) mx = fmax(mx, all[r]);
  if (!(mx > 0.0) || isinf(mx)) return 0;
  const int e = ilogb(mx);
  return e < -kJScaleExp || e > kJScaleExp ? max(-1022, min(1022, e)) : 0;
}

// NR: rows of [X; J] per lane, H = 32 NR.  Bound by the latency of a sub-round (load,
// dot product, reduction, angle, store, barrier: ~0.8 us at k = 160) and of the
// exchange between rounds (~1.1 us).  A pair costs 5 NR / 2 FP64 instructions per
// lane: the dot product runs over the rows of X, the squared norms are carried
// (recomputed every sweep) and exchanged with the blocks.  Four sweeps, before (16
// rows per lane whatever the size, norms from every pair, even block widths) -> now:
// k = 62 244 -> 128 us, k = 98 587 -> 288, k = 128 588 -> 336, k = 160 888 -> 556.
template <class T, int NR>
__global__ void __cluster_dims__(kJP, 1, 1) __launch_bounds__(kJWarps * 32, 1) jacobi_cluster_kernel(JcArgs a) {
  pdl_wait();
  extern __shared__ __align__(16) double jsm[];
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int H = 32 * NR;
  constexpr bool CX = sizeof(T) == 16;
  const int rank = int(cluster.block_rank());
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = a.b, m = a.m, nx = (a.m + 31) >> 5;
  // a slot: b columns of H rows, then their squared norms
  const int be = (b + 1) & ~1;  // players of the round robin inside a block (b odd: one sits out)
  const size_t cols = size_t(b) * H, slot_sz = cols * (sizeof(T) / 8) + be;  // (T's, doubles)
  const T* X = static_cast<const T*>(a.X);
  T *Xout = static_cast<T*>(a.Xout), *J = static_cast<T*>(a.J);
  // buf[cur][slot] columns, then the block ids of the slots per buffer, then the flags
  double* buf = jsm;
  int* blk = reinterpret_cast<int*>(jsm + 4 * slot_sz);  // [2 buffers][2 slots]
  int* flags = blk + 4;                                   // [kJP]
  double* xmax = jsm + 4 * slot_sz + 16;                  // [kJP]
  __shared__ int s_rot;
  __shared__ double red[kJWarps];

  int cur = 0;
  if (tid < 2) blk[tid] = (tid == 0) ? rank : kJBlocks - 1 - rank;
  __syncthreads();
  // load [X; I] columns of both blocks (columns >= k are zero)
  double mx = 0.0;
  for (int s = 0; s < 2; ++s) {
    T* dst = reinterpret_cast<T*>(buf + (0 * 2 + s) * slot_sz);
    const int b0 = blk[s] * b;
    for (int j = warp; j < b; j += kJWarps) {
      const int col = b0 + j;
      for (int r = lane; r < H; r += 32) {
        T v;
        set_real(v, r - m == col ? 1.0 : 0.0);
        if (r < m && col < a.k) v = X[r + int64_t(col) * a.ldx];
        if (col >= a.k) set_real(v, 0.0);
        dst[j * H + r] = v;
        if constexpr (CX)
          if (r < m) mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
      }
    }
  }
  cluster.sync();
  int ex = 0;  // X is rotated as X 2^-ex
  if constexpr (CX) {
    ex = scale_exponent(mx, xmax, red);
    if (ex != 0) {
      for (int s = 0; s < 2; ++s)
        for (int j = warp; j < b; j += kJWarps)
          for (int r = lane; r < m; r += 32) {
            T* x = reinterpret_cast<T*>(buf + s * slot_sz) + j * H + r;
            *x = scaled(*x, -ex);
          }
      __syncthreads();
    }
  }

  int sweep = 0;
  bool converged = false;
  for (; sweep < a.max_sweeps && !converged; ++sweep) {
    if (tid == 0) s_rot = 0;
    for (int j = warp; j < 2 * b; j += kJWarps) {
      double* S = buf + (cur * 2 + (j >= b)) * slot_sz;
      const int jj = j >= b ? j - b : j;
      double n = 0;
      for (int r = lane; r < m; r += 32) n += norm2_of(reinterpret_cast<const T*>(S)[jj * H + r]);
#pragma unroll
      for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
      if (lane == 0) S[cols * (sizeof(T) / 8) + jj] = n;
    }
    __syncthreads();
    bool rot = false;
    for (int round = 0; round < kJBlocks - 1; ++round) {
      T* A = reinterpret_cast<T*>(buf + (cur * 2 + 0) * slot_sz);
      T* B = reinterpret_cast<T*>(buf + (cur * 2 + 1) * slot_sz);
      double *nA = reinterpret_cast<double*>(A + cols), *nB = reinterpret_cast<double*>(B + cols);
      if (round == 0) {
        // pairs inside each block: be - 1 sub-rounds of be/2 pairs per block
        for (int t = 0; t < be - 1; ++t) {
          for (int w = warp; w < be; w += kJWarps) {
            T* base = (w < be / 2) ? A : B;
            double* nb = (w < be / 2) ? nA : nB;
            int p, q;
            circle_pair(w % (be / 2), t, be, p, q);
            if (p >= b || q >= b) continue;
            T u[NR];
            double nu = nb[p];
            load_col<T, NR>(u, base + size_t(p) * H, lane);
            if (rotate_pair<NR>(u, nu, base + size_t(q) * H, nb + q, m, nx, H, lane, a.tol2)) {
              store_col<T, NR>(u, base + size_t(p) * H, lane);
              if (lane == 0) nb[p] = nu;
              rot = true;
            }
          }
          __syncthreads();
        }
      }
      // pairs between the two blocks: warp i keeps column A_i, meets B_{(i+t) % b}
      if (warp < b) {
        T u[NR];
        double nu = nA[warp];
        load_col<T, NR>(u, A + size_t(warp) * H, lane);
        bool any = false;
        int q = warp;
        for (int t = 0; t < b; ++t) {
          // B columns are touched by one warp per sub-round: sync the warps that share them
          if (rotate_pair<NR>(u, nu, B + size_t(q) * H, nB + q, m, nx, H, lane, a.tol2)) any = true;
          q = q + 1 == b ? 0 : q + 1;
          asm volatile("bar.sync 1, %0;" ::"r"(b * 32) : "memory");
        }
        if (any) {
          store_col<T, NR>(u, A + size_t(warp) * H, lane);
          if (lane == 0) nA[warp] = nu;
          rot = true;
        }
      }
      __syncthreads();
      // hand both blocks to the CTAs that hold their next positions
      const int nxt = cur ^ 1;
      for (int s = 0; s < 2; ++s) {
        const int pos = (s == 0) ? rank : kJBlocks - 1 - rank;
        const int np = (pos == 0) ? 0 : (pos == kJBlocks - 1 ? 1 : pos + 1);
        int drank, dslot;
        pos_owner(np, drank, dslot);
        const double2* src = reinterpret_cast<const double2*>(buf + (cur * 2 + s) * slot_sz);
        double2* dst =
            reinterpret_cast<double2*>(cluster.map_shared_rank(buf + (nxt * 2 + dslot) * slot_sz, drank));
        for (int e = tid; e < int(slot_sz / 2); e += kJWarps * 32) dst[e] = src[e];
        if (tid == 0) *cluster.map_shared_rank(blk + nxt * 2 + dslot, drank) = blk[cur * 2 + s];
      }
      cluster.sync();
      cur = nxt;
    }
    // did any CTA rotate in this sweep?
    if (rot) s_rot = 1;
    __syncthreads();
    if (tid < kJP) *cluster.map_shared_rank(flags + rank, tid) = s_rot;
    cluster.sync();
    int any = 0;
    for (int r = 0; r < kJP; ++r) any |= flags[r];
    converged = (any == 0);
    cluster.sync();  // flags are rewritten only after every CTA has read them
  }

  // write back W = X J columns, J, and the column norms of W
  for (int s = 0; s < 2; ++s) {
    const T* src = reinterpret_cast<const T*>(buf + (cur * 2 + s) * slot_sz);
    const int b0 = blk[cur * 2 + s] * b;
    for (int j = warp; j < b; j += kJWarps) {
      const int col = b0 + j;
      if (col >= a.k) continue;
      double nn = 0;
      for (int r = lane; r < H; r += 32) {
        const T v = src[j * H + r];
        if (r < m) {
          Xout[r + int64_t(col) * a.ldx] = scaled(v, ex);
          nn += norm2_of(v);
        } else if (r - m < a.k) {
          J[(r - m) + int64_t(col) * a.ldj] = v;
        }
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
      if (lane == 0) a.S[col] = CX ? sqrt(nn) * pow2(ex) : sqrt(nn);
    }
  }
  if (rank == 0 && tid == 0) {
    if (!converged) atomicOr(a.status, 4);
    *a.sweeps_out = sweep;
  }
  cluster.sync();
}

template <class T, int NR>
void launch_cluster(Ctx& c, const JcArgs& a, size_t smem) {
  static SmemAttrOnce attr;
  attr.ensure(jacobi_cluster_kernel<T, NR>, int(kJSmemMax));
  launch(c.stream, jacobi_cluster_kernel<T, NR>, kJP, kJWarps * 32, smem, a);
  IPEPS_LAUNCH_CHECK();
}

// rows of [X; J] per lane, rounded up to the next instance
int rows_per_lane(int m, int k) {
  const int n = (m + k + 31) / 32;
  return n <= 8 ? n : (n + 1) & ~1;
}
int block_width(int k) { return (k + kJBlocks - 1) / kJBlocks; }
size_t cluster_smem(int b, int nr, int words) { return (size_t(4) * (b * 32 * nr * words + ((b + 1) & ~1)) + 64) * 8; }

bool fits(int m, int k, int words, int max_rows) {
  if (m < 1 || k < 2) return false;
  const int b = block_width(k), nr = rows_per_lane(m, k);
  return b <= kJWarps && nr <= max_rows && cluster_smem(b, nr, words) <= kJSmemMax;
}

template <class T>
void svd_cluster(Ctx& c, void* X, int m, int k, int64_t ldx, void* J, int64_t ldj, double* S, int max_sweeps,
                 double tol, int* d_sweeps) {
  if (tol <= 0) tol = double(m) * 2.220446049250313e-16;
  JcArgs a{};
  a.X = X;
  a.ldx = ldx;
  a.m = m;
  a.k = k;
  a.b = block_width(k);
  a.max_sweeps = max_sweeps;
  a.tol2 = tol * tol;
  a.Xout = X;
  a.J = J;
  a.ldj = ldj;
  a.S = S;
  a.status = c.d_status;
  a.sweeps_out = d_sweeps;
  const int nr = rows_per_lane(m, k);
  const size_t smem = cluster_smem(a.b, nr, sizeof(T) / 8);
  ProfScope ps(c, KFam::Jacobi);
  switch (nr) {
    case 1: launch_cluster<T, 1>(c, a, smem); break;
    case 2: launch_cluster<T, 2>(c, a, smem); break;
    case 3: launch_cluster<T, 3>(c, a, smem); break;
    case 4: launch_cluster<T, 4>(c, a, smem); break;
    case 5: launch_cluster<T, 5>(c, a, smem); break;
    case 6: launch_cluster<T, 6>(c, a, smem); break;
    case 7: launch_cluster<T, 7>(c, a, smem); break;
    case 8: launch_cluster<T, 8>(c, a, smem); break;
    default:
      if constexpr (sizeof(T) == 8) {
        switch (nr) {
          case 10: launch_cluster<T, 10>(c, a, smem); break;
          case 12: launch_cluster<T, 12>(c, a, smem); break;
          case 14: launch_cluster<T, 14>(c, a, smem); break;
          default: launch_cluster<T, 16>(c, a, smem); break;
        }
      }
  }
  c.count(KFam::Jacobi, (sizeof(T) == 8 ? 6.0 : 24.0) * double(m + k) * k * k / 2.0);
}

}  // namespace

bool jacobi_cluster_fits(int m, int k) { return fits(m, k, 1, kJMaxRowsPerLane); }
bool jacobi_cluster_c_fits(int m, int k) { return fits(m, k, 2, 8); }

void jacobi_svd_cluster(Ctx& c, double* X, int m, int k, int64_t ldx, double* J, int64_t ldj, double* S,
                        int max_sweeps, double tol, int* d_sweeps) {
  IPEPS_CHECK(jacobi_cluster_fits(m, k), "jacobi_svd_cluster: problem does not fit");
  svd_cluster<double>(c, X, m, k, ldx, J, ldj, S, max_sweeps, tol, d_sweeps);
}

void jacobi_c_svd_cluster(Ctx& c, void* X, int m, int k, int64_t ldx, void* J, int64_t ldj, double* S, int max_sweeps,
                          double tol, int* d_sweeps) {
  IPEPS_CHECK(jacobi_cluster_c_fits(m, k), "jacobi_c_svd_cluster: problem does not fit");
  svd_cluster<double2>(c, X, m, k, ldx, J, ldj, S, max_sweeps, tol, d_sweeps);
}

}  // namespace ipeps
