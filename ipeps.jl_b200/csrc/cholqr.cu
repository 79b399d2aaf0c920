// Cholesky factor and triangular solve of one CholeskyQR pass for sketches of
// up to 192 columns: G = R^T R (shifted, guarded), then Q = Y R^-1.
//
// Both work on 8 x 8 blocks so that all but the 8 x 8 diagonal factors runs on
// the FP64 tensor pipe (mma.sync m8n8k4; tcgen05 has no FP64 kind).  R goes from
// the first kernel to the second in packed blocks, the diagonal ones already
// inverted.
//
// chol_panel is bound by latency: one CTA and k/8 dependent panel steps, of about
// 1650 cycles (0.85 us) each once the trailing updates fit beside them.  The kernel
// this one replaces eliminated column by column, ~900 cycles each for the pivot,
// the barrier and the broadcast loads.  Back-to-back launches at k = 62 / 128 / 160:
// 10.5 / 20.7 / 28.8 us (18.5 us at k = 62 and 74 us at k = 160 before).
// trsm_panel is bound by its dependent DMMA steps (one warp of eight rows per
// scheduler, 33 cycles per DMMA where the pipe takes one in 16): 6.3 us at
// N = 120, k = 62 and 13.1 us at N = 2500, k = 160 (10.7 and 27 us for the
// substitution by rows that it replaces).
// One CholeskyQR pass at N = 2500 without its Gram product, event-timed: 96.9 ->
// 58 us at k = 160, 71.1 -> 45 us at k = 128, 61.5 -> 39 us at k = 101.
// Complex sketches run on the same kernels as real ones of twice the width (66
// columns: one CTA with a barrier per column and a row per warp before; a pass
// without its Gram product ~200 -> ~35 us).
#include "linalg.cuh"

#include <algorithm>

namespace ipeps {
namespace {

// Warp w runs on scheduler w mod 4: warp 0 has scheduler 0 to itself (the FP64
// pipe of each scheduler takes a DMMA every 16 cycles, and the pivots' chain
// must not queue behind those); the update warps share the other three.
constexpr int kCpWarps = 16;
constexpr int kCpThreads = 32 * kCpWarps;
constexpr int kUpdateWarps = kCpWarps / 4 * 3;
constexpr int kUpdateThreads = 32 * kUpdateWarps;

__device__ __forceinline__ void dmma8(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}
// the same with the sum in another register pair
__device__ __forceinline__ void dmma8(double& d0, double& d1, double a, double b, double c0, double c1) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%5};\n"
      : "=d"(d0), "=d"(d1)
      : "d"(a), "d"(b), "d"(c0), "d"(c1));
}
template <int ID, int N>
__device__ __forceinline__ void bar_wait() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void bar_post() {
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}

// Packed upper block triangle of R, block row by block row: block (I, J) at
// col_base(I) + J - I.  Inside a block the entries (2t, g) and (2t + 1, g) are
// neighbours, at 2 (4 g + t): lane (g, t) of a warp then has with one 16-byte
// access what it needs of the block as the B operand of two m8n8k4 products
// over k = {2t} and k = {2t + 1}, and what an accumulator or an A operand
// holds of the transposed block.
__host__ __device__ __forceinline__ int col_base(int I, int nb) { return I * nb - I * (I - 1) / 2; }

// The matrix sits in shared memory in this layout, as the lower-triangle blocks
// (I, J) of L = R^T, I >= J; panel p:
//   warp 0 factors the diagonal block (every lane the whole of it, in registers,
//     without exchange) and inverts it (lane j column j), forms L_{p+1,p} and
//     brings the next diagonal block up to date, then goes on with it; barrier 1
//     tells the others that R_pp^-1 is there;
//   the update warps form L_Ip = C_Ip R_pp^-1 (barrier 3 among them) and subtract
//     L_Ip L_Jp^T from the blocks right of the panel, first from the two that
//     warp 0 reads next (barrier 2).
// So warp 0's chain never waits for the bulk of an update.  The loops are kept
// rolled: with the trailing blocks in registers (unrolled by slot) the SM spent
// its time fetching instructions (55 us at k = 160).
// The contract is that of chol_blocked: shift_factor * trace is added to the
// diagonal, a pivot at or below 1e-32 trace leaves R[j][j] = 1 and row j zero (inside the
// diagonal block by the pivot's factor 0, right of it by leaving its column out of the
// inverse in L_Ip = C_Ip R_pp^-1; `failed` has the panel's failed pivots as bits).
// In the end S holds the packed R; it is also written to Rpk if that is given, and R's
// diagonal blocks to G.
__device__ __forceinline__ void factor_panels(double2* S, int k, double shift_factor, double2* __restrict__ Rpk,
                                              double* G, int64_t ldg) {
  __shared__ int failed[kCholqrMax / 8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2;
  const int nb = (k + 7) >> 3;
  if (warp == 0) {
    double tr = 0;
    for (int i = lane; i < k; i += 32) {
      const double2 q = S[col_base(i >> 3, nb) * 32 + (i & 7) * 4 + ((i & 7) >> 1)];
      tr += fabs((i & 1) ? q.y : q.x);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    const double shift = shift_factor > 0 ? shift_factor * tr : 0.0;
    const double tiny = 1e-300 + 1e-32 * (tr + shift * k);
    const int me = lane & 7;
    for (int p = 0; p < nb; ++p) {
      double2* D = S + col_base(p, nb) * 32;
      double d[8][8], x[8];  // d[c][r], c <= r: entry (r, c) of the block; x: row `me` of the inverse
      int fail = 0;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
#pragma unroll
        for (int c = 0; c <= r; c += 2) {
          const double2 q = D[r * 4 + c / 2];
          d[c][r] = q.x;
          if (c < r) d[c + 1][r] = q.y;
        }
        d[r][r] += 8 * p + r < k ? shift : 0.0;
        x[r] = r == me ? 1.0 : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const double piv = d[j][j];
        const bool ok = piv > tiny || 8 * p + j >= k;
        fail |= int(!ok) << j;
        const double rt = rsqrt_normal(piv);  // (without rsqrt's cases the chain's shadow is filled)
        const double rs = __hiloint2double(ok ? __double2hiint(rt) : 0, ok ? __double2loint(rt) : 0);
        x[j] *= ok ? rs : 1.0;
        d[j][j] = ok ? piv * rs : 1.0;
#pragma unroll
        for (int l = j + 1; l < 8; ++l) d[j][l] *= rs;
#pragma unroll
        for (int i = j + 1; i < 8; ++i) {
#pragma unroll
          for (int l = i; l < 8; ++l) d[i][l] = fma(-d[j][i], d[j][l], d[i][l]);
          x[i] = fma(-d[j][i], x[j], x[i]);
        }
      }
      __syncwarp();
      if (lane < 8) {
        double* inv = reinterpret_cast<double*>(D) + me;
#pragma unroll
        for (int j = 0; j < 8; ++j) inv[8 * j] = x[j];
      }
      __syncwarp();
      const double2 q = D[lane];
      if (p + 1 < nb) {
        if (p > 0) bar_wait<2, 64>();
        const double2 c = D[32 + lane];
        double x0 = 0.0, x1 = 0.0;
        const bool out = fail >> g & 1;
        dmma8(x0, x1, c.x, out ? 0.0 : q.x);
        dmma8(x0, x1, c.y, out ? 0.0 : q.y);
        D[32 + lane] = make_double2(x0, x1);
        double2* N = S + col_base(p + 1, nb) * 32 + lane;
        double2 n = *N;
        dmma8(n.x, n.y, -x0, x0);
        dmma8(n.x, n.y, -x1, x1);
        *N = n;
        if (lane == 0) failed[p] = fail;
        __syncwarp();
        bar_post<1, 32 + kUpdateThreads>();
        if (Rpk) Rpk[(col_base(p, nb) + 1) * 32 + lane] = make_double2(x0, x1);
      }
      if (Rpk) Rpk[col_base(p, nb) * 32 + lane] = q;
      if (G && lane < 8) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c == me && 8 * p + c < k) {
#pragma unroll
            for (int r = 0; r <= c; ++r) G[8 * p + r + int64_t(8 * p + c) * ldg] = d[r][c];
          }
      }
    }
  } else if (warp & 3) {
    const int u = warp - 1 - (warp >> 2);
    for (int p = 0; p + 1 < nb; ++p) {
      double2* L = S + (col_base(p, nb) - p) * 32 + lane;  // L_Ip at L[32 I]
      bar_wait<1, 32 + kUpdateThreads>();
      double2 q = L[32 * p];
      if (failed[p] >> g & 1) q = make_double2(0.0, 0.0);
      for (int I = p + 2 + u; I < nb; I += kUpdateWarps) {
        const double2 c = L[32 * I];
        double x0 = 0.0, x1 = 0.0;
        dmma8(x0, x1, c.x, q.x);
        dmma8(x0, x1, c.y, q.y);
        L[32 * I] = make_double2(x0, x1);
        if (Rpk) Rpk[(col_base(p, nb) + I - p) * 32 + lane] = make_double2(x0, x1);
      }
      bar_wait<3, kUpdateThreads>();
      // the blocks right of the panel in 2 x 2 groups of rows I, I + 1 and columns J, J + 1
      // (each block of L read once for two products); group 0 holds what warp 0 reads next
      auto update = [&](int I, int J) {
        const bool i1 = I + 1 < nb, diag = I == J;
        const double2 a0 = L[32 * I], a1 = L[32 * (i1 ? I + 1 : I)];
        const double2 b0 = diag ? a0 : L[32 * J], b1 = diag ? a1 : L[32 * (J + 1)];
        double2* C0 = S + (col_base(J, nb) + I - J) * 32 + lane;      // (I, J), (I + 1, J)
        double2* C1 = S + (col_base(J + 1, nb) + I - J) * 32 + lane;  // (I + 1, J + 1) at 0, (I, J + 1) before it
        if (I > p + 1) {  // (p + 1, p + 1) is warp 0's
          double2 c = C0[0];
          dmma8(c.x, c.y, -a0.x, b0.x);
          dmma8(c.x, c.y, -a0.y, b0.y);
          C0[0] = c;
        }
        if (i1) {
          double2 c = C0[32], d = C1[0];
          dmma8(c.x, c.y, -a1.x, b0.x);
          dmma8(d.x, d.y, -a1.x, b1.x);
          dmma8(c.x, c.y, -a1.y, b0.y);
          dmma8(d.x, d.y, -a1.y, b1.y);
          C0[32] = c;
          C1[0] = d;
        }
        if (!diag) {
          double2 c = C1[-32];
          dmma8(c.x, c.y, -a0.x, b1.x);
          dmma8(c.x, c.y, -a0.y, b1.y);
          C1[-32] = c;
        }
      };
      if (u == 0 && p + 2 < nb) {
        update(p + 1, p + 1);
        bar_post<2, 64>();
      }
      // the other groups (i, j), j <= i, row by row, dealt to the warps in turn
      const int m = (nb - p) / 2;  // groups per side, over the rows p + 1 .. nb - 1
      int i = 1, j = u == 0 ? kUpdateWarps - 1 : u - 1;
      for (;;) {
        while (i < m && j > i) {
          j -= i + 1;
          ++i;
        }
        if (i >= m) break;
        update(p + 1 + 2 * i, p + 1 + 2 * j);
        j += kUpdateWarps;
      }
    }
  }
}

// CX: G is complex Hermitian of k / 2 columns, taken as the real symmetric matrix of
// its 2 x 2 blocks [[re, -im], [im, re]].  The factor of that is the same form of the
// complex factor (the Cholesky factor is unique), so the real kernels do the work.
template <bool CX>
__global__ void __launch_bounds__(kCpThreads, 1)
    chol_panel_kernel(double* G, int k, int64_t ldg, double shift_factor, double2* __restrict__ Rpk, int write_g) {
  pdl_wait();
  extern __shared__ __align__(16) double2 S[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nb = (k + 7) >> 3, nblk = nb * (nb + 1) / 2;

  // G's upper triangle (columns from k on: the identity)
  {
    constexpr int U = 7;  // blocks in flight per warp
    int J = 0, first = 0;
    for (int b0 = warp; b0 < nblk; b0 += U * kCpWarps) {
      double2 v[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int b = b0 + q * kCpWarps;
        while (J < nb && b >= first + nb - J) {
          first += nb - J;
          ++J;
        }
        const int I = J + b - first, r = 8 * I + g, c = 8 * J + 2 * t;
        v[q] = make_double2(r == c ? 1.0 : 0.0, r == c + 1 ? 1.0 : 0.0);
        if constexpr (CX) {
          if (b < nblk && r < k && c < k) {
            const int rr = r >> 1, cc = c >> 1;
            double2 z = reinterpret_cast<const double2*>(G)[min(rr, cc) + int64_t(max(rr, cc)) * ldg];
            if (rr > cc) z.y = -z.y;  // the upper triangle is stored
            if (rr == cc) z.y = 0.0;
            v[q] = (r & 1) ? make_double2(z.y, z.x) : make_double2(z.x, -z.y);
          }
        } else if (b < nblk && r < k) {
          if (c < k) v[q].x = G[min(r, c) + int64_t(max(r, c)) * ldg];
          if (c + 1 < k) v[q].y = G[min(r, c + 1) + int64_t(max(r, c + 1)) * ldg];
        }
      }
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (b0 + q * kCpWarps < nblk) S[(b0 + q * kCpWarps) * 32 + lane] = v[q];
    }
  }
  __syncthreads();

  factor_panels(S, k, shift_factor, Rpk, write_g ? G : nullptr, ldg);
  if (write_g) {
    // R's rows right of the diagonal blocks, and zeros below the diagonal
    __syncthreads();
    for (int c = warp; c < k; c += kCpWarps)
      for (int r = lane; r < k; r += 32) {
        if (r > c) G[r + int64_t(c) * ldg] = 0.0;
        else if ((r >> 3) < (c >> 3)) {
          const double2 q = S[(col_base(r >> 3, nb) + (c >> 3) - (r >> 3)) * 32 + (c & 7) * 4 + ((r & 7) >> 1)];
          G[r + int64_t(c) * ldg] = (r & 1) ? q.y : q.x;
        }
      }
  }
}

// x R = y for eight rows per warp, held as NB accumulator blocks, the current block
// column in a[0] (the array moves down by one block per step, so the loop's code stays
// small: executed once, an unrolled one waits for its own instructions).  X_J = T_J
// R_JJ^-1 with the inverse from R's diagonal block, then X_J times R's block row J is
// subtracted from the columns after it.  An accumulator block is an A operand as it
// stands: lane (g, t) holds the columns 2t and 2t + 1.  R: the packed factor at the
// lane's offset; three blocks after its end are read.
template <int NB, class Store>
__device__ __forceinline__ void solve_rows(double (&a)[NB][2], const double2* R, int nb, Store store) {
  for (int J = 0; J < nb; ++J) {
    const double2 b = R[0];
    double x0 = 0.0, x1 = 0.0;
    dmma8(x0, x1, a[0][0], b.x);
    dmma8(x0, x1, a[0][1], b.y);
    store(J, x0, x1);
    const double m0 = -x0, m1 = -x1;
    // four blocks at a time, as far as there are any (a group may run over the end of
    // the block row: what it computes there is not used)
#pragma unroll
    for (int K0 = 1; K0 < NB; K0 += 4)
      if (J + K0 < nb) {
        double2 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = R[(K0 + i) * 32];
#pragma unroll
        for (int i = 0; i < 4 && K0 + i < NB; ++i)
          dmma8(a[K0 + i - 1][0], a[K0 + i - 1][1], m0, q[i].x, a[K0 + i][0], a[K0 + i][1]);
#pragma unroll
        for (int i = 0; i < 4 && K0 + i < NB; ++i) dmma8(a[K0 + i - 1][0], a[K0 + i - 1][1], m1, q[i].y);
      }
    R += (nb - J) * 32;
  }
}

// Q = Y R^-1.  The CTA's warps beyond those with rows only help to stage R.
constexpr int kTpThreads = 256;

// CX: complex Y and Q of k / 2 columns; a row enters as (re, -im) pairs, the first row
// of its 2 x 2 blocks, one element per lane and block.
template <int NB, bool CX>
__global__ void __launch_bounds__(kTpThreads) trsm_panel_kernel(const double* __restrict__ Y, int64_t ldy, int64_t N,
                                                                int k, int warps, const double2* __restrict__ Rpk,
                                                                double* __restrict__ Q, int64_t ldq) {
  pdl_wait();
  extern __shared__ __align__(16) double2 Rs[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nb = (k + 7) >> 3, n2 = nb * (nb + 1) / 2 * 32;
  const int64_t row = (int64_t(blockIdx.x) * warps + warp) * 8 + g;
  const bool mine = warp < warps && row < N;
  double a[NB][2];
#pragma unroll
  for (int J = 0; J < NB; ++J) {
    const int c = 8 * J + 2 * t;
    if constexpr (CX) {
      double2 z = make_double2(0.0, 0.0);
      if (mine && c < k) z = reinterpret_cast<const double2*>(Y)[row + int64_t(c >> 1) * ldy];
      a[J][0] = z.x;
      a[J][1] = -z.y;
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e) a[J][e] = (mine && c + e < k) ? Y[row + int64_t(c + e) * ldy] : 0.0;
    }
  }
  // (all of R in flight at once: 16-byte copies that bypass the registers)
  for (int i = tid; i < n2; i += kTpThreads)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(unsigned(__cvta_generic_to_shared(Rs + i))),
                 "l"(Rpk + i));
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (warp >= warps) return;
  solve_rows<NB>(a, Rs + lane, nb, [&](int J, double x0, double x1) {
    const int c = 8 * J + 2 * t;
    if constexpr (CX) {
      if (mine && c < k) reinterpret_cast<double2*>(Q)[row + int64_t(c >> 1) * ldq] = make_double2(x0, -x1);
    } else {
      if (mine && c < k) Q[row + int64_t(c) * ldq] = x0;
      if (mine && c + 1 < k) Q[row + int64_t(c + 1) * ldq] = x1;
    }
  });
}

// All passes of one orthonormalisation in one launch of one CTA: the Gram product (one
// warp per strip of a block and the one below it), the factor and the solve, in shared
// memory.  The separate kernels of a pass are three launches of 5 to 10 us, most of
// it the way to global memory and back.  Gradient at D = 2, chi = 16 71.4 -> 65.4 ms
// (64 rows), chi = 30 75.6 -> 70.9 ms (120 rows); complex energy at chi = 8 24.8 -> 21.1
// ms (32 rows), chi = 14 25.6 -> 22.6 ms.
// The columns from k to 8 nb are zero (G: the identity).  CX: complex rows enter the
// Gram product as both rows of their 2 x 2 blocks.
// smem: R, then Y row by row, ld = 8 nb + 4 (the fragments' reads then meet no bank conflict).
__host__ __device__ __forceinline__ int orth_ld(int nb) { return 8 * nb + 4; }

struct OrthArgs {
  const double* Y;
  double* Q;
  double2* Rpk;  // packed R per pass, or null
  int64_t N, ldy, ldq;
  int k, rows, passes;  // rows: N rounded up to a multiple of 8
  double shift;         // first pass
};

template <int NB, bool CX>
__global__ void __launch_bounds__(kCpThreads, 1) orth_kernel(OrthArgs o) {
  pdl_wait();
  extern __shared__ __align__(16) double2 S[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int k = o.k, nb = (k + 7) >> 3, nblk = nb * (nb + 1) / 2, ld = orth_ld(nb);
  double* Ys = reinterpret_cast<double*>(S + (nblk + 3) * 32);  // (the solve reads three blocks past R)
  const int groups = o.rows >> 3, steps = o.rows / 4 * (CX ? 2 : 1);

  // rows from global memory, a warp 8 rows of 4 columns at a time (complex: 16 of 2)
  {
    constexpr int CPW = CX ? 2 : 4;
    const int cols = CX ? k / 2 : k, wide = CX ? 4 * nb : 8 * nb;
    constexpr int RPW = 32 / CPW;
    const int cc = lane % CPW, rr = lane / CPW;
    const int cg_ = (wide + CPW - 1) / CPW, rg = (o.rows + RPW - 1) / RPW;
    for (int u = warp; u < cg_ * rg; u += kCpWarps) {
      const int c = (u / rg) * CPW + cc, r = (u % rg) * RPW + rr;
      if (r >= o.rows || c >= wide) continue;
      const bool in = r < o.N && c < cols;
      if constexpr (CX) {
        double2 z = make_double2(0.0, 0.0);
        if (in) z = reinterpret_cast<const double2*>(o.Y)[r + int64_t(c) * o.ldy];
        *reinterpret_cast<double2*>(Ys + (2 * r) * ld + 2 * c) = make_double2(z.x, -z.y);
        *reinterpret_cast<double2*>(Ys + (2 * r + 1) * ld + 2 * c) = make_double2(z.y, z.x);
      } else {
        Ys[r * ld + c] = in ? o.Y[r + int64_t(c) * o.ldy] : 0.0;
      }
    }
  }
  __syncthreads();

  for (int pass = 0; pass < o.passes; ++pass) {
    // the Gram product's lower blocks (I, J), (I + 1, J) for strips of two block rows
    int J = 0, first = 0;
    for (int u = warp;; u += kCpWarps) {
      while (J < nb && u - first >= (nb - J + 1) / 2) {
        first += (nb - J + 1) / 2;
        ++J;
      }
      if (J >= nb) break;
      const int I = J + 2 * (u - first);
      const bool two = I + 1 < nb;
      const double *yi = Ys + t * ld + 8 * I + g, *yj = Ys + t * ld + 8 * J + g, *yk = two ? yi + 8 : yi;
      double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 4
      for (int q = 0; q < steps; ++q) {
        const double b = yj[q * 4 * ld];
        dmma8(c[0][0], c[0][1], yi[q * 4 * ld], b);
        dmma8(c[1][0], c[1][1], yk[q * 4 * ld], b);
      }
      if (I == J) {  // columns from k on
        const int r = 8 * I + g, cc = 8 * J + 2 * t;
        if (r >= k && r == cc) c[0][0] = 1.0;
        if (r >= k && r == cc + 1) c[0][1] = 1.0;
      }
      double2* d = S + (col_base(J, nb) + I - J) * 32 + lane;
      d[0] = make_double2(c[0][0], c[0][1]);
      if (two) d[32] = make_double2(c[1][0], c[1][1]);
    }
    __syncthreads();
    factor_panels(S, k, pass == 0 ? o.shift : 0.0, o.Rpk ? o.Rpk + int64_t(pass) * nblk * 32 : nullptr,
                  nullptr, 0);
    __syncthreads();
    const bool last = pass + 1 == o.passes;
    for (int w = warp; w < groups; w += kCpWarps) {
      double* y = Ys + (CX ? 2 : 1) * (w * 8 + g) * ld + 2 * t;  // this lane's row
      double a[NB][2];
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double2 v = j < nb ? *reinterpret_cast<const double2*>(y + 8 * j) : make_double2(0.0, 0.0);
        a[j][0] = v.x;
        a[j][1] = v.y;
      }
      const int64_t row = w * 8 + g;
      const bool mine = row < o.N;
      solve_rows<NB>(a, S + lane, nb, [&](int j, double x0, double x1) {
        const int c = 8 * j + 2 * t;
        if (!last) {
          *reinterpret_cast<double2*>(y + 8 * j) = make_double2(x0, x1);
          if constexpr (CX) *reinterpret_cast<double2*>(y + ld + 8 * j) = make_double2(-x1, x0);
        } else if constexpr (CX) {
          if (mine && c < k) reinterpret_cast<double2*>(o.Q)[row + int64_t(c >> 1) * o.ldq] = make_double2(x0, -x1);
        } else {
          if (mine && c < k) o.Q[row + int64_t(c) * o.ldq] = x0;
          if (mine && c + 1 < k) o.Q[row + int64_t(c + 1) * o.ldq] = x1;
        }
      });
    }
    __syncthreads();
  }
}

constexpr size_t kOrthSmem = 226 * 1024;

int orth_rows(int64_t N) { return int((N + 7) / 8 * 8); }
size_t orth_smem(int k, int64_t N, bool cx) {
  const int nb = (k + 7) / 8, nblk = nb * (nb + 1) / 2;
  return size_t(nblk + 3) * 512 + size_t(orth_rows(N)) * (cx ? 2 : 1) * orth_ld(nb) * 8;
}

// Up to 128 rows (64 complex ones, 128 in shared memory).  Gradient with one CTA's kernel
// up to 0 / 128 / 400 rows, ms: 120 rows 75.6 / 70.9 / 71.0, 200 rows 92.4 / 91.5 / 102.7,
// 252 rows 84.9 / 83.1 / 85.8: beyond that the Gram product and the solve take longer on
// one SM than they save.  Clusters of 2 to 8 CTAs with the sum through distributed
// shared memory gave nothing at 333 and 1024 rows and lost 8% at 432.
constexpr int kOrthMaxRows = 128;

// k real columns
bool fits_one(int64_t N, int k, bool cx) {
  return N >= 1 && k >= 1 && N * (cx ? 2 : 1) <= kOrthMaxRows && k <= kOrthMaxK && orth_smem(k, N, cx) <= kOrthSmem;
}

template <int NB, bool CX>
void launch_orth(Ctx& c, const OrthArgs& o) {
  static SmemAttrOnce attr;
  attr.ensure(orth_kernel<NB, CX>, int(kOrthSmem));
  launch(c.stream, orth_kernel<NB, CX>, 1, kCpThreads, orth_smem(o.k, o.N, CX), o);
  IPEPS_LAUNCH_CHECK();
}

template <bool CX>
void orth_by_width(Ctx& c, const OrthArgs& o) {
  switch ((o.k + 31) / 32) {
    case 1: launch_orth<4, CX>(c, o); break;
    case 2: launch_orth<8, CX>(c, o); break;
    case 3: launch_orth<12, CX>(c, o); break;
    default: launch_orth<16, CX>(c, o); break;
  }
}

template <bool CX>
void launch_chol(Ctx& c, double* G, int k, int64_t ldg, double shift_factor, double* Rpk, bool write_g) {
  static SmemAttrOnce attr;
  attr.ensure(chol_panel_kernel<CX>, int(size_t(cholqr_packed(kCholqrMax)) * 8));
  launch(c.stream, chol_panel_kernel<CX>, 1, kCpThreads, size_t(cholqr_packed(k)) * 8, G, k, ldg, shift_factor,
         reinterpret_cast<double2*>(Rpk), write_g);
  IPEPS_LAUNCH_CHECK();
}

template <int NB, bool CX>
void launch_trsm(Ctx& c, const double* Y, int64_t ldy, int64_t N, int k, const double* Rpk, double* Q, int64_t ldq) {
  const size_t pad = 3 * 512;  // a group of four blocks reads over the end
  const size_t smem = size_t(cholqr_packed(k)) * 8 + pad;
  static SmemAttrOnce attr;
  attr.ensure(trsm_panel_kernel<NB, CX>, int(size_t(cholqr_packed(8 * NB)) * 8 + pad));
  // eight rows per warp; one CTA per SM as long as eight warps hold its rows (R is staged once per CTA)
  const int64_t groups = (N + 7) / 8;
  const int64_t warps = std::min<int64_t>(kTpThreads / 32, (groups + c.sm_count - 1) / c.sm_count);
  launch(c.stream, trsm_panel_kernel<NB, CX>, unsigned((groups + warps - 1) / warps), kTpThreads, smem, Y, ldy, N, k,
         int(warps), reinterpret_cast<const double2*>(Rpk), Q, ldq);
  IPEPS_LAUNCH_CHECK();
}

template <bool CX>
void trsm_by_width(Ctx& c, const double* Y, int64_t ldy, int64_t N, int k, const double* Rpk, double* Q, int64_t ldq) {
  switch ((k + 31) / 32) {
    case 1: launch_trsm<4, CX>(c, Y, ldy, N, k, Rpk, Q, ldq); break;
    case 2: launch_trsm<8, CX>(c, Y, ldy, N, k, Rpk, Q, ldq); break;
    case 3: launch_trsm<12, CX>(c, Y, ldy, N, k, Rpk, Q, ldq); break;
    case 4: launch_trsm<16, CX>(c, Y, ldy, N, k, Rpk, Q, ldq); break;
    case 5: launch_trsm<20, CX>(c, Y, ldy, N, k, Rpk, Q, ldq); break;
    default: launch_trsm<24, CX>(c, Y, ldy, N, k, Rpk, Q, ldq); break;
  }
}

}  // namespace

int64_t cholqr_packed(int k) {
  const int64_t nb = (k + 7) / 8;
  return nb * (nb + 1) / 2 * 64;
}

void chol_packed(Ctx& c, double* G, int k, int64_t ldg, double shift_factor, double* Rpk, bool write_g) {
  IPEPS_CHECK(cholqr_fits(k), "chol_packed: k out of range");
  ProfScope ps(c, KFam::SmallLinalg);
  launch_chol<false>(c, G, k, ldg, shift_factor, Rpk, write_g);
  c.count(KFam::SmallLinalg, double(k) * k * k / 3.0);
}

void trsm_packed(Ctx& c, const double* Y, int64_t ldy, int64_t N, int k, const double* Rpk, double* Q, int64_t ldq) {
  IPEPS_CHECK(cholqr_fits(k), "trsm_packed: k out of range");
  if (N == 0) return;
  ProfScope ps(c, KFam::SmallLinalg);
  trsm_by_width<false>(c, Y, ldy, N, k, Rpk, Q, ldq);
  c.count(KFam::SmallLinalg, double(N) * k * k);
}

// the real form of G has twice its trace: half the shift factor is the same shift
void chol_packed_c(Ctx& c, const void* G, int k, int64_t ldg, double shift_factor, double* Rpk) {
  IPEPS_CHECK(cholqr_fits(2 * k), "chol_packed_c: k out of range");
  ProfScope ps(c, KFam::SmallLinalg);
  launch_chol<true>(c, static_cast<double*>(const_cast<void*>(G)), 2 * k, ldg, 0.5 * shift_factor, Rpk, false);
  c.count(KFam::SmallLinalg, 8.0 * double(k) * k * k / 6.0);
}

void trsm_packed_c(Ctx& c, const void* Y, int64_t ldy, int64_t N, int k, const double* Rpk, void* Q, int64_t ldq) {
  IPEPS_CHECK(cholqr_fits(2 * k), "trsm_packed_c: k out of range");
  if (N == 0) return;
  ProfScope ps(c, KFam::SmallLinalg);
  trsm_by_width<true>(c, static_cast<const double*>(Y), ldy, N, 2 * k, Rpk, static_cast<double*>(Q), ldq);
  c.count(KFam::SmallLinalg, 4.0 * double(N) * k * k);
}

bool orth_fits(int64_t N, int k) { return fits_one(N, k, false); }
bool orth_fits_c(int64_t N, int k) { return fits_one(N, 2 * k, true); }

void orth_small(Ctx& c, const double* Y, int64_t N, int k, int passes, double shift_factor, double* Rpk, double* Q) {
  IPEPS_CHECK(orth_fits(N, k) && passes > 0, "orth_small: size out of range");
  ProfScope ps(c, KFam::SmallLinalg);
  orth_by_width<false>(c, OrthArgs{Y, Q, reinterpret_cast<double2*>(Rpk), N, N, N, k, orth_rows(N), passes, shift_factor});
  c.count(KFam::SmallLinalg, passes * (2.0 * N * k * k + double(k) * k * k / 3.0));
}

// (the real form of G has twice its trace: half the shift factor is the same shift)
void orth_small_c(Ctx& c, const void* Y, int64_t N, int k, int passes, double shift_factor, void* Q) {
  IPEPS_CHECK(orth_fits_c(N, k) && passes > 0, "orth_small_c: size out of range");
  ProfScope ps(c, KFam::SmallLinalg);
  orth_by_width<true>(c, OrthArgs{static_cast<const double*>(Y), static_cast<double*>(Q), nullptr, N, N, N, 2 * k,
                                  orth_rows(N), passes, 0.5 * shift_factor});
  c.count(KFam::SmallLinalg, passes * (8.0 * N * k * k + 8.0 * double(k) * k * k / 6.0));
}

}  // namespace ipeps
