// Mixed-precision preconditioned conjugate gradient for k right-hand sides at
// once (the batched-RHS solve of the predictive variance), device resident.
//
// Iteration, every scalar per column and on the device (solve_2d,
// laker/solvers.py:297-394):
//   AP = lam P + K32 P                    multi-RHS FP32 operator
//   pAp_c, |p_c|, |Ap_c|                   -> alpha_c; breakdown if any column
//                                             has p_c^T A p_c <= -eps |p_c| |Ap_c|
//   X += P diag(alpha); R -= AP diag(alpha)        (X, R in FP64); |R|_F
//   reliable update: R = B - A64 X (FP64 multi-RHS residual) when |R|_F fell
//     by `delta` from its running maximum since the last recomputation, when
//     the recurrence says the stop test may hold, and at max_iter; the stop
//     test is only taken on that FP64 residual:
//       default      |R|_F <= tol |B|_F   (the reference's global Frobenius
//                                         test, solvers.py:365-368)
//       column_stop  every column c with |r_c| <= tol |b_c| is frozen (its
//                    alpha, beta and search direction become zero) and the
//                    solve ends when all are
//   Z = P R (factored CCCP apply, multi-RHS); rz_c -> beta_c
//   P = Z + P diag(beta)
// Every kernel reads the device state first and does nothing once the solve
// has ended, so the host replays the captured iteration several times between
// polls.  Column reductions are fixed-order (per-CTA partials over a fixed row
// partition, then a fixed-order sum by the last CTA), so results do not depend
// on scheduling.  Data are row-major n x k with leading dimension k.
//
// A column whose search direction is exactly zero (a zero right-hand side) is
// solved exactly (x_c = 0, alpha_c = 0); the reference's breakdown test
// reports p^T A p = 0 <= -eps * 0 as a breakdown for it instead.
#include <chrono>

#include "pcg_state.cuh"
#include "sym.cuh"

namespace laker {

bool precond_valid(const laker_precond* pc);

namespace {

constexpr int kMT = 256;         // threads of the vector kernels
constexpr int kCW = 32;          // columns per CTA of the column-reduction kernels
constexpr int kRW = kMT / kCW;   // row lanes per CTA
constexpr int kGThreads = 128;   // threads of the apply's GEMMs
constexpr int kGT = 128;         // rows of their output tiles (8 per thread)
constexpr int kGK = 16;          // their K step

struct alignas(256) MpcgState {
  double bnorm;       // |B|_F
  double tol_abs;     // tol |B|_F
  double tol;         // relative tolerance
  double rnorm;       // |R|_F of the recurrence (after the last update)
  double rmax;        // running max of |R|_F since the last FP64 recomputation
  double true_rnorm;  // |B - A X|_F from the last FP64 recomputation
  double delta;       // reliable-update factor
  double eps;         // breakdown threshold
  int iter;           // iterations (FP32 operator applications)
  int n_accurate;     // FP64 residual recomputations
  int max_iter;
  int active;         // 1 while the solve runs (gate of the operator)
  int need_update;    // 1 when this iteration ends with an FP64 recomputation
  int done;
  int status;
  int column_stop;    // 1: per-column stop test with freezing
  int n_live;         // columns still iterating
  int pad;
  unsigned int counters[8];
};

enum { kMCtrInit = 0, kMCtrMatvec, kMCtrUpdate, kMCtrResid, kMCtrPrecond };

// Per-column state (k entries each), in the workspace.
struct MpcgCols {
  double* bnorm;  // |b_c|
  double* rz;     // r_c . z_c
  double* alpha;
  double* beta;
  double* rn;     // |r_c|: recurrence, or the FP64 residual after a recomputation
  int* live;      // 1 while column c iterates
  double* ypart;  // [kind][column chunk][3]: per-chunk results of the reductions
  unsigned int* yctr;  // [kind][column chunk]: arrival counters of the chunk reductions
};
constexpr int kMKinds = 5;

__device__ __forceinline__ void mp_stop(MpcgState* st, int status) {
  st->status = status;
  st->done = 1;
  st->active = 0;
}

// Column-reduction grid: blockIdx.y covers columns [32 y, 32 y + 32),
// blockIdx.x rows x*8 + r + gx*8*t (r = thread row lane).
struct ColGrid {
  int gx, gy;
};

ColGrid col_grid(int64_t n, int k) {
  ColGrid g{};
  g.gy = (int)ceil_div(k, kCW);
  // Four CTAs per SM keep more rows in flight (n = 20,000, k = 256: x and r updated in
  // 41 us, 81 with two CTAs and one row's loads at a time); at most two per SM in one
  // column group, whose last CTA adds the partial sums of all.
  int64_t gx = ceil_div(4 * (int64_t)sm_count(), g.gy);
  if (gx > 2 * (int64_t)sm_count()) gx = 2 * (int64_t)sm_count();
  const int64_t lim = ceil_div(n, kRW);
  if (gx > lim) gx = lim;
  if (gx > 512) gx = 512;
  g.gx = (int)(gx < 1 ? 1 : gx);
  return g;
}

// Stores this CTA's per-column partial sums of NQ quantities (fixed order over
// the CTA's row lanes) at bp[q * qstride + blockIdx.x * k + c].
template <int NQ>
__device__ __forceinline__ void store_col_partials(const double (&v)[NQ], double* bp,
                                                   int64_t qstride, int k) {
  __shared__ double s[NQ][kRW][kCW];
  const int tc = threadIdx.x % kCW, tr = threadIdx.x / kCW;
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q][tr][tc] = v[q];
  __syncthreads();
  if (tr == 0) {
    const int c = blockIdx.y * kCW + tc;
    if (c < k) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        double t = 0.0;
#pragma unroll
        for (int r = 0; r < kRW; ++r) t += s[q][r][tc];
        bp[q * qstride + (int64_t)blockIdx.x * k + c] = t;
      }
    }
  }
}

// Two-level fixed-order reduction of the per-CTA column partials.  Level 1:
// the last CTA of each column chunk (blockIdx.y) adds its 32 columns' partials
// over the grid's CTAs (row lane r takes CTAs r, r + 8, ..., coalesced over the
// columns; then the lanes in order) and applies the per-column logic in warp
// 0 (lane = column); level 2: the last of those CTAs combines the chunks'
// results (in chunk order) for the solve-wide decisions.

// Level 1 entry: true in the CTA that completes this column chunk.
__device__ __forceinline__ bool chunk_last(MpcgCols cols, int kind) {
  return arrive_last_of(&cols.yctr[kind * gridDim.y + blockIdx.y], gridDim.x);
}

// Column totals of this chunk's 32 columns, valid in warp 0 (column
// blockIdx.y * 32 + lane; zero for columns past k).  Whole CTA.
template <int NQ>
__device__ __forceinline__ void chunk_totals(const double* bp, int64_t qs, int k, double (&tot)[NQ]) {
  __shared__ double sred[NQ][kRW][kCW];
  const int tc = threadIdx.x % kCW, tr = threadIdx.x / kCW;
  const int c = blockIdx.y * kCW + tc;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double t = 0.0;
    if (c < k)
#pragma unroll 8
      for (unsigned int b = tr; b < gridDim.x; b += kRW) t += __ldcg(bp + q * qs + (int64_t)b * k + c);
    sred[q][tr][tc] = t;
  }
  __syncthreads();
  if (tr == 0) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      double t = 0.0;
#pragma unroll
      for (int r = 0; r < kRW; ++r) t += sred[q][r][tc];
      tot[q] = t;
    }
  }
}

// Level 2 entry (whole CTA, after warp 0 stored the chunk's results): true in
// the CTA that completes the last chunk.
__device__ __forceinline__ bool solve_last(MpcgState* st, int kind) {
  return arrive_last_of(&st->counters[kind], gridDim.y);
}

// Sum of slot j of the chunks' results, in chunk order (one thread).
__device__ __forceinline__ double chunks_sum(MpcgCols cols, int kind, int j) {
  double t = 0.0;
  for (unsigned int y = 0; y < gridDim.y; ++y) t += __ldcg(cols.ypart + ((int64_t)kind * gridDim.y + y) * 3 + j);
  return t;
}

__device__ __forceinline__ void put_chunk(MpcgCols cols, int kind, double a, double b, double c) {
  double* d = cols.ypart + ((int64_t)kind * gridDim.y + blockIdx.y) * 3;
  d[0] = a;
  d[1] = b;
  d[2] = c;
}

// X = 0 and R = B (unless warm start), |b_c| -> bnorm, |B|_F, tolerances.
__global__ void __launch_bounds__(kMT)
    mp_init_kernel(const double* __restrict__ B, double* __restrict__ X, double* __restrict__ R,
                   int64_t n, int k, int has_x0, double* bp, MpcgState* st, MpcgCols cols) {
  const int c = blockIdx.y * kCW + threadIdx.x % kCW;
  double acc = 0.0;
  if (c < k) {
#pragma unroll 4  // the loads of four rows in flight
    for (int64_t i = (int64_t)blockIdx.x * kRW + threadIdx.x / kCW; i < n;
         i += (int64_t)gridDim.x * kRW) {
      const int64_t e = i * k + c;
      const double b = B[e];
      if (!has_x0) {
        R[e] = b;
        X[e] = 0.0;
      }
      acc = fma(b, b, acc);
    }
  }
  const double v[1] = {acc};
  store_col_partials<1>(v, bp, 0, k);
  if (!chunk_last(cols, kMCtrInit)) return;
  double tot[1];
  chunk_totals<1>(bp, 0, k, tot);
  if (threadIdx.x < kCW) {
    const int cc = blockIdx.y * kCW + threadIdx.x;
    double fro = 0.0;
    if (cc < k) {
      const double bn = sqrt(tot[0]);
      cols.bnorm[cc] = bn;
      cols.rn[cc] = bn;
      cols.live[cc] = 1;
      fro = tot[0];
    }
    fro = warp_sum(fro);
    if (threadIdx.x == 0) put_chunk(cols, kMCtrInit, fro, 0.0, 0.0);
  }
  if (!solve_last(st, kMCtrInit)) return;
  if (threadIdx.x == 0) {
    const double bn = sqrt(chunks_sum(cols, kMCtrInit, 0));
    st->bnorm = bn;
    st->tol_abs = st->tol * bn;
    st->rnorm = bn;
    st->rmax = bn;
    st->true_rnorm = bn;
    st->n_live = k;
    if (!isfinite(bn)) mp_stop(st, LAKER_ERR_NONFINITE);
  }
}

// pAp_c, p_c.p_c, Ap_c.Ap_c -> alpha_c and the breakdown test.  A device-side
// failure of the operator (its status word) ends the solve with that status.
__global__ void __launch_bounds__(kMT)
    mp_after_matvec_kernel(const float* __restrict__ P, const float* __restrict__ AP, int64_t n,
                           int k, double* bp, MpcgState* st, MpcgCols cols, const int* dstatus) {
  if (st->done) return;
  const int c = blockIdx.y * kCW + threadIdx.x % kCW;
  double d0 = 0.0, d1 = 0.0, d2 = 0.0;
  if (c < k) {
#pragma unroll 4  // the loads of four rows in flight
    for (int64_t i = (int64_t)blockIdx.x * kRW + threadIdx.x / kCW; i < n;
         i += (int64_t)gridDim.x * kRW) {
      const double p = P[i * k + c], a = AP[i * k + c];
      d0 = fma(p, a, d0);
      d1 = fma(p, p, d1);
      d2 = fma(a, a, d2);
    }
  }
  const int64_t qs = (int64_t)gridDim.x * k;
  const double v[3] = {d0, d1, d2};
  store_col_partials<3>(v, bp, qs, k);
  if (!chunk_last(cols, kMCtrMatvec)) return;
  double tot[3];
  chunk_totals<3>(bp, qs, k, tot);
  if (threadIdx.x < kCW) {
    const int cc = blockIdx.y * kCW + threadIdx.x;
    bool nonfinite = false, breakdown = false;
    if (cc < k) {
      if (!cols.live[cc]) {
        cols.alpha[cc] = 0.0;
      } else {
        const double pap = tot[0], pp = tot[1], aa = tot[2];
        if (!isfinite(pap) || !isfinite(pp) || !isfinite(aa)) {
          nonfinite = true;
        } else if (pp > 0.0 && pap <= -st->eps * sqrt(pp) * sqrt(aa)) {
          breakdown = true;  // non-positive curvature (laker/solvers.py:343-352)
        }
        cols.alpha[cc] = (pp > 0.0 && pap != 0.0) ? cols.rz[cc] / pap : 0.0;
      }
    }
    const bool nf = __any_sync(0xffffffffu, nonfinite), bd = __any_sync(0xffffffffu, breakdown);
    if (threadIdx.x == 0) put_chunk(cols, kMCtrMatvec, nf ? 1.0 : 0.0, bd ? 1.0 : 0.0, 0.0);
  }
  if (!solve_last(st, kMCtrMatvec)) return;
  if (threadIdx.x == 0) {
    const bool nf = chunks_sum(cols, kMCtrMatvec, 0) != 0.0;
    const bool bd = chunks_sum(cols, kMCtrMatvec, 1) != 0.0;
    if (status_failed(dstatus)) mp_stop(st, *dstatus);
    else if (nf) mp_stop(st, LAKER_ERR_NONFINITE);
    else if (bd) mp_stop(st, LAKER_ERR_BREAKDOWN);
  }
}

// X += alpha P; R -= alpha AP; |r_c|, |R|_F -> decide on the FP64 recomputation.
__global__ void __launch_bounds__(kMT)
    mp_update_xr_kernel(const float* __restrict__ P, const float* __restrict__ AP,
                        double* __restrict__ X, double* __restrict__ R, int64_t n, int k, double* bp,
                        MpcgState* st, MpcgCols cols) {
  if (st->done) return;
  const int c = blockIdx.y * kCW + threadIdx.x % kCW;
  double acc = 0.0;
  if (c < k) {
    const double a = cols.alpha[c];
    // four rows at a time, every load before the first store (a store to X or R may
    // alias the next row's load, so the compiler keeps their order)
    const int64_t step = (int64_t)gridDim.x * kRW;
    for (int64_t i = (int64_t)blockIdx.x * kRW + threadIdx.x / kCW; i < n; i += 4 * step) {
      double x[4], r[4];
      float p[4], ap[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t e = min(i + u * step, n - 1) * k + c;
        x[u] = X[e];
        r[u] = R[e];
        p[u] = P[e];
        ap[u] = AP[e];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i + u * step >= n) break;
        const int64_t e = (i + u * step) * k + c;
        X[e] = fma(a, (double)p[u], x[u]);
        r[u] = fma(-a, (double)ap[u], r[u]);
        R[e] = r[u];
        acc = fma(r[u], r[u], acc);
      }
    }
  }
  const double v[1] = {acc};
  store_col_partials<1>(v, bp, 0, k);
  if (!chunk_last(cols, kMCtrUpdate)) return;
  double tot[1];
  chunk_totals<1>(bp, 0, k, tot);
  if (threadIdx.x < kCW) {
    const int cc = blockIdx.y * kCW + threadIdx.x;
    double fro = 0.0;
    bool below = true;  // every live column's recurrence residual at its tolerance
    if (cc < k) {
      const double rn = sqrt(tot[0]);
      cols.rn[cc] = rn;
      fro = tot[0];
      if (cols.live[cc] && !(rn <= st->tol * cols.bnorm[cc])) below = false;
    }
    fro = warp_sum(fro);
    const bool all = __all_sync(0xffffffffu, below);
    if (threadIdx.x == 0) put_chunk(cols, kMCtrUpdate, fro, all ? 0.0 : 1.0, 0.0);
  }
  if (!solve_last(st, kMCtrUpdate)) return;
  if (threadIdx.x == 0) {
    const int all_below = chunks_sum(cols, kMCtrUpdate, 1) == 0.0 ? 1 : 0;
    const double rn = sqrt(chunks_sum(cols, kMCtrUpdate, 0));
    st->rnorm = rn;
    st->iter += 1;
    if (rn > st->rmax) st->rmax = rn;
    const bool may_stop = st->column_stop ? (all_below != 0) : (rn <= st->tol_abs);
    st->need_update =
        (rn <= st->delta * st->rmax || may_stop || st->iter >= st->max_iter || !isfinite(rn)) ? 1 : 0;
  }
}

// After the FP64 residual R = B - A64 X: |r_c|, |R|_F and the stop test.
// `init` (warm start) seeds the state without a stop test.
__global__ void __launch_bounds__(kMT)
    mp_after_residual_kernel(const double* __restrict__ R, int64_t n, int k, int init, double* bp,
                             MpcgState* st, MpcgCols cols) {
  if (st->done || (!init && !st->need_update)) return;
  const int c = blockIdx.y * kCW + threadIdx.x % kCW;
  double acc = 0.0;
  if (c < k) {
#pragma unroll 4  // the loads of four rows in flight
    for (int64_t i = (int64_t)blockIdx.x * kRW + threadIdx.x / kCW; i < n;
         i += (int64_t)gridDim.x * kRW) {
      const double r = R[i * k + c];
      acc = fma(r, r, acc);
    }
  }
  const double v[1] = {acc};
  store_col_partials<1>(v, bp, 0, k);
  if (!chunk_last(cols, kMCtrResid)) return;
  double tot[1];
  chunk_totals<1>(bp, 0, k, tot);
  if (threadIdx.x < kCW) {
    const int cc = blockIdx.y * kCW + threadIdx.x;
    const bool freeze = st->column_stop && !init;
    double fro = 0.0, live = 0.0;
    bool nonfinite = false;
    if (cc < k) {
      const double rn = sqrt(tot[0]);
      cols.rn[cc] = rn;
      fro = tot[0];
      if (!isfinite(rn)) nonfinite = true;
      if (freeze && cols.live[cc] && rn <= st->tol * cols.bnorm[cc]) cols.live[cc] = 0;
      live = cols.live[cc] ? 1.0 : 0.0;
    }
    fro = warp_sum(fro);
    live = warp_sum(live);
    const bool nf = __any_sync(0xffffffffu, nonfinite);
    if (threadIdx.x == 0) put_chunk(cols, kMCtrResid, fro, live, nf ? 1.0 : 0.0);
  }
  if (!solve_last(st, kMCtrResid)) return;
  if (threadIdx.x == 0) {
    const bool nf = chunks_sum(cols, kMCtrResid, 2) != 0.0;
    const double rn = sqrt(chunks_sum(cols, kMCtrResid, 0));
    const double live_total = chunks_sum(cols, kMCtrResid, 1);
    st->rnorm = rn;
    st->true_rnorm = rn;
    st->rmax = rn;
    st->n_accurate += 1;
    st->need_update = 0;
    st->n_live = (int)live_total;
    if (nf) {
      mp_stop(st, LAKER_ERR_NONFINITE);
    } else if (!init && (st->column_stop ? st->n_live == 0 : rn <= st->tol_abs)) {
      mp_stop(st, LAKER_OK);
    } else if (!init && st->iter >= st->max_iter) {
      mp_stop(st, LAKER_ERR_NOT_CONVERGED);
    }
  }
}

// r_c . z_c -> beta_c (or rz_c seeded when `init`).  IDENT: the identity
// preconditioner, Z = R rounded to FP32, written here.
template <bool IDENT>
__global__ void __launch_bounds__(kMT)
    mp_after_precond_kernel(const double* __restrict__ R, float* __restrict__ Z, int64_t n, int k,
                            int init, double* bp, MpcgState* st, MpcgCols cols) {
  if (st->done) return;
  const int c = blockIdx.y * kCW + threadIdx.x % kCW;
  double acc = 0.0;
  if (c < k) {
#pragma unroll 4  // the loads of four rows in flight
    for (int64_t i = (int64_t)blockIdx.x * kRW + threadIdx.x / kCW; i < n;
         i += (int64_t)gridDim.x * kRW) {
      const int64_t e = i * k + c;
      const double r = R[e];
      float z;
      if (IDENT) {
        z = (float)r;
        Z[e] = z;
      } else {
        z = Z[e];
      }
      acc = fma(r, (double)z, acc);
    }
  }
  const double v[1] = {acc};
  store_col_partials<1>(v, bp, 0, k);
  if (!chunk_last(cols, kMCtrPrecond)) return;
  double tot[1];
  chunk_totals<1>(bp, 0, k, tot);
  if (threadIdx.x < kCW) {
    const int cc = blockIdx.y * kCW + threadIdx.x;
    bool nonfinite = false;
    if (cc < k) {
      const double t = tot[0];
      if (!isfinite(t)) nonfinite = true;
      if (init) {
        cols.beta[cc] = 0.0;
      } else {
        const double rz = cols.rz[cc];
        cols.beta[cc] = (cols.live[cc] && rz != 0.0) ? t / rz : 0.0;
      }
      cols.rz[cc] = t;
    }
    const bool nf = __any_sync(0xffffffffu, nonfinite);
    if (threadIdx.x == 0) put_chunk(cols, kMCtrPrecond, nf ? 1.0 : 0.0, 0.0, 0.0);
  }
  if (!solve_last(st, kMCtrPrecond)) return;
  if (threadIdx.x == 0 && chunks_sum(cols, kMCtrPrecond, 0) != 0.0) mp_stop(st, LAKER_ERR_NONFINITE);
}

// P = Z + P diag(beta) (P = Z when `init`); frozen columns get P_c = 0.
__global__ void __launch_bounds__(kMT)
    mp_update_p_kernel(const float* __restrict__ Z, float* __restrict__ P, int64_t n, int k,
                       const MpcgState* st, MpcgCols cols, int init) {
  if (st->done) return;
  const int c = blockIdx.y * kCW + threadIdx.x % kCW;
  if (c >= k) return;
  const bool live = cols.live[c] != 0;
  const float beta = (float)cols.beta[c];
  const int64_t step = (int64_t)gridDim.x * kRW;
  for (int64_t i = (int64_t)blockIdx.x * kRW + threadIdx.x / kCW; i < n; i += 4 * step) {
    float z[4], p[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // every load before the first store, as above
      const int64_t e = min(i + u * step, n - 1) * k + c;
      z[u] = Z[e];
      p[u] = init ? 0.0f : P[e];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * step < n)
        P[(i + u * step) * k + c] = !live ? 0.0f : (init ? z[u] : fmaf(beta, p[u], z[u]));
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Multi-RHS factored CCCP apply Z = c^-1/2 R + Q (W (Q^T R)), three tiled
//   project  U_chunk = Q[rows of the chunk]^T R[rows of the chunk]  (FP32
//            products summed in FP32 within a row chunk, stored as FP64)
//   core     U = sum of the chunks in chunk order, V = W U          (FP64)
//   expand   Z = c^-1/2 R + Q V                                      (FP32 sum)
// It is only a preconditioner: FP32 sums change the iteration count, not the
// accuracy of the solution, whose stop test is on the FP64 residual.  The
// kernels read the first nq = round_up(N_r, 4) columns of Q (the columns from
// N_r on are zero in the factor layout); ldq is Q's row stride.
// ---------------------------------------------------------------------------
namespace {

// Tiles of the projection and the expansion: 128 rows x 8 CT columns (CT = 8, 4 or 2,
// pcm_ct), 8 x CT outputs per thread.  The shared-memory loads of the operands bind
// these GEMMs: with 4 x 4 outputs a thread read two float4 for 16 FMAs (L1 at 79 % of
// its peak, 138 and 98 us at n = 20,000, N_r = 200, k = 256); 8 x 8 reads four for 64
// (106 and 84 us).  k = 16 in 16-column tiles does a quarter of the work of 64
// (variance of 16 queries at n = 30,011: 241 -> 227 ms).

// acc += A^T B over a K step: a thread's rows are ty 4 .. + 3 and 64 + ty 4 .. + 3, its
// columns tx 4 .. + 3 and 32 + tx 4 .. + 3 (CT = 8) or tx CT .. + CT - 1.
template <int CT, int SA, int SB>
__device__ __forceinline__ void pcm_step(const float (*As)[SA], const float (*Bs)[SB], int ty, int tx,
                                         float2 (&acc)[8][CT / 2]) {
#pragma unroll
  for (int kk = 0; kk < kGK; ++kk) {
    const float4 a0 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
    const float4 a1 = *reinterpret_cast<const float4*>(&As[kk][64 + ty * 4]);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    float2 bv[CT / 2];
    if constexpr (CT == 2) {
      bv[0] = *reinterpret_cast<const float2*>(&Bs[kk][tx * 2]);
    } else {
#pragma unroll
      for (int h = 0; h < CT / 4; ++h) {
        const float4 b = *reinterpret_cast<const float4*>(&Bs[kk][h * 32 + tx * 4]);
        bv[2 * h] = make_float2(b.x, b.y);
        bv[2 * h + 1] = make_float2(b.z, b.w);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int v = 0; v < CT / 2; ++v) acc[u][v] = __ffma2_rn(make_float2(av[u], av[u]), bv[v], acc[u][v]);
  }
}

__device__ __forceinline__ int pcm_row(int ty, int u) { return (u < 4 ? 0 : 60) + ty * 4 + u; }
template <int CT>
__device__ __forceinline__ int pcm_col(int tx, int v) {
  return CT == 2 ? tx * 2 + v : (v < 4 ? 0 : 28) + tx * 4 + v;
}

template <int CT>
__global__ void __launch_bounds__(kGThreads)
    pcm_project_kernel(const float* __restrict__ Q, int ldq, int nq, const double* __restrict__ R,
                       int64_t n, int k, int64_t chunk_rows, double* __restrict__ upart,
                       const int* gate) {
  if (gate && *gate == 0) return;
  constexpr int TW = 8 * CT;
  __shared__ __align__(16) float Qs[2][kGK][kGT];
  __shared__ __align__(16) float Rs[2][kGK][TW];
  const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
  const int j0 = blockIdx.x * kGT, c0 = blockIdx.y * TW;
  const int64_t i_begin = (int64_t)blockIdx.z * chunk_rows;
  const int64_t i_end = min(n, i_begin + chunk_rows);
  float2 acc[8][CT / 2];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < CT / 2; ++v) acc[u][v] = make_float2(0.f, 0.f);
  // the next K step's tiles are loaded into registers while this one computes
  float4 qn[4];
  float rn[CT];
  const int qc = tid % 32 * 4, qr = tid / 32;  // Q: 4 rows at a time, 32 float4 of a row
  const int rc = tid % TW, rr = tid / TW;      // R: 128 / TW rows at a time
  const bool q_ok = j0 + qc < nq, r_ok = c0 + rc < k;
  auto fetch = [&](int64_t i) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int64_t ii = i + qr + 4 * h;
      qn[h] = (ii < i_end && q_ok) ? *reinterpret_cast<const float4*>(Q + ii * ldq + j0 + qc)
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int h = 0; h < CT; ++h) {
      const int64_t ii = i + rr + (kGThreads / TW) * h;
      rn[h] = (ii < i_end && r_ok) ? (float)R[ii * k + c0 + rc] : 0.0f;
    }
  };
  auto store = [&](int b) {
#pragma unroll
    for (int h = 0; h < 4; ++h) *reinterpret_cast<float4*>(&Qs[b][qr + 4 * h][qc]) = qn[h];
#pragma unroll
    for (int h = 0; h < CT; ++h) Rs[b][rr + (kGThreads / TW) * h][rc] = rn[h];
  };
  if (i_begin < i_end) {
    fetch(i_begin);
    store(0);
  }
  __syncthreads();
  int b = 0;
  for (int64_t i = i_begin; i < i_end; i += kGK, b ^= 1) {
    const bool more = i + kGK < i_end;
    if (more) fetch(i + kGK);
    pcm_step<CT>(Qs[b], Rs[b], ty, tx, acc);
    if (more) store(b ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int j = j0 + pcm_row(ty, u);
    if (j >= nq) continue;
#pragma unroll
    for (int v = 0; v < CT; ++v) {
      const int c = c0 + pcm_col<CT>(tx, v);
      if (c < k)
        upart[((int64_t)blockIdx.z * nq + j) * k + c] = (double)(v & 1 ? acc[u][v / 2].y : acc[u][v / 2].x);
    }
  }
}

// U = sum of the projection's row chunks, in chunk order.
__global__ void __launch_bounds__(kMT)
    pcm_sum_kernel(const double* __restrict__ upart, int nchunk, int64_t total, double* __restrict__ U,
                   const int* gate) {
  if (gate && *gate == 0) return;
  for (int64_t e = blockIdx.x * (int64_t)kMT + threadIdx.x; e < total; e += (int64_t)gridDim.x * kMT) {
    double u = 0.0;
#pragma unroll 8
    for (int ch = 0; ch < nchunk; ++ch) u += upart[(int64_t)ch * total + e];
    U[e] = u;
  }
}

// V = W U (FP64).  The product is small (N_r^2 k FMAs) and was bound by latency: 64 x 64
// tiles left 16 CTAs walking N_r with the chunk sums inside the loop (214 us at N_r =
// 200, k = 256).  16 x 32 tiles give ~100 CTAs; a thread owns two outputs and adds the
// N_r products in order, U and W staged 64 rows at a time.
constexpr int kCoreJ = 16, kCoreC = 32, kCoreK = 64;
__global__ void __launch_bounds__(kMT)
    pcm_core_kernel(const float* __restrict__ W, int nr, int nq, const double* __restrict__ U, int k,
                    double* __restrict__ V, const int* gate) {
  if (gate && *gate == 0) return;
  __shared__ double Ws[kCoreK][kCoreJ];
  __shared__ double Us[kCoreK][kCoreC];
  const int tid = threadIdx.x, c = tid % kCoreC, j = tid / kCoreC;  // outputs (j, c), (j + 8, c)
  const int j0 = blockIdx.x * kCoreJ, c0 = blockIdx.y * kCoreC;
  double a0 = 0.0, a1 = 0.0;
  for (int jp = 0; jp < nr; jp += kCoreK) {
    for (int e = tid; e < kCoreK * kCoreJ; e += kMT) {
      const int r = e / kCoreJ, q = e % kCoreJ;
      // W is symmetric: W[j][jj] = W[jj][j] (row jj read contiguously)
      Ws[r][q] = (jp + r < nr && j0 + q < nr) ? (double)W[(int64_t)(jp + r) * nr + j0 + q] : 0.0;
    }
    for (int e = tid; e < kCoreK * kCoreC; e += kMT) {
      const int r = e / kCoreC, q = e % kCoreC;
      Us[r][q] = (jp + r < nr && c0 + q < k) ? U[(int64_t)(jp + r) * k + c0 + q] : 0.0;
    }
    __syncthreads();
#pragma unroll 16
    for (int r = 0; r < kCoreK; ++r) {
      const double u = Us[r][c];
      a0 = fma(Ws[r][j], u, a0);
      a1 = fma(Ws[r][j + 8], u, a1);
    }
    __syncthreads();
  }
  if (c0 + c < k) {
    if (j0 + j < nq) V[(int64_t)(j0 + j) * k + c0 + c] = a0;
    if (j0 + j + 8 < nq) V[(int64_t)(j0 + j + 8) * k + c0 + c] = a1;
  }
}

template <int CT, typename ZT>
__global__ void __launch_bounds__(kGThreads)
    pcm_expand_kernel(const float* __restrict__ Q, int ldq, int nq, int nr,
                      const double* __restrict__ V, const double* __restrict__ R, double cis,
                      int64_t n, int k, ZT* __restrict__ Z, const int* gate) {
  if (gate && *gate == 0) return;
  constexpr int TW = 8 * CT;
  __shared__ __align__(16) float Qs[2][kGK][kGT + 4];  // transposed: Qs[j][i]
  __shared__ __align__(16) float Vs[2][kGK][TW];
  const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
  const int64_t i0 = (int64_t)blockIdx.x * kGT;
  const int c0 = blockIdx.y * TW;
  float2 acc[8][CT / 2];
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < CT / 2; ++v) acc[u][v] = make_float2(0.f, 0.f);
  float4 qn[4];
  float vn[CT];
  const int qi = tid / 4, qg = tid % 4 * 4;  // Q: 32 rows at a time, 4 float4 of a row
  const int vc = tid % TW, vr = tid / TW;    // V: 128 / TW rows at a time
  const bool v_ok = c0 + vc < k;
  auto fetch = [&](int j) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int64_t i = i0 + qi + 32 * h;
      qn[h] = (i < n && j + qg < nq) ? *reinterpret_cast<const float4*>(Q + i * ldq + j + qg)
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int h = 0; h < CT; ++h) {
      const int jr = j + vr + (kGThreads / TW) * h;
      vn[h] = (jr < nr && v_ok) ? (float)V[(int64_t)jr * k + c0 + vc] : 0.0f;
    }
  };
  auto store = [&](int b) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      Qs[b][qg + 0][qi + 32 * h] = qn[h].x;
      Qs[b][qg + 1][qi + 32 * h] = qn[h].y;
      Qs[b][qg + 2][qi + 32 * h] = qn[h].z;
      Qs[b][qg + 3][qi + 32 * h] = qn[h].w;
    }
#pragma unroll
    for (int h = 0; h < CT; ++h) Vs[b][vr + (kGThreads / TW) * h][vc] = vn[h];
  };
  if (nr > 0) {
    fetch(0);
    store(0);
  }
  __syncthreads();
  int b = 0;
  for (int j = 0; j < nr; j += kGK, b ^= 1) {
    const bool more = j + kGK < nr;
    if (more) fetch(j + kGK);
    pcm_step<CT>(Qs[b], Vs[b], ty, tx, acc);
    if (more) store(b ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int64_t i = i0 + pcm_row(ty, u);
    if (i >= n) continue;
#pragma unroll
    for (int v = 0; v < CT; ++v) {
      const int c = c0 + pcm_col<CT>(tx, v);
      if (c < k) {
        const int64_t e = i * k + c;
        Z[e] = (ZT)(cis * R[e] + (double)(v & 1 ? acc[u][v / 2].y : acc[u][v / 2].x));
      }
    }
  }
}

// Columns of Q the apply reads: N_r rounded up to a float4.
int pcm_cols(int nr) { return (int)round_up(nr, 4); }

// Columns per thread of the apply's tiles.  Wide tiles load less per FMA, but where
// the expansion has few of them a CTA's chain of steps is what takes the time: a width
// is passed over for the next only when it gives more than 3 (16 columns) or 4 (32)
// CTAs per SM.  us at widths 16 / 32 / 64: n = 1,000, N_r = 32, k = 64 23 / 27 / 40;
// n = 5,000, N_r = 200, k = 64 49 / 55 / 74, k = 200 73 / 64 / 94; n = 20,000,
// N_r = 200, k = 64 79 / 78 / 90, k = 100 128 / 112 / 119, k = 200 206 / 185 / 185.
// With 64 columns whenever k > 32 the smallest applies were slower than the 64 x 64
// tiles before (n = 1,000, N_r = 32, k = 64: 29 us).
int pcm_ct(int64_t n, int k) {
  const int64_t rows = ceil_div(n, kGT), sms = sm_count();
  if (k <= 16 || rows * ceil_div(k, 16) <= 3 * sms) return 2;
  if (k <= 32 || rows * ceil_div(k, 32) <= 4 * sms) return 4;
  return 8;
}

int pcm_tiles(int64_t n, int nq, int k) {
  return (int)(ceil_div(nq, kGT) * ceil_div(k, 8 * pcm_ct(n, k)));
}

int pcm_chunks(int64_t n, int nq, int k) {
  int64_t c = ceil_div(2 * (int64_t)sm_count(), pcm_tiles(n, nq, k));
  const int64_t lim = ceil_div(n, 256);
  if (c > lim) c = lim;
  if (c > 64) c = 64;
  return (int)(c < 1 ? 1 : c);
}

}  // namespace

size_t precond_multi_scratch_bytes(int64_t n, int nr, int k) {
  const int nq = pcm_cols(nr);
  const int nch = pcm_chunks(n, nq, k);
  return (size_t)round_up((int64_t)((size_t)nch * nq * k * sizeof(double)), 256) +
         2 * (size_t)round_up((int64_t)((size_t)nq * k * sizeof(double)), 256);
}

template <typename ZT>
cudaError_t launch_precond_multi(const laker_precond* pc, const double* R, int k, ZT* Z,
                                 void* scratch, const int* gate, cudaStream_t s) {
  const int64_t n = pc->n;
  const int ldq = pc->ldq, nr = pc->nr, nq = pcm_cols(nr);
  const int nch = pcm_chunks(n, nq, k);
  double* upart = static_cast<double*>(scratch);
  double* V = reinterpret_cast<double*>(static_cast<char*>(scratch) +
                                        round_up((int64_t)((size_t)nch * nq * k * sizeof(double)), 256));
  const int64_t chunk_rows = round_up(ceil_div(n, nch), kGK);
  const int ct = pcm_ct(n, k);
  const unsigned gy = (unsigned)ceil_div(k, 8 * ct);
  const dim3 pg((unsigned)ceil_div(nq, kGT), gy, (unsigned)nch), eg((unsigned)ceil_div(n, kGT), gy);
  auto project = ct == 2 ? pcm_project_kernel<2> : ct == 4 ? pcm_project_kernel<4> : pcm_project_kernel<8>;
  auto expand = ct == 2 ? pcm_expand_kernel<2, ZT> : ct == 4 ? pcm_expand_kernel<4, ZT> : pcm_expand_kernel<8, ZT>;
  project<<<pg, kGThreads, 0, s>>>(pc->q_basis, ldq, nq, R, n, k, chunk_rows, upart, gate);
  double* U = V + round_up((int64_t)nq * k, 32);
  const int64_t total = (int64_t)nq * k;
  pcm_sum_kernel<<<(unsigned)ceil_div(total, kMT), kMT, 0, s>>>(upart, nch, total, U, gate);
  pcm_core_kernel<<<dim3((unsigned)ceil_div(nq, kCoreJ), (unsigned)ceil_div(k, kCoreC)), kMT, 0, s>>>(
      pc->w_core, nr, nq, U, k, V, gate);
  expand<<<eg, kGThreads, 0, s>>>(pc->q_basis, ldq, nq, nr, V, R, pc->inv_sqrt_iso, n, k, Z, gate);
  return cudaGetLastError();
}

template cudaError_t launch_precond_multi<float>(const laker_precond*, const double*, int, float*,
                                                 void*, const int*, cudaStream_t);
template cudaError_t launch_precond_multi<double>(const laker_precond*, const double*, int, double*,
                                                  void*, const int*, cudaStream_t);

// ---------------------------------------------------------------------------
// The multi-RHS solve.
// ---------------------------------------------------------------------------
namespace {

struct MpcgWs {
  WsHeader* hdr;
  MpcgState* st;
  MpcgCols cols;
  double* R;
  float* P;
  float* AP;
  float* Z;
  double* bp;
  void* pscratch;
  uint8_t* img;  // operator scratch: FP32 products and, at other times, the FP64 residual
  size_t img_bytes;
  size_t bytes;
};

// Graph of one iteration (released when the solve returns).
struct MpcgGraph {
  cudaStream_t cap = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  ~MpcgGraph() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (cap) cudaStreamDestroy(cap);
  }
};

MpcgWs carve_multi(void* base, int64_t n, int k, int nr) {
  MpcgWs w{};
  char* p = static_cast<char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = p ? p + off : nullptr;
    off += (size_t)round_up((int64_t)bytes, 256);
    return q;
  };
  const size_t nk = (size_t)n * (size_t)k;
  const ColGrid g = col_grid(n, k);
  w.hdr = reinterpret_cast<WsHeader*>(take(kWsHeader));
  w.st = reinterpret_cast<MpcgState*>(take(sizeof(MpcgState)));
  w.cols.bnorm = reinterpret_cast<double*>(take((size_t)k * sizeof(double)));
  w.cols.rz = reinterpret_cast<double*>(take((size_t)k * sizeof(double)));
  w.cols.alpha = reinterpret_cast<double*>(take((size_t)k * sizeof(double)));
  w.cols.beta = reinterpret_cast<double*>(take((size_t)k * sizeof(double)));
  w.cols.rn = reinterpret_cast<double*>(take((size_t)k * sizeof(double)));
  w.cols.live = reinterpret_cast<int*>(take((size_t)k * sizeof(int)));
  w.cols.ypart = reinterpret_cast<double*>(take((size_t)kMKinds * g.gy * 3 * sizeof(double)));
  w.cols.yctr = reinterpret_cast<unsigned int*>(take((size_t)kMKinds * g.gy * sizeof(unsigned int)));
  w.R = reinterpret_cast<double*>(take(nk * sizeof(double)));
  w.P = reinterpret_cast<float*>(take(nk * sizeof(float)));
  w.AP = reinterpret_cast<float*>(take(nk * sizeof(float)));
  w.Z = reinterpret_cast<float*>(take(nk * sizeof(float)));
  w.bp = reinterpret_cast<double*>(take((size_t)3 * g.gx * (size_t)k * sizeof(double)));
  w.pscratch = nr > 0 ? take(precond_multi_scratch_bytes(n, nr, k)) : nullptr;
  {
    // operator workspace: the tensor-core multi-RHS kernels' operand images
    size_t b = k2_use_tensor_cores() ? k2_image_bytes(n, n, k) : 0;
    const size_t bf = k2f_reserve_bytes(n, n, k, true);
    if (bf > b) b = bf;
    const size_t avail = b > kSegScratch ? b : kSegScratch;
    const size_t u32 = k2f_enabled(k, 0) ? k2f_workspace_bytes(n, n, k, true, avail) : 0;
    const size_t u64 = f64m_workspace_bytes(n, n, k, avail);
    if (u32 > b) b = u32;
    if (u64 > b) b = u64;
    w.img = reinterpret_cast<uint8_t*>(take(b));
    w.img_bytes = b;
  }
  w.bytes = off;
  return w;
}

}  // namespace

size_t pcg_multi_workspace_bytes(int64_t n, int d, int nr, int k) {
  (void)d;
  return carve_multi(nullptr, n, k, nr).bytes;
}

int pcg_solve_multi(const laker_operator* op, const laker_precond* pc, const double* B, int k,
                    double* X, const laker_pcg_params* prm, void* workspace, laker_pcg_result* res,
                    cudaStream_t s) {
  const int64_t n = op->n;
  const int d = op->d;
  const int nr = pc ? pc->nr : 0;
  MpcgWs w = carve_multi(workspace, n, k, nr);
  const ColGrid g = col_grid(n, k);
  const dim3 cgrid((unsigned)g.gx, (unsigned)g.gy);
  int* dstatus = &w.hdr->status;
  const float lam32 = (float)op->lambda_reg;

  *res = laker_pcg_result{};
  MpcgState h{};
  h.tol = prm->tol;
  h.delta = prm->reliable_delta;
  h.eps = prm->breakdown_eps;
  h.max_iter = prm->max_iter;
  h.active = 1;
  h.column_stop = prm->column_stop ? 1 : 0;
  cudaError_t e = cudaMemsetAsync(w.hdr, 0, kWsHeader, s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(w.cols.yctr, 0, (size_t)kMKinds * g.gy * sizeof(unsigned int), s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w.st, &h, sizeof(MpcgState), cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return fail_cuda(e);

  int launches = 0;
  // R = B - A64 X (gated by `gate`; ungated for the warm start)
  auto launch_residual = [&](int init, const int* gate, cudaStream_t cs) -> cudaError_t {
    cudaError_t ee = launch_multi_f64(op->packed64, n, op->packed64, n, d, op->lambda_reg, op->clamp,
                                      X, k, k, B, k, w.R, k, reinterpret_cast<double*>(w.img),
                                      w.img_bytes, cs, gate);
    if (ee == cudaSuccess)
      mp_after_residual_kernel<<<cgrid, kMT, 0, cs>>>(w.R, n, k, init, w.bp, w.st, w.cols);
    launches += f64m_workspace_bytes(n, n, k, w.img_bytes) > 0 ? 3 : 2;
    return ee;
  };
  auto launch_precond = [&](int init, cudaStream_t cs) -> cudaError_t {
    cudaError_t ee = cudaSuccess;
    if (pc) {
      ee = launch_precond_multi<float>(pc, w.R, k, w.Z, w.pscratch, &w.st->active, cs);
      mp_after_precond_kernel<false><<<cgrid, kMT, 0, cs>>>(w.R, w.Z, n, k, init, w.bp, w.st, w.cols);
      launches += 5;
    } else {
      mp_after_precond_kernel<true><<<cgrid, kMT, 0, cs>>>(w.R, w.Z, n, k, init, w.bp, w.st, w.cols);
      launches += 1;
    }
    mp_update_p_kernel<<<cgrid, kMT, 0, cs>>>(w.Z, w.P, n, k, w.st, w.cols, init);
    launches += 1;
    return ee;
  };

  // ---- initialisation ------------------------------------------------------
  mp_init_kernel<<<cgrid, kMT, 0, s>>>(B, X, w.R, n, k, prm->has_x0, w.bp, w.st, w.cols);
  launches += 1;
  e = cudaGetLastError();
  if (e == cudaSuccess && prm->has_x0) e = launch_residual(1, nullptr, s);
  if (e != cudaSuccess) return fail_cuda(e);
  e = cudaMemcpyAsync(&h, w.st, sizeof(MpcgState), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail_cuda(e);
  res->rhs_norm = h.bnorm;
  res->kernel_launches = launches;
  if (h.bnorm == 0.0) {
    // zero right-hand side: X is returned unchanged (zero, or the warm start)
    res->status = LAKER_OK;
    res->residual_norm = 0.0;
    return LAKER_OK;
  }
  if (h.done) {
    res->status = h.status;
    res->residual_norm = h.true_rnorm;
    return h.status;
  }
  e = launch_precond(1, s);
  if (e != cudaSuccess) return fail_cuda(e);

  // ---- iterations ------------------------------------------------------------
  auto iteration = [&](cudaStream_t cs) -> cudaError_t {
    cudaError_t ee;
    if (k2f_enabled(k, op->clamp)) {
      ee = launch_k2f(op->packed32, n, op->packed32, n, d, lam32, w.P, k, k, w.AP, k, w.img,
                      w.img_bytes, dstatus, cs, &w.st->active);
      launches += 4;
    } else if (k2_use_tensor_cores()) {
      ee = launch_k2(op->packed32, n, op->packed32, n, d, op->clamp, lam32, w.P, k, k, w.AP, k, w.img,
                     dstatus, cs, &w.st->active);
      launches += 3;
    } else {
      ee = launch_multi_f32(op->packed32, n, op->packed32, n, d, lam32, op->clamp, w.P, k, k, w.AP, k,
                            cs, &w.st->active);
      launches += 1;
    }
    if (ee != cudaSuccess) return ee;
    mp_after_matvec_kernel<<<cgrid, kMT, 0, cs>>>(w.P, w.AP, n, k, w.bp, w.st, w.cols, dstatus);
    mp_update_xr_kernel<<<cgrid, kMT, 0, cs>>>(w.P, w.AP, X, w.R, n, k, w.bp, w.st, w.cols);
    launches += 2;
    ee = launch_residual(0, &w.st->need_update, cs);
    if (ee != cudaSuccess) return ee;
    return launch_precond(0, cs);
  };
  MpcgGraph ig;
  int iter_launches = 0;
  {
    const int before = launches;
    e = cudaStreamCreateWithFlags(&ig.cap, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamBeginCapture(ig.cap, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      const cudaError_t ie = iteration(ig.cap);
      const cudaError_t ce = cudaGetLastError();
      e = cudaStreamEndCapture(ig.cap, &ig.graph);
      if (e == cudaSuccess) e = ie != cudaSuccess ? ie : ce;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&ig.exec, ig.graph, 0);
    if (e != cudaSuccess) return fail_cuda(e);
    iter_launches = launches - before;
    launches = before;
  }
  // Polls: the first after one iteration, whose host-measured time sets the
  // replays between later polls (about 10 ms of work, at most 64).
  int check = prm->check_every > 0 ? prm->check_every : 1;
  bool calibrate = prm->check_every <= 0;
  int launched = 0;
  while (launched < prm->max_iter) {
    const int chunk = (prm->max_iter - launched) < check ? (prm->max_iter - launched) : check;
    const auto t0 = std::chrono::steady_clock::now();
    for (int c = 0; c < chunk; ++c) {
      e = cudaGraphLaunch(ig.exec, s);
      if (e != cudaSuccess) return fail_cuda(e);
      launches += iter_launches;
    }
    launched += chunk;
    e = cudaMemcpyAsync(&h, w.st, sizeof(MpcgState), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail_cuda(e);
    if (h.done) break;
    if (calibrate) {
      const double dt = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
      const double per = dt / chunk;
      check = per > 0.0 ? (int)(0.01 / per) : 64;
      if (check < 1) check = 1;
      if (check > 64) check = 64;
      calibrate = false;
    }
  }

  int dev_status = 0;
  e = cudaMemcpyAsync(&dev_status, dstatus, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail_cuda(e);
  res->iterations = h.iter;
  res->accurate_matvecs = h.n_accurate;
  res->residual_norm = h.true_rnorm;
  res->recurrence_norm = h.rnorm;
  res->rhs_norm = h.bnorm;
  res->kernel_launches = launches;
  if (dev_status != 0) {
    res->status = dev_status;
    return dev_status;
  }
  if (!h.done) {
    res->status = LAKER_ERR_NOT_CONVERGED;
    return LAKER_ERR_NOT_CONVERGED;
  }
  res->status = h.status;
  return h.status;
}

}  // namespace laker
