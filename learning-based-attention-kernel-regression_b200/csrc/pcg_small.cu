// Small single-RHS solves (n <= 3072) as one cooperative kernel.
//
// The iteration of pcg.cu is about eight kernels; at n = 2000 each lasts 3 to 30 us
// of which most is launch, fill and a last block's serial tail, 66 us together
// against 1 us of operator arithmetic.  Here the whole solve is one launch of at most
// one CTA per SM that keeps its operands on chip -- every CTA holds all FP32
// embeddings and the direction p in shared memory, and its own rows of Q and Q W --
// and exchanges scalars and short vectors through L2 between four grid barriers per
// iteration:
//   1. Ap of the own rows; p.Ap, |p|^2, |Ap|^2             -> barrier, alpha
//   2. x += alpha p, r -= alpha Ap; |r|^2 and Q_own^T r     -> barrier
//   3. u = sum of the CTAs' Q^T r, a few columns per CTA    -> barrier, |r|
//   4. z = c^-1/2 r + (Q W)_own u; r.z                      -> barrier, beta
//   5. p = z + beta p, all of it, in every CTA.
// When |r| asks for it (the reliable update and stop test of pcg.cu), x is published
// and r = b - A64 x is recomputed for the own rows before 3 is done again.
// Every CTA adds the same partial sums in the same order, so all take the same
// decisions without a broadcast, and a solve gives the same bits every time.
//
// Precision: as pcg.cu (FP32 entries, p, z, Ap; FP64 x, r, dots, residuals); the
// preconditioner is applied in FP64 from the FP32 factors (pcg.cu: FP32 products).
//
// n = 2000 (N_r = 200, tol 1e-10): 18.0 -> 6.4 ms, 66 -> 19 us per iteration; n = 500:
// 12 us, n = 3000: 24 us.  About 10 us of an iteration is the chain of four barriers and
// the L2 round trips between them (a 40-point solve takes that), the rest the operator
// on the CUDA cores (6 us at n = 3000).  Measured the same: 16 warps per CTA, three rows
// per warp throughout, sleeping between polls.  The line at n = 3072 is where the
// points no longer fit and the symmetric tensor-core operator takes over.
//
// Grid barriers are bounded waits: a CTA that gives up records LAKER_ERR_TIMEOUT and
// raises a flag that the others' waits see; all leave.
#include <cstring>

#include "pcg_state.cuh"

namespace laker {
namespace {

constexpr int kSWarps = 8, kSThreads = kSWarps * 32;
constexpr int kSMaxRows = 3;  // rows per warp
constexpr int kSMaxTiles = 16;

struct None {
  static constexpr int value = 0;
};
struct One {
  static constexpr int value = 1;
};
struct Three {
  static constexpr int value = 3;
};

struct SmallArgs {
  const float* E32;
  const double* E64;
  int64_t n;
  int clamp, has_x0, max_iter;
  double lam, tol, delta, eps;
  PcView pc;  // nr == 0: no preconditioner
  const double* b;
  double* x;
  // exchange through L2
  double *dots, *rr, *rzp, *upart, *u;
  float* z;
  unsigned int* bar;  // [0] arrivals, [1] abort flag
  PcgState* st;
  int* status;
};

// Shared-memory plan (bytes from a 128-byte aligned base).
struct SmallSmem {
  uint32_t off_p, off_q, off_qw, off_u, total;
};

__host__ __device__ inline SmallSmem small_smem(int64_t n, int dp, int rows, int nr, int ldq) {
  const uint32_t pts = (uint32_t)ceil_div(n, kTileCols32) * kTileCols32;
  SmallSmem s;
  s.off_p = pts / 2 * pair_stride(dp) * 4;
  s.off_qw = s.off_p + pts * 4;
  s.off_u = s.off_qw + (uint32_t)rows * (uint32_t)nr * 8;
  s.off_q = s.off_u + (uint32_t)nr * 8;
  s.total = s.off_q + (uint32_t)rows * (uint32_t)ldq * 4 + 128;
  return s;
}

template <int DP, int R>
__global__ void __launch_bounds__(kSThreads, 1) pcg_small_kernel(SmallArgs a) {
  constexpr int ROWS = kSWarps * R;
  constexpr int TC = kTileCols32;
  constexpr int PS = pair_stride(DP);
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int nr = a.pc.nr, ldq = a.pc.ldq;
  const SmallSmem L = small_smem(a.n, DP, ROWS, nr, ldq);
  float* sP = reinterpret_cast<float*>(sm + L.off_p);
  double* sQW = reinterpret_cast<double*>(sm + L.off_qw);  // [ROWS][nr]
  double* sU = reinterpret_cast<double*>(sm + L.off_u);
  float* sQ = reinterpret_cast<float*>(sm + L.off_q);      // [ROWS][ldq]
  __shared__ __align__(8) uint64_t bar;
  __shared__ double sExp[64];
  __shared__ double sRed[3 * kSWarps];
  __shared__ double sR[ROWS], sScal[3];
  __shared__ int sOk;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = gridDim.x;
  const int64_t n = a.n;
  const int ntiles = (int)ceil_div(n, TC);
  const int row0 = blockIdx.x * ROWS;

  if (tid == 0) {
    sOk = 1;
    mbar_init(&bar, kSThreads);
    mbar_fence_init();
  }
  __syncthreads();
  stage_pairs<DP, kSThreads>(reinterpret_cast<float*>(sm), a.E32, ntiles * (TC / 2), &bar, tid);
  exp_table_to_shared(sExp, tid, kSThreads);
  for (int e = tid; e < ROWS * ldq; e += kSThreads) {
    const int i = e / ldq;
    sQ[e] = nr > 0 && row0 + i < n ? a.pc.Q[(int64_t)(row0 + i) * ldq + (e - i * ldq)] : 0.0f;
  }
  __syncthreads();

  // rows of this warp: row0 + warp R .. + R - 1
  const int i0 = row0 + warp * R;
  float2 ev[R][DP];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = i0 + r;
    const float* blk = a.E32 + (int64_t)(i >> 1) * (DP * 2) + (i & 1);
#pragma unroll
    for (int k = 0; k < DP; ++k) {
      const float v = i < n ? blk[2 * k] * kLog2e : 0.0f;
      ev[r][k] = make_float2(v, v);
    }
  }
  // (Q W) of the own rows, FP64
  for (int c = tid; c < nr; c += kSThreads) {
    double acc[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) acc[i] = 0.0;
    for (int k = 0; k < nr; ++k) {
      const double w = (double)__ldg(a.pc.W + (int64_t)k * nr + c);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) acc[i] = fma((double)sQ[i * ldq + k], w, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) sQW[i * nr + c] = acc[i];
  }

  if (!mbar_wait_bounded(&bar, 0u, a.status)) {
    asm volatile("cp.async.wait_all;" ::: "memory");  // its copies land before it exits
    sOk = 0;
    atomicExch(&a.bar[1], 1u);
  }

  // Grid barrier number `phase` (from 1), by warp 0; the other warps wait for it.
  // False when this or another CTA gave up; uniform over the CTA.  Writes before it
  // are visible to reads (ld.cg) after it.  With NQ > 0, warp 0 then adds the CTAs'
  // values v[NQ cta + q] (a fixed order, the same in every CTA) into t3 for all
  // threads: only one warp per CTA touches those lines.
  unsigned int phase = 0;
  double t3[3] = {0.0, 0.0, 0.0};
  auto grid_sync = [&](const double* v, auto nq) -> bool {
    constexpr int NQ = decltype(nq)::value;
    ++phase;
    __syncthreads();
    if (warp == 0) {
      if (lane == 0 && sOk) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        const unsigned int target = phase * (unsigned int)G;
        const unsigned long long limit = wait_limit_ns();
        uint64_t t0 = 0;  // the first polls usually find the barrier complete
        bool done = false;
        for (uint32_t it = 0; it < (1u << 30) && limit != 0; ++it) {
          unsigned int n_arrived;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n_arrived) : "l"(a.bar) : "memory");
          if ((int)(n_arrived - target) >= 0) {
            done = true;
            break;
          }
          if ((it & 63u) == 63u) {
            if (*reinterpret_cast<volatile unsigned int*>(a.bar + 1)) break;
            const uint64_t now = global_timer_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 >= limit) break;
          }
        }
        if (!done) {
          record_status(a.status, LAKER_ERR_TIMEOUT);
          atomicExch(&a.bar[1], 1u);
          sOk = 0;
        }
      }
      __syncwarp();
      if constexpr (NQ > 0) {
        double t[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) t[q] = 0.0;
        for (int c = lane; c < G; c += 32)
#pragma unroll
          for (int q = 0; q < NQ; ++q) t[q] += __ldcg(v + NQ * c + q);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          t[q] = warp_sum(t[q]);
          if (lane == 0) sScal[q] = t[q];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) t3[q] = sScal[q];
    return sOk != 0;
  };

  // Lane 0 of each warp holds x, r, b, p, Ap of the warp's rows.
  double xv[R], rv[R], bv[R];
  float ap[R];
  auto own = [&](int r) { return i0 + r < n; };
#pragma unroll
  for (int r = 0; r < R; ++r) {
    bv[r] = own(r) ? a.b[i0 + r] : 0.0;
    xv[r] = own(r) && a.has_x0 ? a.x[i0 + r] : 0.0;
    rv[r] = bv[r];
    ap[r] = 0.0f;
  }
  // |r|^2 and Q_own^T r of this CTA into rr and upart
  auto publish_r = [&]() {
    double rr = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) rr = fma(rv[r], rv[r], rr);
    if (lane == 0) {
      sRed[warp] = rr;
#pragma unroll
      for (int r = 0; r < R; ++r) sR[warp * R + r] = rv[r];
    }
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kSWarps; ++w) s += sRed[w];
      __stcg(a.rr + blockIdx.x, s);
    }
    for (int c = tid; c < nr; c += kSThreads) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < ROWS; ++i) s = fma((double)sQ[i * ldq + c], sR[i], s);
      __stcg(a.upart + (int64_t)blockIdx.x * nr + c, s);
    }
    __syncthreads();
  };
  // u[c] for this CTA's share of the columns: one warp per column
  auto reduce_u = [&]() {
    for (int c = blockIdx.x + warp * G; c < nr; c += G * kSWarps) {
      double s = 0.0;
      for (int q = lane; q < G; q += 32) s += __ldcg(a.upart + (int64_t)q * nr + c);
      s = warp_sum(s);
      if (lane == 0) __stcg(a.u + c, s);
    }
  };
  // r = b - (lam x + K64 x) of the own rows from the published x
  auto residual = [&]() {
    double acc[R];
    double er[R][DP];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      acc[r] = 0.0;
#pragma unroll
      for (int k = 0; k < DP; ++k) er[r][k] = own(r) ? __ldg(a.E64 + (int64_t)(i0 + r) * DP + k) : 0.0;
    }
    for (int64_t j = lane; j < n; j += 32) {
      const double2* cp = reinterpret_cast<const double2*>(a.E64 + j * DP);
      double c[DP];
#pragma unroll
      for (int h = 0; h < DP / 2; ++h) {
        const double2 v = __ldg(cp + h);
        c[2 * h] = v.x;
        c[2 * h + 1] = v.y;
      }
      const double xj = __ldcg(a.x + j);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double s = er[r][0] * c[0];
#pragma unroll
        for (int k = 1; k < DP; ++k) s = fma(er[r][k], c[k], s);
        if (a.clamp) s = fmin(s, kClamp64);
        acc[r] = fma(exp_tab(s, sExp), xj, acc[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const double k = warp_sum(acc[r]);
      rv[r] = own(r) ? bv[r] - fma(a.lam, xv[r], k) : 0.0;
    }
  };
  auto publish_x = [&]() {
    if (lane == 0)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (own(r)) __stcg(a.x + i0 + r, xv[r]);
  };

  // state shared by all CTAs (each computes the same values)
  double bnorm = 0.0, rz = 0.0, rn = 0.0, rmax = 0.0, true_rn = 0.0;
  int iter = 0, n_acc = 0, status = LAKER_ERR_NOT_CONVERGED, finished = 0;

  // |b|
  publish_r();
  bool go = grid_sync(a.rr, One{});
  if (go) {
    bnorm = sqrt(t3[0]);
    rn = rmax = true_rn = bnorm;
    if (!isfinite(bnorm)) status = LAKER_ERR_NONFINITE, finished = 1;
    else if (bnorm == 0.0) status = LAKER_OK, finished = 1;
    if (!finished && a.has_x0) {
      // warm start: r = b - A x0 with the FP64 operator (x0 is in a.x already)
      residual();
      go = grid_sync(nullptr, None{});  // every CTA has read rr and x0
      if (go) {
        publish_r();
        go = grid_sync(a.rr, One{});
      }
      if (go) {
        rn = rmax = true_rn = sqrt(t3[0]);
        ++n_acc;
        if (!isfinite(rn)) status = LAKER_ERR_NONFINITE, finished = 1;
      }
    }
  }
  const double tol_abs = a.tol * bnorm;
  bool first = true;
  while (go && !finished) {
    if (!first) {
      // 1. operator on the own rows
      float2 acc[R];
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = make_float2(0.0f, 0.0f);
      const float2* P2 = reinterpret_cast<const float2*>(sP);
#pragma unroll 2
      for (int q = lane; q < ntiles * (TC / 2); q += 32) {
        const float4* cp = reinterpret_cast<const float4*>(sm) + q * (PS / 4);
        float2 c[DP];
#pragma unroll
        for (int h = 0; h < DP / 2; ++h) {
          const float4 v = cp[h];
          c[2 * h] = make_float2(v.x, v.y);
          c[2 * h + 1] = make_float2(v.z, v.w);
        }
        const float2 xv2 = P2[q];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float2 s = __fmul2_rn(ev[r][0], c[0]);
#pragma unroll
          for (int k = 1; k < DP; ++k) s = __ffma2_rn(ev[r][k], c[k], s);
          if (a.clamp) {
            s.x = fminf(s.x, kClampLog2);
            s.y = fminf(s.y, kClampLog2);
          }
          acc[r] = __ffma2_rn(make_float2(ex2_approx(s.x), ex2_approx(s.y)), xv2, acc[r]);
        }
      }
      double d[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double s = warp_sum((double)acc[r].x + (double)acc[r].y);
        const double pi = own(r) ? (double)sP[i0 + r] : 0.0;
        ap[r] = own(r) ? (float)(a.lam * pi + s) : 0.0f;
        d[0] = fma(pi, (double)ap[r], d[0]);
        d[1] = fma(pi, pi, d[1]);
        d[2] = fma((double)ap[r], (double)ap[r], d[2]);
      }
      if (lane == 0)
#pragma unroll
        for (int q = 0; q < 3; ++q) sRed[q * kSWarps + warp] = d[q];
      __syncthreads();
      if (tid < 3) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kSWarps; ++w) s += sRed[tid * kSWarps + w];
        __stcg(a.dots + 3 * blockIdx.x + tid, s);
      }
      if (!(go = grid_sync(a.dots, Three{}))) break;
      if (!isfinite(t3[0]) || !isfinite(t3[1]) || !isfinite(t3[2])) {
        status = LAKER_ERR_NONFINITE;
        break;
      }
      if (t3[0] <= -a.eps * sqrt(t3[1]) * sqrt(t3[2])) {
        status = LAKER_ERR_BREAKDOWN;  // non-positive curvature
        break;
      }
      const double alpha = rz / t3[0];
      // 2. x, r
#pragma unroll
      for (int r = 0; r < R; ++r) {
        xv[r] = fma(alpha, own(r) ? (double)sP[i0 + r] : 0.0, xv[r]);
        rv[r] = fma(-alpha, (double)ap[r], rv[r]);
      }
      publish_r();
      if (!(go = grid_sync(a.rr, One{}))) break;
      // 3. |r| and the decision
      rn = sqrt(t3[0]);
      ++iter;
      if (rn > rmax) rmax = rn;
      if (rn <= a.delta * rmax || rn <= tol_abs || iter >= a.max_iter || !isfinite(rn)) {
        publish_x();
        if (!(go = grid_sync(nullptr, None{}))) break;
        residual();
        publish_r();
        if (!(go = grid_sync(a.rr, One{}))) break;
        const double tr = sqrt(t3[0]);
        rn = rmax = true_rn = tr;
        ++n_acc;
        if (!isfinite(tr)) {
          status = LAKER_ERR_NONFINITE;
          break;
        }
        if (tr <= tol_abs) {
          status = LAKER_OK;
          break;
        }
        if (iter >= a.max_iter) break;  // LAKER_ERR_NOT_CONVERGED
      }
    } else if (a.max_iter < 1) {
      break;
    }
    if (nr > 0) {
      reduce_u();
      if (!(go = grid_sync(nullptr, None{}))) break;
      for (int c = tid; c < nr; c += kSThreads) sU[c] = __ldcg(a.u + c);
      __syncthreads();
    }
    // 4. z, r.z
    double rzp = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double s = 0.0;
      for (int c = lane; c < nr; c += 32) s = fma(sQW[(warp * R + r) * nr + c], sU[c], s);
      s = warp_sum(s);
      const float zi = own(r) ? (float)(nr > 0 ? fma(a.pc.cis, rv[r], s) : rv[r]) : 0.0f;
      rzp = fma(rv[r], (double)zi, rzp);
      if (lane == 0 && own(r)) __stcg(a.z + i0 + r, zi);
    }
    if (lane == 0) sRed[warp] = rzp;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < kSWarps; ++w) s += sRed[w];
      __stcg(a.rzp + blockIdx.x, s);
    }
    if (!(go = grid_sync(a.rzp, One{}))) break;
    if (!isfinite(t3[0])) {
      status = LAKER_ERR_NONFINITE;
      break;
    }
    // 5. p
    const float beta = first ? 0.0f : (float)(t3[0] / rz);
    rz = t3[0];
    for (int j = tid; j < ntiles * TC; j += kSThreads) {
      const float zj = j < n ? __ldcg(a.z + j) : 0.0f;
      sP[j] = first ? zj : fmaf(beta, sP[j], zj);
    }
    __syncthreads();
    first = false;
  }
  if (bnorm != 0.0 || !a.has_x0) publish_x();  // a zero right-hand side leaves x0
  if (blockIdx.x == 0 && tid == 0) {
    a.st->bnorm = bnorm;
    a.st->rnorm = rn;
    a.st->true_rnorm = true_rn;
    a.st->iter = iter;
    a.st->n_accurate = n_acc;
    a.st->status = status;
    a.st->done = 1;
  }
}

int small_rows(int64_t n) {
  const int64_t r = ceil_div(n, (int64_t)kSWarps * sm_count());
  return r <= 1 ? 1 : r == 2 ? 2 : 3;
}

template <int DP, int R>
cudaError_t launch_small(const SmallArgs& a, int grid, uint32_t smem, cudaStream_t s) {
  static SmemOptIn optin;
  const cudaError_t e = optin.allow(pcg_small_kernel<DP, R>, 224 * 1024);
  if (e != cudaSuccess) return e;
  SmallArgs args = a;
  void* params[] = {&args};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&pcg_small_kernel<DP, R>), dim3(grid),
                                     dim3(kSThreads), params, smem, s);
}

template <int DP>
cudaError_t launch_small_r(int rows, const SmallArgs& a, int grid, uint32_t smem, cudaStream_t s) {
  switch (rows) {
    case 1: return launch_small<DP, 1>(a, grid, smem, s);
    case 2: return launch_small<DP, 2>(a, grid, smem, s);
    default: return launch_small<DP, 3>(a, grid, smem, s);
  }
}

}  // namespace

// Whether a solve takes the one-kernel form: at most three rows per warp of one
// CTA per SM, the embeddings and the CTA's rows of Q and Q W within shared memory.
bool pcg_small_fits(int64_t n, int d, int nr, int ldq) {
  if (n < 1 || n > (int64_t)kSMaxTiles * kTileCols32) return false;
  if (ceil_div(n, (int64_t)kSWarps * sm_count()) > kSMaxRows) return false;
  return small_smem(n, padded_dim(d), kSWarps * small_rows(n), nr, nr > 0 ? ldq : 0).total <= 224 * 1024;
}

// header | state | barrier | dots, rr, rz (per CTA) | upart | u | z
size_t pcg_small_workspace_bytes(int64_t n, int nr) {
  const size_t G = (size_t)sm_count();
  return kWsHeader + sizeof(PcgState) + 256 +
         (size_t)round_up((int64_t)(8 * (5 * G + (G + 1) * (size_t)nr)), 256) +
         (size_t)round_up(n * 4, 256);
}

int pcg_solve_small(const laker_operator* op, const laker_precond* pc, const double* B, double* X,
                    const laker_pcg_params* prm, void* workspace, laker_pcg_result* res,
                    cudaStream_t s) {
  const int64_t n = op->n;
  const int nr = pc ? pc->nr : 0, ldq = pc ? pc->ldq : 0;
  const int rows = small_rows(n), grid = (int)ceil_div(n, kSWarps * rows);
  char* p = static_cast<char*>(workspace);
  WsHeader* hdr = reinterpret_cast<WsHeader*>(p);
  PcgState* st = reinterpret_cast<PcgState*>(p + kWsHeader);
  SmallArgs a{};
  a.E32 = op->packed32;
  a.E64 = op->packed64;
  a.n = n;
  a.clamp = op->clamp;
  a.has_x0 = prm->has_x0;
  a.max_iter = prm->max_iter;
  a.lam = op->lambda_reg;
  a.tol = prm->tol;
  a.delta = prm->reliable_delta;
  a.eps = prm->breakdown_eps;
  a.pc = PcView{pc ? pc->q_basis : nullptr, pc ? pc->w_core : nullptr, n, nr, ldq,
                pc ? pc->inv_sqrt_iso : 1.0};
  a.b = B;
  a.x = X;
  a.bar = reinterpret_cast<unsigned int*>(p + kWsHeader + sizeof(PcgState));
  a.dots = reinterpret_cast<double*>(p + kWsHeader + sizeof(PcgState) + 256);
  const size_t G = (size_t)sm_count();
  a.rr = a.dots + 3 * G;
  a.rzp = a.rr + G;
  a.upart = a.rzp + G;
  a.u = a.upart + G * (size_t)nr;
  a.z = reinterpret_cast<float*>(reinterpret_cast<char*>(a.dots) +
                                 round_up((int64_t)(8 * (5 * G + (G + 1) * (size_t)nr)), 256));
  a.st = st;
  a.status = &hdr->status;
  *res = laker_pcg_result{};
  cudaError_t e = cudaMemsetAsync(p, 0, kWsHeader + sizeof(PcgState) + 256, s);
  if (e != cudaSuccess) return fail_cuda(e);
  const uint32_t smem = small_smem(n, padded_dim(op->d), kSWarps * rows, nr, ldq).total;
  e = cudaErrorInvalidValue;
  switch (padded_dim(op->d)) {
    case 2: e = launch_small_r<2>(rows, a, grid, smem, s); break;
    case 4: e = launch_small_r<4>(rows, a, grid, smem, s); break;
    case 6: e = launch_small_r<6>(rows, a, grid, smem, s); break;
    case 8: e = launch_small_r<8>(rows, a, grid, smem, s); break;
    case 10: e = launch_small_r<10>(rows, a, grid, smem, s); break;
    case 12: e = launch_small_r<12>(rows, a, grid, smem, s); break;
    case 14: e = launch_small_r<14>(rows, a, grid, smem, s); break;
    case 16: e = launch_small_r<16>(rows, a, grid, smem, s); break;
    default: break;
  }
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    // fewer SMs than the device reports are available to this process
    cudaGetLastError();
    return -1;
  }
  if (e != cudaSuccess) return fail_cuda(e);
  char back[kWsHeader + sizeof(PcgState)];
  e = cudaMemcpyAsync(back, p, sizeof(back), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail_cuda(e);
  const int dev_status = reinterpret_cast<const WsHeader*>(back)->status;
  PcgState h;
  memcpy(&h, back + kWsHeader, sizeof(h));
  res->iterations = h.iter;
  res->accurate_matvecs = h.n_accurate;
  res->residual_norm = h.true_rnorm;
  res->recurrence_norm = h.rnorm;
  res->rhs_norm = h.bnorm;
  res->kernel_launches = 1;
  if (dev_status != 0) {
    res->status = dev_status;
    return dev_status;
  }
  if (h.bnorm == 0.0 && h.status == LAKER_OK) res->residual_norm = 0.0;
  res->status = h.status;
  return h.status;
}

cudaError_t set_wait_limit_small(unsigned long long ns) { return set_wait_limit_this_unit(ns); }

}  // namespace laker
