// FP64 fused multi-RHS attention-kernel matvec: Y = lam X + exp(Er Ec^T) X, or
// the residual B - (...), for X (n x k), k > 1 (residuals of multi-RHS solves,
// float64 operators).
//
// What bounds it: the FP64 pipe, 64 FMAs per clock and SM, which FP64 MMAs
// (mma.sync m8n8k4) and DFMAs share.  Per entry: d (padded to 4) FMAs of logit,
// an 11-operation table-driven exp, k FMAs.  The contraction runs as MMAs whose
// operands come straight out of registers, so the pipe is not starved by shared-
// memory loads: a warp keeps MT 8-row tiles; per 8 columns it forms the logits
// (MMA), exponentiates them in the accumulator layout and feeds them back as the
// A operand.  The accumulator holds columns 2t and 2t + 1 in lane t, the operand
// wants column t: the contraction index may be taken in any order, so the first
// K step takes columns {0, 2, 4, 6} and the second {1, 3, 5, 7}, with X's rows
// read in the same order.  No entry passes through shared memory and no barrier
// separates the exponentials from the products.
//
// Measured (whole product; before: 64 x 64 tiles of DFMA microtiles with the
// entries in shared memory, bound by its shared-memory loads and barriers):
// n = 20,000, k = 512: 37.8 -> 17.6 ms (0.73 of the FP64 pipe's rate);
// n = 8,009, k = 200: 3.61 -> 1.23 ms; n = 30,011, k = 16: 2.5 ms (0.76).  Error
// against 64-bit torch at n = 8,009, k = 200: 3.1e-15 -> 1.9e-15.
//
// CTA: 4 warps, 32 MT rows, one chunk of NT 8-column tiles of right-hand sides
// (as few chunks as 128 columns allow, evenly filled: an entry is evaluated once
// per chunk) and one segment of the columns.  X and the column embeddings arrive
// 32 columns at a time by cp.async, double-buffered.  Segments are used where row
// tiles x chunks leave SMs idle (f64m_plan); their partial sums are added in
// segment order.
#include "internal.cuh"

namespace laker {
namespace {

constexpr int kFmWarps = 4, kFmThreads = kFmWarps * 32;
constexpr int kFmCols = 32;       // columns per stage
constexpr int kFmMaxTiles = 16;   // 8-column tiles of right-hand sides per chunk

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// 8 / 16 byte asynchronous copies global -> shared; zeros when !ok (src is then
// not read).
__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src),
               "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// KS K steps of 4 embedding dimensions, NT 8-column tiles of right-hand sides,
// MT 8-row tiles per warp.
template <int KS, int NT, int MT>
struct FmCfg {
  // row strides (doubles) that spread a half warp's 8-byte loads over all banks:
  // embeddings 4 or 12 mod 16, X 2 mod 8
  static constexpr int kLe = KS == 1 ? 4 : KS <= 3 ? 12 : 20;
  static constexpr int kLx = NT * 8 + 2;
  static constexpr int kStage = kFmCols * (kLe + kLx);
  static constexpr size_t kSmem = (size_t)(2 * kStage + 64) * sizeof(double);
  static constexpr int kRows = kFmWarps * MT * 8;
  static constexpr int kMinCtas = MT * NT >= 26 ? 2 : 3;
};

// A16: the column embeddings lie on 16 bytes (else they are copied 8 at a time; a
// choice at run time cost 4.6 % at 16 tiles, n = 20,000, k = 256).
template <int KS, int NT, int MT, bool CLAMP, bool A16>
__global__ void __launch_bounds__(kFmThreads, FmCfg<KS, NT, MT>::kMinCtas)
    f64m_matvec(const double* __restrict__ rows, int64_t m, const double* __restrict__ cols,
                int64_t n, int DP, double lam, const double* __restrict__ X, int k, int64_t ldx,
                const double* __restrict__ B, int64_t ldb, double* __restrict__ Y, int64_t ldy,
                double* __restrict__ part, int64_t cols_per_seg, const int* gate) {
  if (gate && *gate == 0) return;
  using Cfg = FmCfg<KS, NT, MT>;
  extern __shared__ __align__(16) double sm[];
  double* sExp = sm + 2 * Cfg::kStage;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t i0 = (int64_t)blockIdx.x * Cfg::kRows + warp * (MT * 8);
  const int c0 = blockIdx.y * (NT * 8);
  const int64_t j_begin = (int64_t)blockIdx.z * cols_per_seg;
  const int64_t j_end = min(n, j_begin + cols_per_seg);
  const int nst = j_begin < j_end ? (int)ceil_div(j_end - j_begin, kFmCols) : 0;
  exp_table_to_shared(sExp, tid, kFmThreads);
  // dimensions past DP are never copied
  for (int e = tid; e < 2 * kFmCols * Cfg::kLe; e += kFmThreads) {
    const int st = e / (kFmCols * Cfg::kLe);
    sm[st * Cfg::kStage + e - st * kFmCols * Cfg::kLe] = 0.0;
  }
  __syncthreads();

  // the packed layout is padded with zero points to whole 128-point tiles and a
  // stage starts at a multiple of 32 points: embedding copies stay in bounds
  auto fetch = [&](int s, int st) {
    const int64_t j0 = j_begin + (int64_t)s * kFmCols;
    double* se = sm + st * Cfg::kStage;
    double* sx = se + kFmCols * Cfg::kLe;
    const int ch = DP >> 1;  // 16-byte chunks of an embedding
    for (int e = tid; e < kFmCols * ch; e += kFmThreads) {
      const int jj = e / ch, c = e - jj * ch;
      double* dst = se + jj * Cfg::kLe + 2 * c;
      const double* src = cols + (j0 + jj) * DP + 2 * c;
      if constexpr (A16) {
        cp_async16(dst, src);
      } else {
        cp_async8(dst, src, true);
        cp_async8(dst + 1, src + 1, true);
      }
    }
    for (int e = tid; e < kFmCols * NT * 8; e += kFmThreads) {
      const int jj = e / (NT * 8), c = e - jj * (NT * 8);
      const bool ok = j0 + jj < j_end && c0 + c < k;
      cp_async8(sx + jj * Cfg::kLx + c, ok ? X + (j0 + jj) * ldx + c0 + c : X, ok);
    }
    cp_async_commit();
  };

  double a[MT][KS];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    const int64_t i = i0 + mt * 8 + g;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const int kk = ks * 4 + t;
      a[mt][ks] = (i < m && kk < DP) ? rows[i * DP + kk] : 0.0;
    }
  }
  double acc[MT][NT][2];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;

  if (nst > 0) fetch(0, 0);
#pragma unroll 1
  for (int s = 0; s < nst; ++s) {
    if (s + 1 < nst) {
      fetch(s + 1, (s + 1) & 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double* se = sm + (s & 1) * Cfg::kStage + g * Cfg::kLe + t;
    const double* sx = sm + (s & 1) * Cfg::kStage + kFmCols * Cfg::kLe + 2 * t * Cfg::kLx + g;
#pragma unroll 1
    for (int jg = 0; jg < kFmCols / 8; ++jg) {
      double p[MT][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) p[mt][0] = p[mt][1] = 0.0;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        const double b = se[jg * 8 * Cfg::kLe + ks * 4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) mma_f64(p[mt], a[mt][ks], b);
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          p[mt][h] = exp_tab(CLAMP && p[mt][h] > kClamp64 ? kClamp64 : p[mt][h], sExp);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const double b = sx[(jg * 8 + h) * Cfg::kLx + nt * 8];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma_f64(acc[mt][nt], p[mt][h], b);
        }
    }
    __syncthreads();  // this stage is refilled by the next step's fetch
  }

  const bool square = m == n;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    const int64_t i = i0 + mt * 8 + g;
    if (i >= m) continue;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
    {
      const int c = c0 + nt * 8 + 2 * t;
      if (part && (k & 1) == 0 && c < k) {  // both columns, 16-byte aligned
        *reinterpret_cast<double2*>(part + ((int64_t)blockIdx.z * m + i) * k + c) =
            make_double2(acc[mt][nt][0], acc[mt][nt][1]);
        continue;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (c + h >= k) continue;
        double y = acc[mt][nt][h];
        if (part) {
          part[((int64_t)blockIdx.z * m + i) * k + c + h] = y;
        } else {
          if (square) y = fma(lam, X[i * ldx + c + h], y);
          Y[i * ldy + c + h] = B ? B[i * ldb + c + h] - y : y;
        }
      }
    }
  }
}

// Y = [B -] (lam X + the segments' partial sums, in segment order).
__global__ void f64m_reduce_kernel(const double* __restrict__ part, int S, int64_t m, int k,
                                   int square, double lam, const double* __restrict__ X, int64_t ldx,
                                   const double* __restrict__ B, int64_t ldb, double* __restrict__ Y,
                                   int64_t ldy, const int* gate) {
  if (gate && *gate == 0) return;
  const int64_t total = m * (int64_t)k;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / k;
    const int c = (int)(e - i * k);
    double y = 0.0;
#pragma unroll 4  // loads in flight, added in segment order
    for (int s = 0; s < S; ++s) y += part[(int64_t)s * total + e];
    if (square) y = fma(lam, X[i * ldx + c], y);
    Y[i * ldy + c] = B ? B[i * ldb + c] - y : y;
  }
}

// Tiles of right-hand sides per chunk: the chunks that k needs at 16 tiles
// each, evenly filled, rounded up to an instantiated width.  The widths are at most
// 1.5 times apart from 4 on, 1.3 times from 8 on (every absent tile of a chunk costs
// as much as a present one); each further width is eight more kernels to build.
constexpr int kFmWidths[] = {1, 2, 4, 6, 8, 10, 13, 16};
constexpr int kFmOddWidth = 4;

struct FmPlan {
  int nt, mt, chunks, S;
  int64_t cols_per_seg;
};

constexpr int fm_mt(int nt) { return nt <= 4 ? 4 : nt <= 8 ? 3 : 2; }

// `avail`: bytes for the segments' partial sums.  `a16`: whether the column embeddings
// lie on 16 bytes; where they do not, one width serves every k.
FmPlan f64m_plan(int64_t m, int64_t n, int k, size_t avail, bool a16 = true) {
  FmPlan p{};
  const int tiles = (k + 7) / 8;
  p.chunks = (tiles + kFmMaxTiles - 1) / kFmMaxTiles;
  const int want = (tiles + p.chunks - 1) / p.chunks;
  for (int w : kFmWidths)
    if (w >= want) {
      p.nt = w;
      break;
    }
  if (!a16) {
    p.nt = kFmOddWidth;
    p.chunks = (tiles + kFmOddWidth - 1) / kFmOddWidth;
  }
  p.mt = fm_mt(p.nt);
  // Segments: the FP64 pipe is shared by an SM's CTAs, so the time is the most
  // CTAs on an SM over S; each further segment writes and reads m k partial sums
  // (charged 0.5 % of a segment-free pass, at least 256 columns per segment).  Up to
  // 511 columns that would be one segment and a few CTAs: there shorter segments fill
  // the SMs once and no more, as the partial sums weigh more than the entries (n = 300,
  // k = 500: 58 us in one segment, 23 in four; 51 in the DFMA tiles before).
  const int64_t ctas = ceil_div(m > 0 ? m : 1, kFmWarps * p.mt * 8) * p.chunks;
  const bool wide = p.nt >= 10;  // below 128 columns the sum's launch pays only there
  int64_t smax = n / (n < 128 && wide ? 32 : n < 512 ? 64 : 256);
  if (n < 512 && smax > sm_count() / ctas) smax = sm_count() / ctas;
  smax = smax < 1 ? 1 : (smax > 16 ? 16 : smax);
  const int64_t nn = n > 0 ? n : 1;
  double best = 1e300;
  for (int64_t S = 1; S <= smax; ++S) {
    const double cost = (double)ceil_div(ctas * S, sm_count()) / (double)S *
                        (1.0 + 0.005 * (double)(S - 1));
    const int64_t cols = round_up(ceil_div(nn, S), kFmCols), segs = ceil_div(nn, cols);
    if (cost < best - 1e-12 &&
        (segs == 1 || (size_t)segs * (size_t)m * (size_t)k * sizeof(double) <= avail)) {
      best = cost;
      p.S = (int)segs;
      p.cols_per_seg = cols;
    }
  }
  return p;
}

template <int KS, int NT, bool CLAMP, bool A16 = true>
cudaError_t launch_f64m_t(const double* rows, int64_t m, const double* cols, int64_t n, int DP,
                          double lam, const double* X, int k, int64_t ldx, const double* B,
                          int64_t ldb, double* Y, int64_t ldy, double* part, const FmPlan& p,
                          const int* gate, cudaStream_t s) {
  constexpr int MT = fm_mt(NT);
  using Cfg = FmCfg<KS, NT, MT>;
  static SmemOptIn optin;
  const cudaError_t e = optin.allow(f64m_matvec<KS, NT, MT, CLAMP, A16>, Cfg::kSmem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)ceil_div(m, Cfg::kRows), (unsigned)p.chunks, (unsigned)p.S);
  f64m_matvec<KS, NT, MT, CLAMP, A16><<<grid, kFmThreads, Cfg::kSmem, s>>>(
      rows, m, cols, n, DP, lam, X, k, ldx, B, ldb, Y, ldy, p.S > 1 ? part : nullptr,
      p.cols_per_seg, gate);
  return cudaGetLastError();
}

template <int KS, bool CLAMP>
cudaError_t launch_f64m_nt(const double* rows, int64_t m, const double* cols, int64_t n, int DP,
                           double lam, const double* X, int k, int64_t ldx, const double* B,
                           int64_t ldb, double* Y, int64_t ldy, double* part, const FmPlan& p,
                           const int* gate, cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(cols) % 16 != 0)
    return launch_f64m_t<KS, kFmOddWidth, CLAMP, false>(rows, m, cols, n, DP, lam, X, k, ldx, B, ldb, Y,
                                                        ldy, part, p, gate, s);
  switch (p.nt) {
#define LAKER_FM_CASE(W)                                                                         \
  case W:                                                                                        \
    return launch_f64m_t<KS, W, CLAMP>(rows, m, cols, n, DP, lam, X, k, ldx, B, ldb, Y, ldy, part, \
                                       p, gate, s);
    LAKER_FM_CASE(1) LAKER_FM_CASE(2) LAKER_FM_CASE(4) LAKER_FM_CASE(6) LAKER_FM_CASE(8)
    LAKER_FM_CASE(10) LAKER_FM_CASE(13) LAKER_FM_CASE(16)
#undef LAKER_FM_CASE
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

size_t f64m_workspace_bytes(int64_t m, int64_t n, int k, size_t avail) {
  const FmPlan p = f64m_plan(m, n, k, avail);
  return p.S > 1 ? (size_t)p.S * (size_t)m * (size_t)k * sizeof(double) : 0;
}

cudaError_t launch_multi_f64(const double* rows64, int64_t m, const double* cols64, int64_t n, int d,
                             double lam, int clamp, const double* X, int k, int64_t ldx,
                             const double* B, int64_t ldb, double* Y, int64_t ldy, double* part,
                             size_t part_bytes, cudaStream_t s, const int* gate) {
  if (m <= 0) return cudaSuccess;
  // (the partial sums' 16-byte stores; a single segment needs no scratch)
  if (reinterpret_cast<uintptr_t>(part) % 16 != 0) part_bytes = 0;
  const FmPlan p = f64m_plan(m, n, k, part_bytes, reinterpret_cast<uintptr_t>(cols64) % 16 == 0);
  if (p.chunks > 65535) return cudaErrorInvalidValue;
  const int DP = padded_dim(d);
  cudaError_t e = cudaErrorInvalidValue;
#define LAKER_FM_KS(KSv)                                                                        \
  case KSv:                                                                                     \
    e = clamp ? launch_f64m_nt<KSv, true>(rows64, m, cols64, n, DP, lam, X, k, ldx, B, ldb, Y,   \
                                          ldy, part, p, gate, s)                                \
              : launch_f64m_nt<KSv, false>(rows64, m, cols64, n, DP, lam, X, k, ldx, B, ldb, Y,  \
                                           ldy, part, p, gate, s);                              \
    break;
  switch ((DP + 3) / 4) {
    LAKER_FM_KS(1) LAKER_FM_KS(2) LAKER_FM_KS(3) LAKER_FM_KS(4)
    default: break;
  }
#undef LAKER_FM_KS
  if (e != cudaSuccess || p.S == 1) return e;
  int g = (int)ceil_div(m * (int64_t)k, 256);
  if (g > sm_count() * 8) g = sm_count() * 8;
  f64m_reduce_kernel<<<g, 256, 0, s>>>(part, p.S, m, k, m == n ? 1 : 0, lam, X, ldx, B, ldb, Y, ldy,
                                       gate);
  return cudaGetLastError();
}

}  // namespace laker
