// Narrow multi-RHS FP32 matvec of unclamped operators (few right-hand sides):
// Y = lam X + exp(Er Ec^T) X, flash-attention style -- the kernel entries live
// only in registers between two tensor-core products.
//
// Why warp-level MMAs (mma.sync) and not tcgen05: with N = 16 .. 64 right-hand
// sides the tcgen05 form of this product (logits into tensor memory, entries
// exponentiated, split and stored back as the A operand, P X from there) was
// bound by its chain of hand-offs (MMA -> barrier -> tcgen05.ld -> exp2 ->
// tcgen05.st -> barrier -> MMA with a nearly empty N): about 230 cycles of an SM
// sub-partition per 128 entries at k = 16.  Here a warp forms the logits of a 16 x 8
// tile with two FP16 MMAs or FP32 FMAs, exponentiates the accumulator registers and
// feeds them straight back as the A operand of the TF32 products, so nothing waits
// for another warp; the MMAs themselves are what bounds it (per 128 entries
// 2 x 8.5 cycles of FP16 logits, 25 cycles per 8 right-hand sides; 32 cycles of MUFU
// ex2 run beside them, 4 d FP32 FMAs a lane only in part).
//
// Logits.  Up to 32 right-hand sides: the split-FP16 image of matvec_symtc.cu
// (kK1tF16x2: V0 W0 + V1 W1 = H H' + Hs L' + L Hs'; kK1tF16: (H L' + L H') 2^12
// scaled down, then H H'), 22 bits an operand, as the single-RHS operator has it.
// Above: FP32 FMAs in the order of the wide kernel (matvec_tc.cu), whose products
// these would otherwise be and which holds the operands in FP32.  22 bits are not
// enough there: with |e|^2 up to 79 split-FP16 logits cost 3 to 28 times the error
// (n = 300 .. 30,011: 2e-7 .. 7e-6 with FP32 logits, 2e-6 .. 1.5e-5 without).  FP32
// logits take 3 to 5 % more time at d = 4, 7 to 24 % at d = 10, 18 to 36 % at d = 16
// (n from 5,003).  P X: split TF32, P_hi X_hi + P_hi X_lo + P_lo X_hi, P_hi by truncation,
// the other parts rounded.  The accumulator of a tile holds columns 2t and 2t + 1
// in lane t where the A operand wants columns t and t + 4: the K index may be
// taken in any order, so X's rows are stored in that order (k2m_pack_x: one
// 16-byte load gives a lane its four X values of an 8 x 8 tile).
//
// Measured (whole product, before: the tcgen05 form; k = 64 the wide kernel):
// n = 50,000, k = 16: 3.44 -> 1.55 ms, k = 32: 3.47 -> 2.45 ms; n = 10,007, k = 16:
// 188 -> 101 us, k = 64: 405 -> 255 us.  Error against 64 bits, random X, |e| up to 2:
// 6e-5 -> 7e-7 at n = 50,000, 3e-6 -> 7e-7 at n = 10,007.
//
// CTA: 8 warps of MT 16-row tiles, one chunk of NT 8-column tiles of right-hand
// sides and one segment of the columns; two CTAs per SM.  Column operands and X
// arrive 64 columns at a time by bulk copies into a ring of stages (bounded
// waits).  Segment partial sums are added in a fixed order (launch_seg_reduce).
#include <cstdlib>

#include "sym.cuh"

namespace laker {
namespace {

constexpr int kFWarps = 8, kFThreads = kFWarps * 32;
constexpr int kFSlab = 64;                        // columns per stage
constexpr uint32_t kFVar = 512u * 32u;            // one variant of a 512-point image block
constexpr int64_t kFImgBlock = 131072;            // image bytes per 512 points
constexpr uint32_t kFColVar = kFSlab * 32u;       // a stage's share of a column variant
constexpr int kFMaxTiles = 8;                     // 8-column tiles of right-hand sides per chunk

constexpr int kFMaxF16 = 32;                      // more right-hand sides: FP32 logits

// NT tiles of right-hand sides per chunk; MT row tiles per warp; DP > 0: FP32 logits
// of DP dimensions.
template <int NT, int DP>
struct K2fCfg {
  static constexpr int kMT = NT <= 4 ? 2 : 1;
  static constexpr int kRows = kFWarps * kMT * 16;
  static constexpr uint32_t kXBytes = kFSlab / 8 * NT * 512u;
  static constexpr uint32_t kColBytes = DP > 0 ? kFSlab * DP * 4u : 2 * kFColVar;
  static constexpr uint32_t kStage = kColBytes + kXBytes;
  static constexpr int kStages = NT <= 4 ? 4 : 3;
  static constexpr uint32_t kOffBar = kStages * kStage;
  static constexpr uint32_t kSmem = kOffBar + kStages * 8 + 128;  // + alignment slack
  static_assert(2 * (kSmem + 1024) <= 227 * 1024, "two CTAs per SM");
};

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                              uint32_t b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]),
        "f"(c[2]), "f"(c[3]));
}

__device__ __forceinline__ void mma_tf32_1688(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                              uint32_t b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]),
        "f"(c[2]), "f"(c[3]));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(saddr));
}

__device__ __forceinline__ uint32_t rna_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

// Byte offset of 16-byte chunk c (0, 1) of point row r in a variant (32-byte
// swizzle: chunk XOR bit 2 of the row).
__device__ __forceinline__ uint32_t img16_chunk(uint32_t r, uint32_t c) {
  return r * 32u + ((c ^ ((r >> 2) & 1u)) << 4);
}

// X (n x k) as the B operands of the P X products: chunk, stage of 64 columns,
// 8-column group, tile of 8 right-hand sides, lane (g, t) -> {hi, hi, lo, lo} of
// X[2t][g] and X[2t + 1][g] of the group's rows; zero past n and k.
__global__ void k2m_pack_x(const float* __restrict__ X, int64_t n, int64_t ldx, int k, int NT,
                           int64_t nst, int64_t total, float4* __restrict__ img, const int* gate) {
  if (gate && *gate == 0) return;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int lane = (int)(e & 31);
    int64_t q = e >> 5;
    const int nt = (int)(q % NT);
    q /= NT;
    const int64_t grp = q % (nst * (kFSlab / 8)), chunk = q / (nst * (kFSlab / 8));
    const int64_t j = grp * 8 + 2 * (lane & 3), c = chunk * NT * 8 + nt * 8 + (lane >> 2);
    const float v0 = j < n && c < k ? X[j * ldx + c] : 0.0f;
    const float v1 = j + 1 < n && c < k ? X[(j + 1) * ldx + c] : 0.0f;
    const uint32_t h0 = rna_tf32(v0), h1 = rna_tf32(v1);
    img[e] = make_float4(__uint_as_float(h0), __uint_as_float(h1),
                         __uint_as_float(rna_tf32(v0 - __uint_as_float(h0))),
                         __uint_as_float(rna_tf32(v1 - __uint_as_float(h1))));
  }
}

// Column embeddings for FP32 logits: 8-column group, dimension pair h, lane t ->
// {e[2t][2h], e[2t + 1][2h], e[2t][2h + 1], e[2t + 1][2h + 1]} of the group's points,
// 16-byte chunks of the packed layout put in the order in which the four lanes of a
// quad read them (at DP = 16 the packed order has them all on the same banks).
__global__ void k2m_pack_e(const float4* __restrict__ packed32, int hp, int64_t total,
                           float4* __restrict__ img, const int* gate) {
  if (gate && *gate == 0) return;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = e >> 2;  // (group, h)
    const int64_t grp = q / hp;
    img[e] = packed32[(grp * 4 + (e & 3)) * hp + (q - grp * hp)];
  }
}

template <int NT, int FMT, int DP>
__global__ void __launch_bounds__(kFThreads, 2)
    k2f_matvec(const uint8_t* __restrict__ rimg, int64_t m, const uint8_t* __restrict__ cimg,
               const uint8_t* __restrict__ ximg, int64_t nst, int64_t stages_per_seg, float lam,
               const float* __restrict__ X, int64_t ldx, int k, float* __restrict__ Y, int64_t ldy,
               float* __restrict__ part, int* status, const int* gate) {
  if (gate && *gate == 0) return;
  using Cfg = K2fCfg<NT, DP>;
  constexpr int MT = Cfg::kMT, S = Cfg::kStages;
  constexpr bool F32 = DP > 0;
  static_assert(!F32 || MT == 1, "row embeddings in registers");
  constexpr bool X2 = FMT == kK1tF16x2;
  // row operands are variants 0 and 1; the column side starts after the row side
  constexpr uint32_t kColSide = (X2 ? 2u : 3u) * kFVar;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + Cfg::kOffBar);  // [S]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t s_begin = (int64_t)blockIdx.z * stages_per_seg;
  const int ns = (int)(min(nst, s_begin + stages_per_seg) - s_begin);
  if (tid == 0) {
    for (int i = 0; i < S; ++i) mbar_init(&full[i], 1);
    mbar_fence_init();
  }
  __syncthreads();

  auto issue = [&](int s) {
    const int st = s % S;
    const int64_t gs = s_begin + s, pt = gs * kFSlab;
    uint8_t* dst = sm + st * Cfg::kStage;
    mbar_arrive_expect_tx(&full[st], Cfg::kStage);
    if constexpr (F32) {
      bulk_g2s(dst, cimg + gs * Cfg::kColBytes, Cfg::kColBytes, &full[st]);
    } else {
      const uint8_t* src = cimg + (pt / 512) * kFImgBlock + kColSide + (uint32_t)(pt % 512) * 32u;
      bulk_g2s(dst, src, kFColVar, &full[st]);
      bulk_g2s(dst + kFColVar, src + kFVar, kFColVar, &full[st]);
    }
    bulk_g2s(dst + Cfg::kColBytes, ximg + ((int64_t)blockIdx.y * nst + gs) * Cfg::kXBytes, Cfg::kXBytes,
             &full[st]);
  };
  int issued = 0;  // thread 0
  if (tid == 0)
    for (; issued < S - 1 && issued < ns; ++issued) issue(issued);

  // row operands (the image covers whole 512-point blocks, zero past m; FP32: rimg
  // is the packed layout, whole 256-point tiles)
  const int64_t row0 = (int64_t)blockIdx.x * Cfg::kRows + warp * (MT * 16);
  uint32_t A0[MT][4], A1[MT][4];
  float er[2][F32 ? DP : 1];
  if constexpr (F32) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t r = row0 + g + 8 * h;
      const float* src = reinterpret_cast<const float*>(rimg) + (r >> 1) * (2 * DP) + (r & 1);
#pragma unroll
      for (int q = 0; q < DP; ++q) er[h][q] = r < m ? src[2 * q] * kLog2e : 0.0f;
    }
  } else {
    const uint8_t* base = rimg + (row0 / 512) * kFImgBlock;
    const uint32_t r0 = (uint32_t)(row0 % 512) + g;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t o = img16_chunk(r0 + 16 * i + 8 * h, c) + 4 * t;
          A0[i][h + 2 * c] = __ldg(reinterpret_cast<const uint32_t*>(base + o));
          A1[i][h + 2 * c] = __ldg(reinterpret_cast<const uint32_t*>(base + kFVar + o));
        }
  }
  // The MMAs truncate as they accumulate, which shrinks a long sum (1e-4 relative
  // over 50,000 columns): a stage's products are accumulated by themselves and
  // added to the running sums in FP32.
  float sum[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
      for (int u = 0; u < 4; ++u) sum[i][q][u] = 0.0f;

  // logits of an 8-column group (log2 e folded into the rows)
  auto logits = [&](uint32_t addr, float (&c)[MT][4]) {
    if constexpr (F32) {
#pragma unroll
      for (int h = 0; h < DP / 2; ++h) {
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr + 64u * h));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float e0 = er[u][2 * h], e1 = er[u][2 * h + 1];
          c[0][2 * u] = h == 0 ? e0 * v.x : fmaf(e0, v.x, c[0][2 * u]);
          c[0][2 * u + 1] = h == 0 ? e0 * v.y : fmaf(e0, v.y, c[0][2 * u + 1]);
          c[0][2 * u] = fmaf(e1, v.z, c[0][2 * u]);
          c[0][2 * u + 1] = fmaf(e1, v.w, c[0][2 * u + 1]);
        }
      }
      return;
    }
    uint32_t b[4];
    ldmatrix_x4(b, addr);
    const float z[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      if constexpr (X2) {
        mma_f16_16816(c[i], A0[i], b[0], b[1], z);
      } else {
        mma_f16_16816(c[i], A0[i], b[2], b[3], z);
        mma_f16_16816(c[i], A1[i], b[0], b[1], c[i]);
#pragma unroll
        for (int u = 0; u < 4; ++u) c[i][u] *= 1.0f / 4096.0f;
      }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      if constexpr (X2) mma_f16_16816(c[i], A1[i], b[2], b[3], c[i]);
      else mma_f16_16816(c[i], A0[i], b[0], b[1], c[i]);
    }
  };
  // ldmatrix source of this lane: matrix lane / 8 = (variant, chunk), row lane % 8;
  // FP32: the quad lane's chunk of each dimension pair
  const uint32_t lm_off = F32 ? 16u * t
                              : (uint32_t)(lane >> 4) * kFColVar +
                                    img16_chunk((uint32_t)(lane & 7), (uint32_t)((lane >> 3) & 1));
  constexpr uint32_t kGroup = F32 ? 32u * DP : 256u;  // bytes of an 8-column group
  const uint32_t sm0 = smem_u32(sm) + lm_off;
  bool dead = false;
#pragma unroll 1
  for (int s = 0; s < ns; ++s) {
    const int st = s % S;
    if (!dead) dead = !mbar_wait_bounded(&full[st], (uint32_t)((s / S) & 1), status);
    __syncthreads();  // every warp has left the stage that is refilled now
    if (tid == 0 && !dead && s + S - 1 < ns) issue(s + S - 1), ++issued;
    const uint32_t ca = sm0 + st * Cfg::kStage;
    const float4* xb = reinterpret_cast<const float4*>(sm + st * Cfg::kStage + Cfg::kColBytes) + lane;
    float c[2][MT][4], acc[MT][NT][4];
    logits(ca, c[0]);
#pragma unroll
    for (int j = 0; j < kFSlab / 8; ++j) {
      // the next group's logits are issued before this group's exponentials
      if (j + 1 < kFSlab / 8) logits(ca + (j + 1) * kGroup, c[(j + 1) & 1]);
      uint32_t hi[MT][4], lo[MT][4];
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        // accumulator (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1) -> A operand
        // (g, t), (g + 8, t), (g, t + 4), (g + 8, t + 4)
        const int at[4] = {0, 2, 1, 3};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float e = ex2_approx(c[j & 1][i][at[u]]);
          hi[i][u] = __float_as_uint(e) & 0xffffe000u;
          // the exact remainder, rounded to TF32 by half a unit before truncation
          lo[i][u] = (__float_as_uint(e - __uint_as_float(hi[i][u])) + 0x1000u) & 0xffffe000u;
        }
      }
#pragma unroll
      for (int q = 0; q < NT; ++q) {
        const float4 x = xb[(j * NT + q) * 32];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          const float z[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          if (j == 0) mma_tf32_1688(acc[i][q], hi[i], __float_as_uint(x.x), __float_as_uint(x.y), z);
          else mma_tf32_1688(acc[i][q], hi[i], __float_as_uint(x.x), __float_as_uint(x.y), acc[i][q]);
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
          mma_tf32_1688(acc[i][q], hi[i], __float_as_uint(x.z), __float_as_uint(x.w), acc[i][q]);
#pragma unroll
        for (int i = 0; i < MT; ++i)
          mma_tf32_1688(acc[i][q], lo[i], __float_as_uint(x.x), __float_as_uint(x.y), acc[i][q]);
      }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int q = 0; q < NT; ++q)
#pragma unroll
        for (int u = 0; u < 4; ++u) sum[i][q][u] += acc[i][q][u];
  }
  // after a failed wait: this CTA's copies must land before it exits
  if (tid == 0 && dead) {
    for (int i = issued > S ? issued - S : 0; i < issued; ++i)
      mbar_wait_drain(&full[i % S], (uint32_t)((i / S) & 1), status);
  }

#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t row = row0 + 16 * i + g + 8 * h;
        const int col = blockIdx.y * (NT * 8) + q * 8 + 2 * t;  // and col + 1
        if (row >= m || col >= k) continue;
        const float v0 = sum[i][q][2 * h], v1 = sum[i][q][2 * h + 1];
        if (part) {
          float* dst = part + ((int64_t)blockIdx.z * m + row) * k + col;
          if ((k & 1) == 0) {  // 8-byte aligned, and col + 1 < k
            *reinterpret_cast<float2*>(dst) = make_float2(v0, v1);
          } else {
            dst[0] = v0;
            if (col + 1 < k) dst[1] = v1;
          }
        } else {
          Y[row * ldy + col] = lam != 0.0f ? fmaf(lam, X[row * ldx + col], v0) : v0;
          if (col + 1 < k)
            Y[row * ldy + col + 1] = lam != 0.0f ? fmaf(lam, X[row * ldx + col + 1], v1) : v1;
        }
      }
}

// Tiles of right-hand sides per chunk, as few chunks as 64 columns allow,
// evenly filled, rounded up to an instantiated width.
constexpr int kFWidths[] = {1, 2, 3, 4, 6, 8};

struct K2fWork {
  int nt, chunks, segs;
  int64_t nst, sps;  // stages of 64 columns, per segment
};

constexpr int k2f_rows(int nt) { return kFWarps * (nt <= 4 ? 2 : 1) * 16; }

struct K2fLayout {
  size_t x_off, x_bytes, part_off, rimg_off, cimg_off, total;
};

K2fLayout k2f_layout(const K2fWork& w, int64_t m, int64_t n, int k, bool same_points) {
  K2fLayout L{};
  L.x_off = 0;
  L.x_bytes = (size_t)w.chunks * (size_t)w.nst * (kFSlab / 8) * (size_t)w.nt * 512;
  L.part_off = L.x_off + (size_t)round_up((int64_t)L.x_bytes, 1024);
  const size_t part = w.segs > 1 ? (size_t)w.segs * (size_t)m * (size_t)k * 4 : 0;
  L.rimg_off = L.part_off + (size_t)round_up((int64_t)part, 1024);
  L.cimg_off = same_points ? L.rimg_off : L.rimg_off + k1t_image_bytes(m);
  L.total = L.cimg_off + k1t_image_bytes(n);
  return L;
}

// `avail`: bytes of scratch; the segments' partial sums have to fit too.
K2fWork k2f_work(int64_t m, int64_t n, int k, bool same_points, size_t avail) {
  K2fWork w{};
  const int tiles = (k + 7) / 8;
  w.chunks = (tiles + kFMaxTiles - 1) / kFMaxTiles;
  const int want = (tiles + w.chunks - 1) / w.chunks;
  for (int v : kFWidths)
    if (v >= want) {
      w.nt = v;
      break;
    }
  w.nst = ceil_div(n > 0 ? n : 1, kFSlab);
  // Segments: whole waves of two CTAs per SM, at least 4 stages each; a further
  // segment costs m k partial sums (charged 0.5 % of a pass).
  const int64_t ctas = ceil_div(m > 0 ? m : 1, k2f_rows(w.nt)) * w.chunks;
  const int64_t slots = 2 * (int64_t)sm_count();
  const int64_t smax = w.nst / 4 < 1 ? 1 : (w.nst / 4 > 32 ? 32 : w.nst / 4);
  double best = 1e300;
  auto split = [&](int64_t s) {
    w.sps = ceil_div(w.nst, s);
    w.segs = (int)ceil_div(w.nst, w.sps);
  };
  int64_t segs = 1;
  for (int64_t s = 1; s <= smax; ++s) {
    const double cost = (double)ceil_div(ctas * s, slots) / (double)s * (1.0 + 0.005 * (double)(s - 1));
    split(s);
    if (cost < best - 1e-12 && (s == 1 || k2f_layout(w, m, n, k, same_points).total <= avail))
      best = cost, segs = s;
  }
  split(segs);
  return w;
}

// Largest k that takes this kernel (LAKER_VARIANT_MULTI_FLASH_K; 0 off).
int k2f_max_k() { return variant_get(LAKER_VARIANT_MULTI_FLASH_K); }

template <int NT, int FMT, int DP>
cudaError_t launch_k2f_t(const uint8_t* rimg, int64_t m, const uint8_t* cimg, const uint8_t* ximg,
                         const K2fWork& w, float lam, const float* X, int64_t ldx, int k, float* Y,
                         int64_t ldy, float* part, int* status, const int* gate, cudaStream_t s) {
  using Cfg = K2fCfg<NT, DP>;
  static SmemOptIn optin;
  const cudaError_t e = optin.allow(k2f_matvec<NT, FMT, DP>, Cfg::kSmem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)ceil_div(m, Cfg::kRows), (unsigned)w.chunks, (unsigned)w.segs);
  k2f_matvec<NT, FMT, DP><<<grid, kFThreads, Cfg::kSmem, s>>>(rimg, m, cimg, ximg, w.nst, w.sps, lam, X, ldx,
                                                         k, Y, ldy, part, status, gate);
  return cudaGetLastError();
}

// FP32 logits: a chunk has at least five tiles (k > 32), so six or eight.
template <int DP>
cudaError_t launch_k2f_f32(const float* rows32, int64_t m, const uint8_t* cimg, const uint8_t* ximg,
                           const K2fWork& w, float lam, const float* X, int64_t ldx, int k, float* Y,
                           int64_t ldy, float* part, int* status, const int* gate, cudaStream_t s) {
  const uint8_t* rows = reinterpret_cast<const uint8_t*>(rows32);
  switch (w.nt) {
    case 6:
      return launch_k2f_t<6, kK1tF16x2, DP>(rows, m, cimg, ximg, w, lam, X, ldx, k, Y, ldy, part,
                                            status, gate, s);
    case 8:
      return launch_k2f_t<8, kK1tF16x2, DP>(rows, m, cimg, ximg, w, lam, X, ldx, k, Y, ldy, part,
                                            status, gate, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

bool k2f_enabled(int k, int clamp) { return !clamp && k > 1 && k <= k2f_max_k(); }

size_t k2f_workspace_bytes(int64_t m, int64_t n, int k, bool same_points, size_t avail) {
  return k2f_layout(k2f_work(m, n, k, same_points, avail), m, n, k, same_points).total;
}

// What every multi-RHS product is given for this kernel, whatever its k: X in chunks
// of 32 columns, the operand images, partial sums of as many segments as make eight
// 128-row tiles of a chunk per SM.
size_t k2f_reserve_bytes(int64_t m, int64_t n, int k, bool same_points) {
  const int64_t N = round_up(k < 32 ? k : 32, 16), chunks = ceil_div(k, N), slabs = ceil_div(n, kFSlab);
  const int64_t tiles = ceil_div(m, 128) * chunks, want = 8 * (int64_t)sm_count();
  int64_t segs = tiles >= want ? 1 : ceil_div(want, tiles);
  const int64_t most = slabs / 8 > 1 ? slabs / 8 : 1;
  if (segs > most) segs = most;
  if (segs > 64) segs = 64;
  segs = ceil_div(slabs, ceil_div(slabs, segs));
  const size_t part = segs > 1 ? (size_t)segs * (size_t)m * (size_t)k * 4 : 0;
  return (size_t)round_up(chunks * slabs * 512 * N, 1024) + (size_t)round_up((int64_t)part, 1024) +
         (same_points ? 0 : k1t_image_bytes(m)) + k1t_image_bytes(n);
}

cudaError_t launch_k2f(const float* rows32, int64_t m, const float* cols32, int64_t n, int d,
                       float lam, const float* X, int64_t ldx, int k, float* Y, int64_t ldy,
                       uint8_t* ws, size_t ws_bytes, int* status, cudaStream_t s, const int* gate) {
  if (m <= 0 || n <= 0 || k < 1) return cudaSuccess;
  const bool same = rows32 == cols32 && m == n;
  const K2fWork w = k2f_work(m, n, k, same, ws_bytes);
  if (w.chunks > 65535) return cudaErrorInvalidValue;
  const K2fLayout L = k2f_layout(w, m, n, k, same);
  if (L.total > ws_bytes) return cudaErrorInvalidValue;
  uint8_t* ximg = ws + L.x_off;
  float* part = w.segs > 1 ? reinterpret_cast<float*>(ws + L.part_off) : nullptr;
  uint8_t* rimg = ws + L.rimg_off;
  uint8_t* cimg = ws + L.cimg_off;
  const int64_t total = (int64_t)(L.x_bytes / 16);
  int g = (int)ceil_div(total, 256);
  if (g > sm_count() * 8) g = sm_count() * 8;
  k2m_pack_x<<<g, 256, 0, s>>>(X, n, ldx, k, w.nt, w.nst, total, reinterpret_cast<float4*>(ximg), gate);
  cudaError_t e = cudaGetLastError();
  const int dp = padded_dim(d);
  if (k > kFMaxF16) {
    if (e != cudaSuccess) return e;
    const int64_t chunks = w.nst * kFSlab / 2 * (dp / 2);
    int ge = (int)ceil_div(chunks, 256);
    if (ge > sm_count() * 8) ge = sm_count() * 8;
    k2m_pack_e<<<ge, 256, 0, s>>>(reinterpret_cast<const float4*>(cols32), dp / 2, chunks,
                                  reinterpret_cast<float4*>(cimg), gate);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaErrorInvalidValue;
    switch (dp) {
#define LAKER_K2F_CASE(D)                                                                            \
  case D:                                                                                            \
    e = launch_k2f_f32<D>(rows32, m, cimg, ximg, w, lam, X, ldx, k, Y, ldy, part, status, gate, s);  \
    break;
      LAKER_K2F_CASE(2) LAKER_K2F_CASE(4) LAKER_K2F_CASE(6) LAKER_K2F_CASE(8) LAKER_K2F_CASE(10)
      LAKER_K2F_CASE(12) LAKER_K2F_CASE(14) LAKER_K2F_CASE(16)
#undef LAKER_K2F_CASE
      default: break;
    }
  } else {
    const int fmt = dp <= 10 ? kK1tF16x2 : kK1tF16;
    if (e == cudaSuccess) e = launch_k1t_pack(rows32, m, d, rimg, round_up(m, 512), s, fmt);
    if (e == cudaSuccess && !same) e = launch_k1t_pack(cols32, n, d, cimg, round_up(n, 512), s, fmt);
    if (e != cudaSuccess) return e;
    e = cudaErrorInvalidValue;
    switch (w.nt) {
#define LAKER_K2F_CASE(W)                                                                             \
  case W:                                                                                             \
    e = fmt == kK1tF16x2 ? launch_k2f_t<W, kK1tF16x2, 0>(rimg, m, cimg, ximg, w, lam, X, ldx, k, Y,    \
                                                         ldy, part, status, gate, s)                  \
                         : launch_k2f_t<W, kK1tF16, 0>(rimg, m, cimg, ximg, w, lam, X, ldx, k, Y, ldy, \
                                                       part, status, gate, s);                        \
    break;
      LAKER_K2F_CASE(1) LAKER_K2F_CASE(2) LAKER_K2F_CASE(3) LAKER_K2F_CASE(4)
#undef LAKER_K2F_CASE
      default: break;
    }
  }
  if (e != cudaSuccess || w.segs == 1) return e;
  return launch_seg_reduce(part, w.segs, m, k, lam, X, ldx, Y, ldy, gate, s);
}

cudaError_t set_wait_limit_flash(unsigned long long ns) { return set_wait_limit_this_unit(ns); }

}  // namespace laker
