// 3x3 convolution (padding 1, stride 1 or 2) of NHWC BF16 tensors on tcgen05
// tensor cores, forward, input gradient and weight gradient, as implicit
// GEMMs: the taps are TMA boxes of the tensors themselves, so no im2col matrix,
// transpose or per-tap gradient reaches HBM.  No reference counterpart.
//
//   forward  out[m][n]      = sum_{tap, c} x(m, tap)[c] w[n][tap C + c]
//   dgrad    dx[p][c]       = sum_{tap, n} dz(p, tap)[n] w[n][tap C + c]
//   wgrad    gw[n][tap C+c] = sum_m dz[m][n] x(m, tap)[c]
//
// An output pixel m = (b, oy, ox) reads x at (oy s - 1 + ky, ox s - 1 + kx).
// For each tap one 4-D tensor map covers exactly the elements of x that the
// tap reads, in output-pixel coordinates (strides s C and s W C), so a box of
// output pixels is one TMA load and what lies in the padding is zero-filled.
// With stride 2 the input gradient splits into the four parities of (iy, ix),
// each a dense sum over 4, 2, 2 or 1 taps of dz.
//
// One persistent CTA per SM, 10 warps: warp 0 issues the TMA loads of a ring of
// stages, warp 1 issues tcgen05.mma into one of two TMEM accumulators, warps
// 2-9 read the other one back, so a tile's epilogue runs beside the next
// tile's MMAs.  Operand layouts: what is contiguous along K in HBM is loaded
// K-major, what is contiguous along M or N (the weights in dgrad, both operands
// in wgrad) MN-major, so nothing is transposed.  The K order of the forward is
// that of the im2col matrix, hence its results too, bit for bit.
//
// The input gradient sums as the GEMM dz . w with col2im does: the N products of a tap
// are one accumulator of the tensor cores, the taps that reach a pixel are added in FP32
// in their order, hence its results, bit for bit, and chains no longer than N (all nine
// taps in one accumulator round 9 N products in a row).  Each tap's accumulator is
// read back while the next one fills, so the epilogue warps hold a tile's sums in
// registers.
//
// An RGB input (the first layer) has rows of 27 products, too short and too
// unaligned for TMA: conv3x3_rgb_kernel gathers them into shared memory itself.
//
// Every mbarrier wait is bounded as in ds_gemm.cu: on a timeout the CTA sets the
// error word, lets what it issued land, frees its TMEM and returns.
#include <algorithm>

#include "ds_common.cuh"
#include "ds_internal.h"
#include "ds_umma.cuh"

namespace ds {
namespace {

// kConvPair: forward of 32 channels at stride 2.  TMA moves a row of a box in 2.4 (128
// bytes) to 3.6 cycles (64 bytes), and a tile took 128 rows of A and 64 of weights for
// each tap.  Two neighbouring pixels are one row of 64 channels here: the taps kx = 1
// and 2 of an output pixel are the pair it starts at, kx = 0 the second half of the
// pair before, so six boxes serve nine taps, and the weights stay in shared memory.
// 16 x 512 x 512 x 32 -> 64 channels (B200): 0.190 -> 0.128 ms.
enum ConvMode : int { kConvFwd = 0, kConvDgrad = 1, kConvWgrad = 2, kConvPair = 3 };
enum ConvEpi : int { kConvGelu = 0, kConvF32 = 1 };  // forward only

constexpr int kEpiWarps = 8;  // two per 32 TMEM lanes; kEpi has the exception
constexpr int kWgradPixels = 64;  // K block of the weight gradient
// Pixels summed by one accumulation chain of the weight gradient: the tensor
// cores' FP32 sums lose precision with the chain's length (relative error
// 4.6e-6 at 4096 products, the length the im2col path used), so longer
// reductions are split and their partials added in order.  There are at most 512
// partials (64 on the im2col path): beyond 2.1 million pixels the chains grow again.
constexpr int kWgradChain = 4096;

// A rectangle of pixels per tile: bw x bh of each of bb images (powers of two),
// and the number of such tiles along x, y and the images.
struct PixelTiles {
  int lw, lh;      // log2 of bw, bh
  int bb;
  int tx, ty, tb;
};

struct ConvArgs {
  int B, H, W, C, Ho, Wo, N, stride;
  int kp;                       // row pitch of the weights
  int tiles_n;                  // column tiles (forward: of N, dgrad: of C, wgrad: of 9C)
  PixelTiles pt[4];             // dgrad: one per parity class
  int first[5];                 // first work item of each class; [classes] = all items
  int classes;
  int splits, kb_per_split;     // wgrad
  int off_x[9], off_y[9];       // forward / wgrad: coordinate of output pixel 0 in the tap's map
  const float* bias;
  const __nv_bfloat16* zprev;   // dgrad: pre-activation below, or null
  __nv_bfloat16 *y, *z;         // forward outputs; dgrad writes y
  float* d;                     // forward FP32 output; wgrad [splits][N][kp]
  uint32_t* err;
  uint32_t spin;
};

struct ConvMaps {
  CUtensorMap x[9];  // the taps of x (forward, wgrad)
  CUtensorMap w;     // the weights (forward, dgrad)
  CUtensorMap dz;    // the output gradient (dgrad, wgrad)
  CUtensorMap z, y;  // the outputs (forward with GELU)
};

template <int BN, int MODE, int G, int EPI>
struct ConvShape {
  // forward: K block of G channels (pairs: 64); dgrad: 64 output channels; wgrad: 64 pixels
  static constexpr int kBK = MODE == kConvFwd ? G : 64;
  static constexpr int kNB = MODE == kConvFwd || MODE == kConvPair ? BN : (BN < 64 ? 64 : BN);  // columns staged of B
  static constexpr uint32_t kBytesA = 128 * kBK * 2;
  static constexpr uint32_t kBytesB = MODE == kConvPair ? 0 : kNB * kBK * 2;
  static constexpr uint32_t kWeights = MODE == kConvPair ? 9 * BN * 64 : 0;  // resident
  static constexpr uint32_t kStage = kBytesA + kBytesB;
  // The forward's z and gelu(z) leave as TMA tiles of kSlab columns: stored by the lanes
  // (a row each, 16 bytes at a time) every sector was written in two halves (64 -> 128
  // channels, stride 2, 8 x 256 x 256: forward 0.047 -> 0.035 ms, B200).
  static constexpr bool kStaged = (MODE == kConvFwd && EPI == kConvGelu) || MODE == kConvPair;
  static constexpr int kSlab = BN < 64 ? 32 : 64;
  static constexpr uint32_t kTile = 128 * kSlab * 2;
  static constexpr int kBufs = BN == 256 ? 1 : 2;  // pairs of such tiles (256: four stages first)
  static constexpr uint32_t kStaging = kStaged ? kBufs * 2 * kTile : 0;
  static constexpr int kRoom = kStaged ? 230400 - (int)(kStaging + kWeights) : 196608;
  static constexpr int kStages = kRoom / (int)kStage < 8 ? kRoom / (int)kStage : 8;
  static constexpr size_t kSmem = 1024 + (size_t)kStages * kStage + kStaging + kWeights + 256;
  // dgrad: each tap has columns of its own, and as many taps as fit 256 columns are handed
  // to the epilogue together (a hand-over takes it some 1100 cycles, a tap of 64 channels
  // and columns 128 of the tensor cores).  From 128 columns on, four warps per 32 lanes hold the
  // tile's sums.  With gelu'(z), B200: 64 -> 64 channels, 16 x 256 x 256: 0.245 ms (0.341 with a
  // tap a hand-over); 64 -> 128, stride 2, 8 x 256 x 256: 0.091 (0.097); 256 -> 256, 32 x 64 x 64:
  // 0.172.  All taps in one accumulator took 0.185, 0.084 and 0.137, and rounded 9 N products
  // in a row.
  static constexpr int kTogether = MODE == kConvDgrad ? 256 / BN : 1;
  static constexpr uint32_t kAccCols = kTogether * BN;
  static constexpr uint32_t kCols = 2 * kAccCols;  // two accumulators (64 .. 512 columns)
  static constexpr int kEpi = MODE == kConvDgrad && BN >= 128 ? 16 : kEpiWarps;
  static constexpr int kGroups = kEpi / 4;  // column groups: 32 of every 32 kGroups
  static constexpr int kThreads = 64 + 32 * kEpi;
};

struct Item {
  int x0, y0, b0;  // first pixel of the tile
  int n0;          // first column
  int cls;         // dgrad: parity class
  int kb0, kb1;    // wgrad: pixel blocks of the split
  int split;
};

template <int MODE>
__device__ __forceinline__ Item item_of(const ConvArgs& g, int it, int bn) {
  Item r;
  r.cls = 0;
  r.kb0 = r.kb1 = r.split = 0;
  if (MODE == kConvWgrad) {
    // tile of 128 columns of gw innermost: concurrent CTAs share the pixels
    const int jt = (g.kp + 127) / 128, per = jt * g.tiles_n;
    r.split = it / per;
    const int t = it - r.split * per;
    r.x0 = (t % jt) * 128;  // first column of gw
    r.n0 = (t / jt) * bn;   // first output channel
    r.y0 = r.b0 = 0;
    const int total = g.pt[0].tx * g.pt[0].ty * g.pt[0].tb;
    r.kb0 = r.split * g.kb_per_split;
    r.kb1 = min(total, r.kb0 + g.kb_per_split);
    return r;
  }
  if (MODE == kConvDgrad) {
    while (r.cls + 1 < g.classes && it >= g.first[r.cls + 1]) ++r.cls;
    it -= g.first[r.cls];
  }
  const PixelTiles& p = g.pt[MODE == kConvDgrad ? r.cls : 0];
  const int m = it / g.tiles_n;
  r.n0 = (it - m * g.tiles_n) * bn;
  const int row = m / p.tx;
  r.x0 = (m - row * p.tx) << p.lw;
  r.b0 = row / p.ty * p.bb;
  r.y0 = (row % p.ty) << p.lh;
  return r;
}

// Eight neighbouring outputs of the forward (bias added): FP32, or z and gelu(z).
template <int EPI>
__device__ __forceinline__ void store_outputs(float* d, __nv_bfloat16* z, __nv_bfloat16* y,
                                              size_t at, const float (&v)[8]) {
  if (EPI == kConvF32) {
    float4* o = reinterpret_cast<float4*>(d + at);
    o[0] = make_float4(v[0], v[1], v[2], v[3]);
    o[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    __align__(16) __nv_bfloat162 z2[4], y2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      z2[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
      const float2 g = gelu2(make_float2(v[2 * k], v[2 * k + 1]));
      y2[k] = __floats2bfloat162_rn(g.x, g.y);
    }
    *reinterpret_cast<uint4*>(z + at) = *reinterpret_cast<uint4*>(z2);
    *reinterpret_cast<uint4*>(y + at) = *reinterpret_cast<uint4*>(y2);
  }
}

// dgrad with stride 2: class k covers the pixels of parity (py, px), heaviest
// class (four taps) first.
__device__ __forceinline__ int class_py(int cls) { return cls < 2 ? 1 : 0; }
__device__ __forceinline__ int class_px(int cls) { return (cls & 1) ^ 1; }

// Tap k of the taps that reach the pixels of a class, in ascending (ky, kx): pixel (y, x)
// of the class reads dz(y + oy, x + ox) through it.
struct DgradTap {
  int ky, kx, oy, ox;
};
__device__ __forceinline__ int dgrad_taps(int stride, int cls) {
  return stride == 1 ? 9 : (class_py(cls) ? 2 : 1) * (class_px(cls) ? 2 : 1);
}
__device__ __forceinline__ DgradTap dgrad_tap(int stride, int cls, int k) {
  DgradTap t;
  if (stride == 1) {
    t.ky = k / 3, t.kx = k - 3 * t.ky;
    t.oy = 1 - t.ky, t.ox = 1 - t.kx;
  } else {
    // iy = 2 y + py reads oy = (iy + 1 - ky) / 2: ky = 1 for even rows, 0 and 2 for odd
    const int py = class_py(cls), px = class_px(cls);
    t.ky = py ? 2 * (px ? k >> 1 : k) : 1, t.kx = px ? 2 * (k & 1) : 1;
    t.oy = py && t.ky == 0 ? 1 : 0, t.ox = px && t.kx == 0 ? 1 : 0;
  }
  return t;
}

// Barrier of the epilogue's warps, and the same with a vote.
__device__ __forceinline__ void epi_sync() {
  __syncwarp();
  asm volatile("barrier.cta.sync.aligned 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
}
__device__ __forceinline__ bool epi_all(bool mine) {
  __syncwarp();
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.aligned.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"(mine ? 1u : 0u), "n"(32 * kEpiWarps)
      : "memory");
  return all != 0u;
}

template <int BN, int MODE, int G, int EPI>
__global__ void __launch_bounds__(ConvShape<BN, MODE, G, EPI>::kThreads, 1)
    conv3x3_kernel(const __grid_constant__ ConvMaps maps, const __grid_constant__ ConvArgs g) {
  using S = ConvShape<BN, MODE, G, EPI>;
  constexpr int kStages = S::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* staging = smem + (size_t)kStages * S::kStage;
  uint8_t* weights = staging + S::kStaging;
  uint64_t* full = (uint64_t*)(weights + S::kWeights);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* drained = acc_empty + 2;
  uint64_t* wfull = drained + 1;
  uint32_t* tmem_slot = (uint32_t*)(wfull + 1);
  __shared__ int failed;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = g.first[g.classes];

  if (threadIdx.x == 0) {
    failed = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], S::kEpi);
    }
    mbar_init(drained, 1);
    mbar_init(wfull, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(S::kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // A work item is sums_of sums of blocks_of K blocks each, kTogether sums at a time.
  auto sums_of = [&](const Item& t) {
    return MODE == kConvDgrad ? dgrad_taps(g.stride, t.cls) : 1;
  };
  auto blocks_of = [&](const Item& t) {
    if (MODE == kConvFwd) return 9 * (g.C / G);
    if (MODE == kConvPair) return 6;
    if (MODE == kConvWgrad) return t.kb1 - t.kb0;
    return (g.N + 63) / 64;
  };

  int issued = 0;
  if (warp == 0 && lane == 0) {
    bool ok = true;
    if (MODE == kConvPair) {
      mbar_expect_tx(wfull, S::kWeights);
      for (int tap = 0; tap < 9; ++tap)
        tma_load_2d(weights + tap * BN * 64, &maps.w, wfull, tap * 32, 0);
    }
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
      const Item t = item_of<MODE>(g, it, BN);
      const int nkb = sums_of(t) * blocks_of(t);
      for (int i = 0; i < nkb; ++i) {
        const int s = issued % kStages;
        if (!mbar_wait(&empty[s], ((uint32_t)(issued / kStages) & 1u) ^ 1u, g.spin)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], S::kStage);
        uint8_t* a = smem + (size_t)s * S::kStage;
        uint8_t* b = a + S::kBytesA;
        if (MODE == kConvFwd) {
          const int cpb = g.C / G, tap = i / cpb, c = (i - tap * cpb) * G;
          tma_load_4d(a, &maps.x[tap], &full[s], c, t.x0 + g.off_x[tap], t.y0 + g.off_y[tap],
                      t.b0);
          tma_load_2d(b, &maps.w, &full[s], tap * g.C + c, t.n0);
        } else if (MODE == kConvPair) {
          // even blocks: the pairs before, odd ones: the pairs themselves
          const int ky = i >> 1;
          tma_load_4d(a, &maps.x[ky], &full[s], 0, t.x0 - 1 + (i & 1), t.y0 + g.off_y[ky], t.b0);
        } else if (MODE == kConvDgrad) {
          const int nb = (g.N + 63) / 64, k = i / nb, n = (i - k * nb) * 64;
          const DgradTap tap = dgrad_tap(g.stride, t.cls, k);
          tma_load_4d(a, &maps.dz, &full[s], n, t.x0 + tap.ox, t.y0 + tap.oy, t.b0);
          const int c = (tap.ky * 3 + tap.kx) * g.C + t.n0;
#pragma unroll
          for (int j = 0; j < S::kNB / 64; ++j)
            tma_load_2d(b + j * 8192, &maps.w, &full[s], c + 64 * j, n);
        } else {
          const PixelTiles& p = g.pt[0];
          const int m = t.kb0 + i, row = m / p.tx;
          const int x0 = (m - row * p.tx) << p.lw, y0 = (row % p.ty) << p.lh,
                    b0 = row / p.ty * p.bb;
#pragma unroll
          for (int j = 0; j < 128 / G; ++j) {
            // columns past 9C load from past the images: zeros
            const int col = t.x0 + j * G, tap = min(col / g.C, 8), c = col - tap * g.C;
            const bool in = col < 9 * g.C;
            tma_load_4d(a + j * G * 128, &maps.x[tap], &full[s], in ? c : 0,
                        x0 + g.off_x[tap], y0 + g.off_y[tap], in ? b0 : g.B);
          }
#pragma unroll
          for (int j = 0; j < S::kNB / 64; ++j)
            tma_load_4d(b + j * 8192, &maps.dz, &full[s], t.n0 + 64 * j, x0, y0, b0);
        }
        ++issued;
      }
    }
  } else if (warp == 1 && lane == 0) {
    constexpr uint32_t idesc =
        instr_desc_bf16(128, BN, MODE == kConvWgrad, MODE != kConvFwd && MODE != kConvPair);
    bool ok = true;
    if (MODE == kConvPair && !mbar_wait(wfull, 0, g.spin)) {
      atomicExch(&failed, 1);
      ok = false;
    }
    int n = 0, turn = 0;  // K blocks and accumulators issued
    for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
      const Item t = item_of<MODE>(g, it, BN);
      const int nkb = blocks_of(t), sums = sums_of(t);
      for (int j = 0; j < sums && ok; j += S::kTogether, ++turn) {
        const int acc = turn & 1;
        if (!mbar_wait(&acc_empty[acc], ((uint32_t)(turn >> 1) & 1u) ^ 1u, g.spin)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int blocks = min(S::kTogether, sums - j) * nkb;
        uint32_t d = tmem + acc * S::kAccCols;
        for (int k = 0, i = 0; k < blocks; ++k, ++n) {
          const int s = n % kStages;
          if (!mbar_wait(&full[s], (uint32_t)(n / kStages) & 1u, g.spin)) {
            atomicExch(&failed, 1);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = smem_u32(smem + (size_t)s * S::kStage), b = a + S::kBytesA;
#pragma unroll
          for (int kk = 0; kk < S::kBK / 16; ++kk) {
            if (MODE == kConvPair && !(i & 1) && kk < 2) continue;  // the second pixel only
            // K-major rows of G (64) channels: 16 channels further are 32 bytes.
            // MN-major: 8-row groups of 128 (64) bytes, 16 rows further two groups,
            // the next 64 (32) columns a whole K block further.
            const uint64_t da =
                MODE == kConvWgrad
                    ? smem_desc(a + kk * G * 32, G * 128, G * 16, G == 64 ? 2u : 4u)
                    : smem_desc(a + kk * 32, 16, S::kBK * 16, S::kBK == 64 ? 2u : 4u);
            const uint64_t db =
                MODE == kConvPair
                    ? smem_desc(smem_u32(weights) +
                                    ((i >> 1) * 3 + (i & 1 ? 1 + (kk >> 1) : 0)) * BN * 64 +
                                    (kk & 1) * 32,
                                16, 512, 4u)
                : MODE == kConvFwd ? smem_desc(b + kk * 32, 16, G * 16, G == 64 ? 2u : 4u)
                                 : smem_desc(b + kk * 2048, 8192, 1024, 2u);
            umma_bf16(d, da, db, idesc,
                      (i > 0 || kk > (MODE == kConvPair ? 2 : 0)) ? 1u : 0u);
          }
          umma_commit(&empty[s]);
          if (++i == nkb && MODE == kConvDgrad) i = 0, d += BN;  // the next tap
        }
        umma_commit(&acc_full[acc]);
      }
    }
    umma_commit(drained);
  } else if (warp >= 2) {
    const int quad = warp & 3;  // the TMEM lanes this warp may read: 32 quad ..
    const int row = quad * 32 + lane;
    const int group = (warp - 2) / 4;  // of the columns (of a slab's)
    // The accumulator of a turn in this warp's lanes, once it is complete: -1 if the wait
    // ran out.  Staged: the epilogue's warps meet at barriers, so they leave together.
    auto take = [&](int turn) {
      const int acc = turn & 1;
      const bool got = mbar_wait(&acc_full[acc], (uint32_t)(turn >> 1) & 1u, g.spin);
      if (S::kStaged ? !epi_all(got) : !__all_sync(0xffffffffu, got)) {
        atomicExch(&failed, 1);
        return -1;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return (int)(tmem + acc * S::kAccCols + ((uint32_t)(quad * 32) << 16));
    };
    auto give_back = [&](int turn) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                         smem_u32(&acc_empty[turn & 1]))
                     : "memory");
    };
    int turn = 0, slabs = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
      const Item t = item_of<MODE>(g, it, BN);
      bool valid = false;
      size_t pix = 0;
      int x = 0, y = 0;
      if (MODE != kConvWgrad) {
        const PixelTiles& p = g.pt[MODE == kConvDgrad ? t.cls : 0];
        x = t.x0 + (row & ((1 << p.lw) - 1));
        y = t.y0 + ((row >> p.lw) & ((1 << p.lh) - 1));
        const int b = t.b0 + (row >> (p.lw + p.lh));
        if (MODE == kConvFwd || MODE == kConvPair) {
          valid = x < g.Wo && y < g.Ho && b < g.B;
          pix = ((size_t)b * g.Ho + y) * g.Wo + x;
        } else {
          const int s = g.stride, ix = s == 2 ? 2 * x + class_px(t.cls) : x;
          const int iy = s == 2 ? 2 * y + class_py(t.cls) : y;
          valid = ix < g.W && iy < g.H && b < g.B;
          pix = ((size_t)b * g.H + iy) * g.W + ix;
        }
      }
      if (MODE == kConvDgrad) {
        constexpr int kWide = 32 * S::kGroups;
        constexpr int kParts = (BN + kWide - 1) / kWide;  // of 32 columns: 32 group + kWide j
        float sum[kParts][32];
#pragma unroll
        for (int j = 0; j < kParts; ++j)
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[j][q] = 0.f;
        const int taps = dgrad_taps(g.stride, t.cls);
        int ta = 0;
#pragma unroll 1
        for (int k0 = 0; k0 < taps; k0 += S::kTogether, ++turn) {
          ta = take(turn);
          if (ta == -1) break;
          const int k1 = min(taps, k0 + S::kTogether);
#pragma unroll 1
          for (int k = k0; k < k1; ++k) {
            // a tap that reads past dz adds nothing (not 0 times its weight)
            const DgradTap tap = dgrad_tap(g.stride, t.cls, k);
            const bool reads = (unsigned)(y + tap.oy) < (unsigned)g.Ho &&
                               (unsigned)(x + tap.ox) < (unsigned)g.Wo;
#pragma unroll
            for (int j = 0; j < kParts; ++j) {
              if (32 * group + kWide * j >= BN) continue;
              constexpr int kRead = kParts > 1 ? 16 : 32;  // (registers)
#pragma unroll
              for (int h = 0; h < 32; h += kRead) {
                uint32_t r[kRead];
                tmem_ld((uint32_t)ta + (uint32_t)((k - k0) * BN + 32 * group + kWide * j + h), r);
                if (reads) {
#pragma unroll
                  for (int q = 0; q < kRead; ++q) sum[j][h + q] += __uint_as_float(r[q]);
                }
                __syncwarp();
              }
            }
          }
          give_back(turn);
        }
        if (ta == -1) break;
#pragma unroll
        for (int j = 0; j < kParts && valid; ++j) {
          const int c0 = t.n0 + 32 * group + kWide * j;
          const size_t base = pix * g.C + c0;
#pragma unroll
          for (int q = 0; q < 32; q += 8) {
            if (32 * group + kWide * j >= BN || c0 + q >= g.C) break;  // C is a multiple of 8
            if (g.zprev) {
              __align__(16) __nv_bfloat162 z2[4];
              *reinterpret_cast<uint4*>(z2) = *reinterpret_cast<const uint4*>(g.zprev + base + q);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 slope = gelu_grad2(__bfloat1622float2(z2[k]));
                sum[j][q + 2 * k] *= slope.x;
                sum[j][q + 2 * k + 1] *= slope.y;
              }
            }
            __align__(16) __nv_bfloat162 y2[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
              y2[k] = __floats2bfloat162_rn(sum[j][q + 2 * k], sum[j][q + 2 * k + 1]);
            *reinterpret_cast<uint4*>(g.y + base + q) = *reinterpret_cast<uint4*>(y2);
          }
        }
        __syncwarp();
        continue;
      }
      const int got = take(turn);
      if (got == -1) break;
      const uint32_t ta = (uint32_t)got;
      if (S::kStaged) {
#pragma unroll 1
        for (int n = 0; n < BN && t.n0 + n < g.N; n += S::kSlab, ++slabs) {
          uint8_t* tz = staging + (size_t)(slabs % S::kBufs) * 2 * S::kTile;
          uint8_t* ty = tz + S::kTile;
          if (warp == 2 && lane == 0) bulk_wait_read<S::kBufs - 1>();
          epi_sync();
          if (group * 32 < S::kSlab) {
            uint32_t r[32];
            tmem_ld(ta + (uint32_t)(n + 32 * group), r);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float v[8];
              const int c = t.n0 + n + 32 * group + 8 * q;  // N is a multiple of 8
#pragma unroll
              for (int k = 0; k < 8; ++k) v[k] = __uint_as_float(r[8 * q + k]);
              if (c < g.N) {
                const float4* bias = reinterpret_cast<const float4*>(g.bias + c);
                const float4 b0 = bias[0], b1 = bias[1];
                v[0] += b0.x, v[1] += b0.y, v[2] += b0.z, v[3] += b0.w;
                v[4] += b1.x, v[5] += b1.y, v[6] += b1.z, v[7] += b1.w;
              }
              // the tensor maps' swizzle: 128-byte rows, or 64-byte ones
              const int chunk = group * 4 + q;
              const int at = S::kSlab == 64 ? row * 128 + ((chunk ^ (row & 7)) << 4)
                                            : row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
              store_outputs<kConvGelu>(nullptr, reinterpret_cast<__nv_bfloat16*>(tz),
                                       reinterpret_cast<__nv_bfloat16*>(ty), (size_t)(at / 2), v);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          epi_sync();
          if (warp == 2 && lane == 0) {
            tma_store_4d(&maps.z, tz, t.n0 + n, t.x0, t.y0, t.b0);
            tma_store_4d(&maps.y, ty, t.n0 + n, t.x0, t.y0, t.b0);
            bulk_commit();
          }
        }
      } else {
#pragma unroll 1
        for (int c0 = group * 32; c0 < BN; c0 += 32 * S::kGroups) {
          uint32_t r[32];
          tmem_ld(ta + (uint32_t)c0, r);
          if (MODE == kConvWgrad) {
            // rows are columns of gw: the lanes write 128 contiguous bytes
            const int j = t.x0 + row;
            float* dst = g.d + ((size_t)t.split * g.N + t.n0 + c0) * g.kp + j;
            if (j < g.kp) {
#pragma unroll
              for (int q = 0; q < 32; ++q)
                if (t.n0 + c0 + q < g.N) dst[(size_t)q * g.kp] = __uint_as_float(r[q]);
            }
          } else if (valid) {
            const size_t base = pix * g.N + t.n0 + c0;
#pragma unroll
            for (int q = 0; q < 32; q += 8) {
              if (t.n0 + c0 + q >= g.N) break;  // N is a multiple of 8
              float v[8];
              const float4* bias = reinterpret_cast<const float4*>(g.bias + t.n0 + c0 + q);
              const float4 b0 = bias[0], b1 = bias[1];
#pragma unroll
              for (int k = 0; k < 8; ++k) v[k] = __uint_as_float(r[q + k]);
              v[0] += b0.x, v[1] += b0.y, v[2] += b0.z, v[3] += b0.w;
              v[4] += b1.x, v[5] += b1.y, v[6] += b1.z, v[7] += b1.w;
              store_outputs<EPI>(g.d, g.z, g.y, base + q, v);
            }
          }
        }
      }
      give_back(turn++);
    }
    if (S::kStaged && warp == 2 && lane == 0) bulk_wait_all();
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (failed) {
    // Drain before freeing TMEM and shared memory: the copies still in flight
    // (at most the last kStages issued: a stage is reused only once its copy
    // has landed and been consumed) and every MMA, committed to `drained`.
    if (warp == 0 && lane == 0) {
      for (int i = max(0, issued - kStages); i < issued; ++i)
        mbar_wait(&full[i % kStages], (uint32_t)(i / kStages) & 1u, kSpinLimit);
      if (MODE == kConvPair) mbar_wait(wfull, 0, kSpinLimit);
      mbar_wait(drained, 0, kSpinLimit);
      atomicOr(g.err, 1u);
    }
    __syncthreads();
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(S::kCols));
  }
}

// First layer, three input channels: out = x * w + bias with the 27 products of a
// pixel padded to one K block of 32.  Each thread gathers its pixel's row (nine
// taps of three channels) into the swizzled A tile, two tcgen05.mma make the
// 128 x BN tile, and the same threads write z and gelu(z).  Bound by the output
// (2 x 2 BN bytes a pixel): an im2col matrix of 64 columns would move 128 bytes
// a pixel twice more.  Many small CTAs per SM (8 of 128 threads at BN = 32)
// overlap one another's gather, MMA and epilogue, so no warp is specialised.  A row of
// nine values is loaded as five aligned words, and the tiles of z and gelu(z) are
// stored by TMA.  On 16 images of 512 x 512 (B200): 2.3 ms as im2col + GEMM, 0.231 with
// two-byte loads and 16-byte stores a lane, 0.216 with word loads, 0.111 with TMA
// stores; the 0.56 GB alone take 0.086.
constexpr int kRgbThreads = 128;

struct RgbArgs {
  const __nv_bfloat16 *x, *w;
  int B, H, W, Ho, Wo, N, stride, kp;
  uint32_t pixels;
  const float* bias;
  __nv_bfloat16 *z, *y;
  float* d;
  uint32_t* err;
  uint32_t spin;
};

struct RgbMaps {
  CUtensorMap z, y;  // [pixels][N], boxes of 128 x BN
};

template <int BN, int EPI>
__global__ void __launch_bounds__(kRgbThreads)
    conv3x3_rgb_kernel(const RgbArgs g, const __grid_constant__ RgbMaps maps) {
  constexpr int kK = 32;  // 27 products and five zeros
  __shared__ __align__(1024) uint8_t sA[128 * kK * 2];
  __shared__ __align__(1024) uint8_t sB[BN * kK * 2];
  constexpr bool kStaged = EPI == kConvGelu;
  __shared__ __align__(1024) uint8_t sOut[kStaged ? 2 : 1][kStaged ? 128 * BN * 2 : 16];
  __shared__ uint64_t done;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float sBias[BN];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.y * BN;
  if (threadIdx.x == 0) {
    mbar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"((uint32_t)BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // rows of 32 BF16 (64 B), 64-byte swizzle: 16-byte chunk q of row r at q ^ (r >> 1 & 3)
  auto chunk = [](uint8_t* tile, int r, int q) {
    return reinterpret_cast<uint4*>(tile + r * 64 + ((q ^ ((r >> 1) & 3)) << 4));
  };
  auto pack = [](uint32_t lo, uint32_t hi) { return lo | (hi << 16); };
  for (int r = threadIdx.x; r < BN; r += kRgbThreads) {
    uint32_t v[kK];
    const unsigned short* w = reinterpret_cast<const unsigned short*>(g.w) +
                              (size_t)min(n0 + r, g.N - 1) * g.kp;
#pragma unroll
    for (int k = 0; k < kK; ++k) v[k] = n0 + r < g.N && k < 27 ? w[k] : 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *chunk(sB, r, q) = make_uint4(pack(v[8 * q], v[8 * q + 1]), pack(v[8 * q + 2], v[8 * q + 3]),
                                    pack(v[8 * q + 4], v[8 * q + 5]),
                                    pack(v[8 * q + 6], v[8 * q + 7]));
    sBias[r] = n0 + r < g.N ? g.bias[n0 + r] : 0.f;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const uint32_t tiles = (g.pixels + 127) / 128;
  const unsigned short* x = reinterpret_cast<const unsigned short*>(g.x);
  const int64_t values = (int64_t)g.B * g.H * g.W * 3;
  uint32_t phase = 0;
  bool ok = true;
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint32_t m = t * 128 + threadIdx.x;
    uint32_t v[kK / 2];  // pairs of products
#pragma unroll
    for (int k = 0; k < kK / 2; ++k) v[k] = 0u;
    if (m < g.pixels) {
      const uint32_t row = m / (uint32_t)g.Wo;
      const int ox = (int)(m - row * (uint32_t)g.Wo);
      const uint32_t b = row / (uint32_t)g.Ho;
      const int oy = (int)(row - b * (uint32_t)g.Ho);
      const int iy0 = oy * g.stride - 1, ix0 = ox * g.stride - 1;
      // nine neighbouring values per image row
      const int64_t at = (((int64_t)b * g.H + iy0) * g.W + ix0) * 3, pitch = (int64_t)g.W * 3;
      if (iy0 >= 0 && iy0 + 2 < g.H && ix0 >= 0 && ix0 + 2 < g.W && at + 2 * pitch + 9 < values) {
        // inside: five aligned words cover a row, whichever half it starts in
        uint32_t a[3][5];
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          const int64_t h = at + ky * pitch;
          const uint32_t* word = reinterpret_cast<const uint32_t*>(x) + (h >> 1);
          const uint32_t odd = 16u * (uint32_t)(h & 1);
          uint32_t u[6];
#pragma unroll
          for (int k = 0; k < 5; ++k) u[k] = word[k];
          u[5] = 0u;
#pragma unroll
          for (int k = 0; k < 5; ++k) a[ky][k] = __funnelshift_r(u[k], u[k + 1], odd);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[k] = a[0][k];
          v[5 + k] = __funnelshift_r(a[1][k], a[1][k + 1], 16);
          v[9 + k] = a[2][k];
        }
        v[4] = __byte_perm(a[0][4], a[1][0], 0x5410);
        v[13] = a[2][4] & 0xffffu;
      } else {
        uint32_t e[kK];
#pragma unroll
        for (int k = 0; k < kK; ++k) e[k] = 0u;
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          const int iy = iy0 + ky;
#pragma unroll
          for (int kx = 0; kx < 3; ++kx)
            if (iy >= 0 && iy < g.H && ix0 + kx >= 0 && ix0 + kx < g.W) {
#pragma unroll
              for (int c = 0; c < 3; ++c)
                e[(ky * 3 + kx) * 3 + c] = x[at + ky * pitch + kx * 3 + c];
            }
        }
#pragma unroll
        for (int k = 0; k < kK / 2; ++k) v[k] = pack(e[2 * k], e[2 * k + 1]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *chunk(sA, threadIdx.x, q) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int kk = 0; kk < kK / 16; ++kk)
        umma_bf16(tmem, smem_desc(smem_u32(sA) + kk * 32, 16, 512, 4u),
                  smem_desc(smem_u32(sB) + kk * 32, 16, 512, 4u), instr_desc_bf16(128, BN),
                  kk > 0 ? 1u : 0u);
      umma_commit(&done);
    }
    __syncwarp();
    // Every thread polls to the same limit; a timeout is voted on, so that the
    // whole CTA leaves together.
    ok = mbar_wait(&done, phase, g.spin);
    if (kStaged && threadIdx.x == 0) bulk_wait_read<0>();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    phase ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 32) {
      uint32_t r[32];
      tmem_ld(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
      if (kStaged) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(r[8 * q + k]) + sBias[c0 + 8 * q + k];
          const int row = threadIdx.x, chunk = c0 / 8 + q;
          const int at = BN == 64 ? row * 128 + ((chunk ^ (row & 7)) << 4)
                                  : row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
          store_outputs<kConvGelu>(nullptr, reinterpret_cast<__nv_bfloat16*>(sOut[0]),
                                   reinterpret_cast<__nv_bfloat16*>(sOut[kStaged ? 1 : 0]),
                                   (size_t)(at / 2), f);
        }
      } else if (m < g.pixels) {
        const size_t base = (size_t)m * g.N + n0 + c0;
#pragma unroll
        for (int q = 0; q < 32; q += 8) {
          if (n0 + c0 + q >= g.N) break;
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(r[q + k]) + sBias[c0 + q + k];
          store_outputs<EPI>(g.d, g.z, g.y, base + q, f);
        }
      }
    }
    // the accumulator and the A tile are free again once every thread has read
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (kStaged) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (kStaged && threadIdx.x == 0) {
      tma_store_2d(&maps.z, sOut[0], n0, (int)(t * 128));
      tma_store_2d(&maps.y, sOut[kStaged ? 1 : 0], n0, (int)(t * 128));
      bulk_commit();
    }
  }
  if (kStaged && threadIdx.x == 0) bulk_wait_all();
  if (!ok && threadIdx.x == 0) {
    mbar_wait(&done, phase, kSpinLimit);  // the MMAs land before TMEM is freed
    atomicOr(g.err, 1u);
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)BN));
  }
}

// gw = sum of the split partials in split order, four values per thread, eight
// partials in flight.
__global__ void __launch_bounds__(256)
    conv_reduce_kernel(const float4* __restrict__ p, float4* __restrict__ out, int n4,
                       int splits) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = 0; k < splits; ++k) {
    const float4 v = p[(size_t)k * n4 + i];
    s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
  }
  out[i] = s;
}

// ---- host side ----------------------------------------------------------------

// The rectangle of `pixels` (a power of two) pixels over B images of W x H that
// needs the fewest tiles; among equals the widest.
PixelTiles pick_tiles(int pixels, int W, int H, int B) {
  PixelTiles best{};
  int64_t fewest = INT64_MAX;
  int total = 0;
  while ((1 << total) < pixels) ++total;
  for (int lw = total; lw >= 0; --lw)
    for (int lh = total - lw; lh >= 0; --lh) {
      const int bw = 1 << lw, bh = 1 << lh, bb = pixels >> (lw + lh);
      PixelTiles p{lw, lh, bb, (W + bw - 1) / bw, (H + bh - 1) / bh, (B + bb - 1) / bb};
      const int64_t n = (int64_t)p.tx * p.ty * p.tb;
      if (n < fewest) {
        fewest = n;
        best = p;
      }
    }
  return best;
}

int64_t count_of(const PixelTiles& p) { return (int64_t)p.tx * p.ty * p.tb; }

int encode(CUtensorMap* map, int rank, const void* base, const cuuint64_t* dims,
           const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  EncodeFn fn = encode_fn();
  if (!fn) return DS_ERR_CUDA;
  const cuuint32_t one[4] = {1, 1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank,
                        const_cast<void*>(base), dims, strides, box, one,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? DS_OK : DS_ERR_ARG;
}

// Box of `group` channels over a rectangle of pixels of an NHWC view.
int map_pixels(CUtensorMap* map, const __nv_bfloat16* base, int C, int W, int H, int B,
               int64_t sx, int64_t sy, int64_t sb, int group, const PixelTiles& p) {
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)sx * 2, (cuuint64_t)sy * 2, (cuuint64_t)sb * 2};
  const cuuint32_t box[4] = {(cuuint32_t)group, 1u << p.lw, 1u << p.lh, (cuuint32_t)p.bb};
  return encode(map, 4, base, dims, strides, box,
                group == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

// The nine taps of x in output-pixel coordinates (see the file's head).
int map_taps(ConvMaps& maps, ConvArgs& g, const __nv_bfloat16* x, int group,
             const PixelTiles& p) {
  const int s = g.stride;
  for (int tap = 0; tap < 9; ++tap) {
    const int ky = tap / 3, kx = tap - 3 * ky;
    // output rows whose input row oy s - 1 + ky lies inside: [oy0, oy1)
    const int oy0 = ky == 0 ? 1 : 0, ox0 = kx == 0 ? 1 : 0;
    const int oy1 = std::min(g.Ho, (g.H - ky) / s + 1), ox1 = std::min(g.Wo, (g.W - kx) / s + 1);
    const bool none = oy1 <= oy0 || ox1 <= ox0 || g.H < ky || g.W < kx;
    const int iy = oy0 * s - 1 + ky, ix = ox0 * s - 1 + kx;
    const __nv_bfloat16* base = none ? x : x + ((int64_t)iy * g.W + ix) * g.C;
    // a tap that reads nothing gets coordinates outside of a one-pixel map
    g.off_x[tap] = none ? 1 << 24 : -ox0;
    g.off_y[tap] = none ? 1 << 24 : -oy0;
    DS_TRY(map_pixels(&maps.x[tap], base, g.C, none ? 1 : ox1 - ox0, none ? 1 : oy1 - oy0, g.B,
                      (int64_t)s * g.C, (int64_t)s * g.W * g.C, (int64_t)g.H * g.W * g.C, group,
                      p));
  }
  return DS_OK;
}

// The image rows 2 oy - 1 + ky as rows of pixel pairs.
int map_pairs(ConvMaps& maps, ConvArgs& g, const __nv_bfloat16* x, const PixelTiles& p) {
  for (int ky = 0; ky < 3; ++ky) {
    const int oy0 = ky == 0 ? 1 : 0, oy1 = std::min(g.Ho, (g.H - ky) / 2 + 1);
    const bool none = oy1 <= oy0 || g.H < ky;
    g.off_y[ky] = none ? 1 << 24 : -oy0;
    DS_TRY(map_pixels(&maps.x[ky],
                      none ? x : x + (int64_t)(oy0 * 2 - 1 + ky) * g.W * g.C, 64, g.W / 2,
                      none ? 1 : oy1 - oy0, g.B, 64, 2 * (int64_t)g.W * g.C,
                      (int64_t)g.H * g.W * g.C, 64, p));
  }
  return DS_OK;
}

int map_matrix(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_cols,
               int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  return encode(map, 2, base, dims, strides, box,
                box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

int sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int BN, int MODE, int G, int EPI>
int launch_conv(const ConvMaps& maps, const ConvArgs& g, cudaStream_t s) {
  using S = ConvShape<BN, MODE, G, EPI>;
  static std::atomic<uint64_t> set{0};
  DS_CUDA(allow_smem(conv3x3_kernel<BN, MODE, G, EPI>, S::kSmem, set));
  const int grid = std::min(g.first[g.classes], sm_count());
  conv3x3_kernel<BN, MODE, G, EPI><<<grid, S::kThreads, S::kSmem, s>>>(maps, g);
  return cuda_status(cudaGetLastError());
}

template <int MODE, int G, int EPI>
int dispatch_bn(int bn, const ConvMaps& maps, const ConvArgs& g, cudaStream_t s) {
  switch (bn) {
    case 32: return launch_conv<32, MODE, G, EPI>(maps, g, s);
    case 64: return launch_conv<64, MODE, G, EPI>(maps, g, s);
    case 128: return launch_conv<128, MODE, G, EPI>(maps, g, s);
    default: return launch_conv<256, MODE, G, EPI>(maps, g, s);
  }
}

// Tile width for n columns over `tiles` row tiles: the widest that n fills,
// narrowed while SMs would stay idle.
int pick_bn(int n, int64_t tiles, int least = 32) {
  int bn = n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : 256;
  bn = std::max(bn, least);
  while (bn > 64 && tiles * ((n + bn - 1) / bn) < sm_count()) bn /= 2;
  return bn;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Shapes and addresses the tensor maps and the vector accesses take.
bool conv_ok(int B, int H, int W, int C, int N, int stride, int kp) {
  if (B <= 0 || H <= 0 || W <= 0 || N <= 0 || (stride != 1 && stride != 2)) return false;
  if (!(C == 32 || (C > 0 && C % 64 == 0)) || N % 8 != 0) return false;
  if (kp < 9 * C || kp % 8 != 0) return false;
  // items and pixel tiles are counted in 32 bits
  return (int64_t)B * H * W < ((int64_t)1 << 30) && C <= (1 << 16) && N <= (1 << 16);
}

template <int BN, int EPI>
int launch_rgb(const RgbArgs& g, cudaStream_t s) {
  // TMEM holds 512 / BN accumulators per SM; 8 CTAs (4 of 64 columns, with their tiles in
  // shared memory) are what the SM holds
  const int per_sm = BN == 32 ? 8 : EPI == kConvGelu ? 4 : 8;
  RgbMaps maps{};
  if (EPI == kConvGelu) {
    DS_TRY(map_matrix(&maps.z, g.z, (int)g.pixels, g.N, g.N, BN, 128));
    DS_TRY(map_matrix(&maps.y, g.y, (int)g.pixels, g.N, g.N, BN, 128));
  }
  const int tiles = (int)((g.pixels + 127) / 128), ny = (g.N + BN - 1) / BN;
  const dim3 grid(std::max(1, std::min(tiles, sm_count() * per_sm / ny)), ny);
  conv3x3_rgb_kernel<BN, EPI><<<grid, kRgbThreads, 0, s>>>(g, maps);
  return cuda_status(cudaGetLastError());
}

ConvArgs base_args(int B, int H, int W, int C, int N, int stride, int kp, uint32_t* err) {
  ConvArgs g{};
  g.B = B, g.H = H, g.W = W, g.C = C, g.N = N, g.stride = stride, g.kp = kp;
  g.Ho = (H - 1) / stride + 1, g.Wo = (W - 1) / stride + 1;
  g.classes = 1;
  g.err = err;
  g.spin = gemm_spin_limit();
  return g;
}

// Splits of the weight gradient: chains of at most kWgradChain pixels, and
// enough splits that every SM gets a tile.
void pick_splits(ConvArgs& g, int64_t blocks, int tiles) {
  int64_t per = kWgradChain / kWgradPixels;
  const int64_t want = (sm_count() + tiles - 1) / tiles;
  per = std::min(per, std::max<int64_t>(4, (blocks + want - 1) / want));
  // the partials stay within 512 of them
  per = std::max(per, (blocks + 511) / 512);
  g.kb_per_split = (int)per;
  g.splits = (int)((blocks + per - 1) / per);
}

int wgrad_plan(ConvArgs& g, int& bn) {
  g.pt[0] = pick_tiles(kWgradPixels, g.Wo, g.Ho, g.B);
  const int jt = (g.kp + 127) / 128;
  bn = g.N <= 32 ? 32 : g.N <= 64 ? 64 : g.N <= 128 ? 128 : 256;
  g.tiles_n = (g.N + bn - 1) / bn;
  const int64_t blocks = count_of(g.pt[0]);
  if (blocks > INT32_MAX / 2) return DS_ERR_ARG;
  pick_splits(g, blocks, jt * g.tiles_n);
  g.first[1] = jt * g.tiles_n * g.splits;
  return DS_OK;
}

}  // namespace
}  // namespace ds

extern "C" {

int ds_conv3x3_forward(const void* x, int B, int H, int W, int C, int stride, const void* w,
                       int Kp, int N, const float* bias, void* z, void* y, float* d,
                       uint32_t* err, ds_stream stream) {
  using namespace ds;
  if (!x || !w || !bias || !err || (!d && (!z || !y))) return DS_ERR_ARG;
  if (C == 3) {
    if (!conv_ok(B, H, W, 32, N, stride, 288) || Kp < 27) return DS_ERR_ARG;
    if (!aligned16(z) || !aligned16(y) || !aligned16(d)) return DS_ERR_ARG;
    if ((uintptr_t)x & 3) return DS_ERR_ARG;
    RgbArgs g{};
    g.x = (const __nv_bfloat16*)x, g.w = (const __nv_bfloat16*)w;
    g.B = B, g.H = H, g.W = W, g.N = N, g.stride = stride, g.kp = Kp;
    g.Ho = (H - 1) / stride + 1, g.Wo = (W - 1) / stride + 1;
    g.pixels = (uint32_t)B * g.Ho * g.Wo;
    g.bias = bias;
    g.z = (__nv_bfloat16*)z, g.y = (__nv_bfloat16*)y, g.d = d;
    g.err = err;
    g.spin = gemm_spin_limit();
    cudaStream_t s = (cudaStream_t)stream;
    if (N <= 32)
      return d ? launch_rgb<32, kConvF32>(g, s) : launch_rgb<32, kConvGelu>(g, s);
    return d ? launch_rgb<64, kConvF32>(g, s) : launch_rgb<64, kConvGelu>(g, s);
  }
  if (!conv_ok(B, H, W, C, N, stride, Kp)) return DS_ERR_ARG;
  if (!aligned16(x) || !aligned16(w) || !aligned16(bias) || !aligned16(z) || !aligned16(y) ||
      !aligned16(d))
    return DS_ERR_ARG;
  ConvArgs g = base_args(B, H, W, C, N, stride, Kp, err);
  const int G = C == 32 ? 32 : 64;
  g.pt[0] = pick_tiles(128, g.Wo, g.Ho, B);
  const int64_t tiles = count_of(g.pt[0]);
  const int bn = pick_bn(N, tiles);
  g.tiles_n = (N + bn - 1) / bn;
  if (tiles * g.tiles_n > INT32_MAX) return DS_ERR_ARG;
  g.first[1] = (int)(tiles * g.tiles_n);
  g.bias = bias;
  g.z = (__nv_bfloat16*)z;
  g.y = (__nv_bfloat16*)y;
  g.d = d;
  ConvMaps maps;
  const bool pairs = C == 32 && stride == 2 && W % 2 == 0 && !d && N > 32 && N <= 64;
  DS_TRY(map_matrix(&maps.w, w, N, Kp, Kp, G, bn));
  if (pairs) {
    for (int t = 3; t < 9; ++t) maps.x[t] = maps.w;  // not read
    DS_TRY(map_pairs(maps, g, (const __nv_bfloat16*)x, g.pt[0]));
  } else {
    DS_TRY(map_taps(maps, g, (const __nv_bfloat16*)x, G, g.pt[0]));
  }
  maps.dz = maps.z = maps.y = maps.w;  // not read
  if (!d)
    for (int k = 0; k < 2; ++k)
      DS_TRY(map_pixels(k ? &maps.y : &maps.z, k ? g.y : g.z, N, g.Wo, g.Ho, B, N, (int64_t)g.Wo * N,
                        (int64_t)g.Ho * g.Wo * N, bn < 64 ? 32 : 64, g.pt[0]));
  cudaStream_t s = (cudaStream_t)stream;
  if (pairs) return launch_conv<64, kConvPair, 32, kConvGelu>(maps, g, s);
  if (G == 32)
    return d ? dispatch_bn<kConvFwd, 32, kConvF32>(bn, maps, g, s)
             : dispatch_bn<kConvFwd, 32, kConvGelu>(bn, maps, g, s);
  return d ? dispatch_bn<kConvFwd, 64, kConvF32>(bn, maps, g, s)
           : dispatch_bn<kConvFwd, 64, kConvGelu>(bn, maps, g, s);
}

int ds_conv3x3_dgrad(const void* dz, int B, int H, int W, int C, int stride, const void* w,
                     int Kp, int N, const void* zprev, void* dx, uint32_t* err,
                     ds_stream stream) {
  using namespace ds;
  if (!dz || !w || !dx || !err) return DS_ERR_ARG;
  if (!conv_ok(B, H, W, C, N, stride, Kp)) return DS_ERR_ARG;
  if (!aligned16(dz) || !aligned16(w) || !aligned16(zprev) || !aligned16(dx)) return DS_ERR_ARG;
  ConvArgs g = base_args(B, H, W, C, N, stride, Kp, err);
  g.zprev = (const __nv_bfloat16*)zprev;
  g.y = (__nv_bfloat16*)dx;
  int64_t tiles = 0;
  // All classes use one rectangle (the box of the dz map), picked for the
  // largest class: the even rows and columns.
  const int Wc = (W + stride - 1) / stride, Hc = (H + stride - 1) / stride;
  const PixelTiles p = pick_tiles(128, Wc, Hc, B);
  const int bn = pick_bn(C, count_of(p) * stride * stride);
  g.tiles_n = (C + bn - 1) / bn;
  g.classes = stride * stride;
  for (int k = 0; k < g.classes; ++k) {
    const int py = stride == 2 ? (k < 2 ? 1 : 0) : 0, px = stride == 2 ? (k & 1) ^ 1 : 0;
    const int wk = (W - px + stride - 1) / stride, hk = (H - py + stride - 1) / stride;
    g.pt[k] = p;
    g.pt[k].tx = (wk + (1 << p.lw) - 1) >> p.lw;
    g.pt[k].ty = (hk + (1 << p.lh) - 1) >> p.lh;
    g.first[k] = (int)tiles;
    tiles += count_of(g.pt[k]) * g.tiles_n;
  }
  if (tiles > INT32_MAX) return DS_ERR_ARG;
  g.first[g.classes] = (int)tiles;
  ConvMaps maps;
  DS_TRY(map_pixels(&maps.dz, (const __nv_bfloat16*)dz, N, g.Wo, g.Ho, B, N, (int64_t)g.Wo * N,
                    (int64_t)g.Ho * g.Wo * N, 64, p));
  DS_TRY(map_matrix(&maps.w, w, N, Kp, Kp, 64, 64));
  for (int t = 0; t < 9; ++t) maps.x[t] = maps.dz;  // not read
  maps.z = maps.y = maps.dz;
  return dispatch_bn<kConvDgrad, 64, 0>(bn, maps, g, (cudaStream_t)stream);
}

int64_t ds_conv3x3_wgrad_workspace(int B, int H, int W, int C, int stride, int Kp, int N) {
  using namespace ds;
  if (!conv_ok(B, H, W, C, N, stride, Kp)) return -1;
  ConvArgs g = base_args(B, H, W, C, N, stride, Kp, nullptr);
  int bn;
  if (wgrad_plan(g, bn) != DS_OK) return -1;
  return g.splits > 1 ? (int64_t)g.splits * N * Kp : 0;
}

int ds_conv3x3_wgrad(const void* x, const void* dz, int B, int H, int W, int C, int stride,
                     int Kp, int N, float* gw, float* workspace, uint32_t* err,
                     ds_stream stream) {
  using namespace ds;
  if (!x || !dz || !gw || !err) return DS_ERR_ARG;
  if (!conv_ok(B, H, W, C, N, stride, Kp)) return DS_ERR_ARG;
  if (!aligned16(x) || !aligned16(dz) || !aligned16(gw) || !aligned16(workspace))
    return DS_ERR_ARG;
  ConvArgs g = base_args(B, H, W, C, N, stride, Kp, err);
  // like the GEMM over pixels that this replaces: its rows are 16-byte aligned
  if (((int64_t)B * g.Ho * g.Wo) % 8 != 0) return DS_ERR_ARG;
  int bn;
  DS_TRY(wgrad_plan(g, bn));
  if (g.splits > 1 && !workspace) return DS_ERR_ARG;
  g.d = g.splits > 1 ? workspace : gw;
  const int G = C == 32 ? 32 : 64;
  ConvMaps maps;
  DS_TRY(map_taps(maps, g, (const __nv_bfloat16*)x, G, g.pt[0]));
  DS_TRY(map_pixels(&maps.dz, (const __nv_bfloat16*)dz, N, g.Wo, g.Ho, B, N, (int64_t)g.Wo * N,
                    (int64_t)g.Ho * g.Wo * N, 64, g.pt[0]));
  maps.w = maps.z = maps.y = maps.dz;  // not read
  cudaStream_t s = (cudaStream_t)stream;
  if (G == 32) DS_TRY((dispatch_bn<kConvWgrad, 32, 0>(bn, maps, g, s)));
  else DS_TRY((dispatch_bn<kConvWgrad, 64, 0>(bn, maps, g, s)));
  if (g.splits > 1) {
    const int64_t n4 = (int64_t)N * Kp / 4;
    if (n4 > INT32_MAX) return DS_ERR_ARG;
    conv_reduce_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, s>>>(
        (const float4*)workspace, (float4*)gw, (int)n4, g.splits);
    DS_CUDA(cudaGetLastError());
  }
  return DS_OK;
}

}  // extern "C"
