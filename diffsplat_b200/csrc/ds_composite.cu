// Front-to-back compositing of one tile per CTA and its backward.
//
// Semantics: src/layers/tile_rasterize_layer.cu:192-309 (forward) and
// :356-578 (backward): NDC pixel centres, conic from Cov2D, sigma < 0 skip,
// alpha = min(0.99, o exp(-sigma)), alpha < 1/255 skip, termination after
// including the splat that brings T to <= 1e-4, last_ids = sorted-list index of
// the last contributor, backward by reverse traversal with
// T_before = T / max(1 - alpha, 1e-6).
//
// Layout: tiles are TS x TS pixels (16, the reference's TILE_SIZE; batches may
// use 8 or 32), cut into 8x8-pixel blocks of one warp each.  A lane owns two
// pixels of one column, four rows apart, and works on both with packed FP32
// instructions.  A splat is tested once against each warp's block; the warp then
// walks only its own hits, so misses cost nothing in the inner loop.  One warp
// per block at every tile size and in batches, so each pixel's result and each
// splat's gradient sums are the same whatever the launch.  Gradients are summed
// in a fixed order: they are deterministic run to run.
//
// Batch mode (kBatch): tile indices are batch-wide; tile_inst / geom give each
// tile's instance, image size, tile grid and first pixel.
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "ds_common.cuh"
#include "ds_internal.h"

namespace ds {

namespace {

#ifndef DS_FWD_GROUP
#define DS_FWD_GROUP 2
#endif
#ifndef DS_FWD_MIN_BLOCKS
#define DS_FWD_MIN_BLOCKS 6
#endif
#ifndef DS_BWD_MIN_BLOCKS
#define DS_BWD_MIN_BLOCKS 5
#endif
constexpr int kFwdGroup = DS_FWD_GROUP;  // forward hits whose alphas are computed together
constexpr int kBwdHits = 8;  // hits whose gradients a warp sums at once, four lanes each

// Backward CTA of one tile: a warp per 8x8 block.  kLong: batches of 256 splats for
// grids where the longest lists decide (long_batches).
template <int TS, bool kLong>
struct Lay {
  static constexpr int kWarps = (TS / 8) * (TS / 8);
  static constexpr int kThreads = 32 * kWarps;
  // backward batch: the per-warp partials (kWarps x kBwdBatch x 36 B) stay within
  // 9 KB up to 16-pixel tiles (37 KB with kLong), 18 KB at 32
  static constexpr int kBwdBatch = kWarps <= 1 ? 128 : kWarps <= 4 ? (kLong ? 256 : 64) : 32;
  // 16-pixel tiles: 5 CTAs per SM (96 registers); 4 and 6 measured 0.307 and
  // 0.326 ms against 0.301 on the 1280x720 fit at step 25 (B200)
  static constexpr int kMinBlocksBwd = kWarps != 4 ? 1 : kLong ? 2 : DS_BWD_MIN_BLOCKS;
};

// Where a tile lies: its image size, its tile grid, its index in that grid and
// the first pixel of its image in the pixel arrays.
struct TileGeo {
  int W, H, ntx, local, pix_off;
};

template <bool kBatch>
__device__ __forceinline__ TileGeo tile_geo(int tile, int W, int H, int ntx,
                                            const uint16_t* __restrict__ tile_inst,
                                            const InstGeom* __restrict__ geom) {
  if (!kBatch) return TileGeo{W, H, ntx, tile, 0};
  const InstGeom g = geom[tile_inst[tile]];
  return TileGeo{g.width, g.height, g.ntx, tile - g.tile_off, g.pix_off};
}

// The two pixels of a lane in block `blk` of a tile.
struct Pixels {
  int j;     // column
  int i[2];  // rows
  bool inside[2];
  float px;
  float py[2];
  float wx_lo, wx_hi, wy_lo, wy_hi;  // extremes of the warp's pixel centres (NDC)
};

template <int TS>
__device__ __forceinline__ Pixels pixels(int tile, int ntx, int W, int H, int blk) {
  Pixels m;
  const int lane = threadIdx.x & 31;
  const int trow = tile / ntx, tcol = tile - trow * ntx;
  m.j = tcol * TS + blk % (TS / 8) * 8 + lane % 8;
  m.px = 2.f * (m.j + 0.5f) / W - 1.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    m.i[k] = trow * TS + blk / (TS / 8) * 8 + lane / 8 + 4 * k;
    m.inside[k] = m.i[k] < H && m.j < W;
    m.py[k] = 1.f - 2.f * (m.i[k] + 0.5f) / H;
  }
  float xl = m.px, xh = m.px;
  float yl = fminf(m.py[0], m.py[1]), yh = fmaxf(m.py[0], m.py[1]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    xl = fminf(xl, __shfl_xor_sync(0xffffffffu, xl, o));
    xh = fmaxf(xh, __shfl_xor_sync(0xffffffffu, xh, o));
    yl = fminf(yl, __shfl_xor_sync(0xffffffffu, yl, o));
    yh = fmaxf(yh, __shfl_xor_sync(0xffffffffu, yh, o));
  }
  m.wx_lo = xl;
  m.wx_hi = xh;
  m.wy_lo = yl;
  m.wy_hi = yh;
  return m;
}

// Acceptance-box test of a splat record against one warp's pixel box
// {x_lo, x_hi, y_lo, y_hi}.
__device__ __forceinline__ bool misses(const float4& a, const float4& box) {
  return a.x + a.z < box.x || a.x - a.z > box.y || a.y + a.w < box.z || a.y - a.w > box.w;
}

// Whether any point of a warp's pixel box can reach the splat's sigma cut:
// the minimum over the box of a lower bound of the conic's quadratic form
// (diagonal shrunk by 1e-5 relative, as for the acceptance box) is at the
// centre when the box holds it, else at the clamped stationary point of one
// of the four edges.  The 0.01 of slack in the cut covers the rounding, so a
// pixel that can pass the per-pixel tests is never skipped.
__device__ __forceinline__ bool ellipse_hits(const float4& a, const float4& b, float cut,
                                             const float4& box) {
  if (misses(a, box)) return false;
  if (!(a.z <= 3.0e38f && a.w <= 3.0e38f)) return true;  // unbounded region
  const float x0 = box.x - a.x, x1 = box.y - a.x, y0 = box.z - a.y, y1 = box.w - a.y;
  if (x0 <= 0.f && x1 >= 0.f && y0 <= 0.f && y1 >= 0.f) return true;
  const float k = 1e-5f;
  const float qa = b.x - k * (fabsf(b.x) + fabsf(b.y));
  const float qc = b.z - k * (fabsf(b.z) + fabsf(b.y));
  const float qb = b.y;
  if (!(qa > 0.f && qc > 0.f)) return true;
  const float ia = 1.f / qa, ic = 1.f / qc;
  float m = 3.0e38f;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float X = e ? x1 : x0;
    const float y = fminf(fmaxf(-qb * X * ic, y0), y1);
    m = fminf(m, qa * X * X + 2.f * qb * X * y + qc * y * y);
    const float Y = e ? y1 : y0;
    const float x = fminf(fmaxf(-qb * Y * ia, x0), x1);
    m = fminf(m, qa * x * x + 2.f * qb * x * Y + qc * Y * Y);
  }
  return 0.5f * m <= cut;
}

// One splat of a batch, loaded into registers a batch ahead of its use so the
// gathers overlap the current batch's compositing.
struct Staged {
  float4 a, b, c;
  float idet;  // backward
  bool ok;
};

// A splat as the pixel loops read it: every value twice, so that it loads as a
// packed operand.  The conic's off-diagonal is held doubled: (dx dy) 2b rounds
// like (2 dx dy) b.
struct SplatRec {
  float4 pos;     // x, x, y, y
  float4 ab;      // conic a, a, 2b, 2b
  float4 co;      // conic c, c, opacity, opacity
  float4 rg;      // r, r, g, g
  float4 blue;    // b, b, extra, -: the splat's sorted index as bits; backward: 1 / det of Cov2D
  __device__ __forceinline__ void set(const float4& a, const float4& b, const float4& c,
                                      float extra) {
    pos = make_float4(a.x, a.x, a.y, a.y);
    ab = make_float4(b.x, b.x, 2.f * b.y, 2.f * b.y);
    co = make_float4(b.z, b.z, b.w, b.w);
    rg = make_float4(c.x, c.x, c.y, c.y);
    blue = make_float4(c.z, c.z, extra, 0.f);
  }
  // opacity 0: skipped at every pixel
  __device__ __forceinline__ void set_none() {
    pos = ab = co = rg = blue = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ float2 conic_a() const { return make_float2(ab.x, ab.y); }
  __device__ __forceinline__ float2 conic_2b() const { return make_float2(ab.z, ab.w); }
  __device__ __forceinline__ float2 conic_c() const { return make_float2(co.x, co.y); }
  __device__ __forceinline__ float2 x() const { return make_float2(pos.x, pos.y); }
  __device__ __forceinline__ float2 y() const { return make_float2(pos.z, pos.w); }
  __device__ __forceinline__ float2 red() const { return make_float2(rg.x, rg.y); }
  __device__ __forceinline__ float2 green() const { return make_float2(rg.z, rg.w); }
  __device__ __forceinline__ float opacity() const { return co.z; }
};

// Whether the computed quadratic form of a conic can nowhere be negative (or
// NaN): it rounds to within 4 eps (a dx^2 + 2 |b dx dy| + c dy^2), and is at least
// (1 - |b| / sqrt(a c)) (a dx^2 + c dy^2), so b^2 <= 0.9999 a c leaves a margin of
// two orders of magnitude.  Holds for splats up to about 100 times longer than
// wide; the pixel loops then need no test of sigma's sign.
__device__ __forceinline__ bool definite(const float4& b) {
  return b.x >= 1e-12f && b.z >= 1e-12f && b.x <= 1e18f && b.z <= 1e18f &&
         b.y * b.y <= 0.9999f * b.x * b.z;
}
__device__ __forceinline__ bool finite3(float r, float g, float b) {
  return fabsf(r) <= 3.0e38f && fabsf(g) <= 3.0e38f && fabsf(b) <= 3.0e38f;
}

// Mahalanobis distances dx^2 a + 2 dx dy b + dy^2 c of a splat at a pair of pixels, in
// the reference's rounding (tile_rasterize_layer.cu:321, :341), and opacity
// exp(-dist2 / 2) there, exp as 2^(dist2 (-log2(e) / 2)); dxx = dx dx.
__device__ __forceinline__ float2 pair_dist2(float2 dx, float2 dxx, float2 dy,
                                             const SplatRec& r) {
  return fma2(mul2(dy, dy), r.conic_c(),
              fma2(dxx, r.conic_a(), mul2(mul2(dx, dy), r.conic_2b())));
}
__device__ __forceinline__ float2 pair_opacity(float2 dist2, const SplatRec& r) {
  const float2 p = mul2(both(-0.72134752f), dist2);
  return mul2(make_float2(r.co.z, r.co.w), make_float2(exp2f(p.x), exp2f(p.y)));
}

// Mask bits of a staged splat above the warps': its colour may be infinite, NaN or near
// overflow; it is not plain (the sign bit).
constexpr uint32_t kWild = 0x40000000u, kNotPlain = 0x80000000u;

// A warp's hits of a staged batch, listed in order: the splats l of [from, n)
// whose mask has the warp's bit, with the mask's sign bit.  Padded with `none` to an
// even count; returns the count before padding.  A wild splat may leave an infinite or
// NaN sum in the pixels that it covers, which the hits after it that do not cover them must
// not see: it sets *spoilt, and they too get the sign bit.
__device__ __forceinline__ int list_hits(const uint32_t* mask, int w, int lane, int from, int n,
                                         int none, int* list, uint32_t* spoilt) {
  int count = 0;
  const uint32_t lt = (1u << lane) - 1u;
  for (int k = 0; k < n; k += 32) {
    const int l = k + lane;
    const uint32_t mk = l >= from && l < n ? mask[l] : 0u;
    const bool hit = (mk >> w) & 1u;
    const uint32_t word = __ballot_sync(0xffffffffu, hit);
    const uint32_t wild = __ballot_sync(0xffffffffu, hit && (mk & kWild));
    const bool odd = (mk & kNotPlain) || *spoilt || (wild & lt);
    if (hit) list[count + __popc(word & lt)] = odd ? l | (int)kNotPlain : l;
    if (wild) {
      __syncwarp();
      if (lane == 0) *spoilt = 1u;
      __syncwarp();
    }
    count += __popc(word);
  }
  if (lane == 0) list[count] = none;
  __syncwarp();
  return count;
}

// Bit w set: the splat can reach warp w's pixel block.
template <int NW>
__device__ __forceinline__ uint32_t warp_hits(const float4& a, const float4& b, float cut,
                                              const float4* box) {
  uint32_t mk = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) mk |= ellipse_hits(a, b, cut, box[w]) ? (1u << w) : 0u;
  return mk;
}

// Forward of a tile's 8x8-pixel blocks, one warp each, two pixels per lane (the
// same column, four rows apart) handled by packed instructions.  Bound by
// instruction issue, so the warps share nothing that would make one wait for
// another: each walks its tile's list by itself, 32 splats at a time (one
// test of one splat against the warp's block per lane, the next 32 records in
// flight), compacts the records of its hits into its own shared memory and
// composites them.  Staging a tile's batch once for all its warps saves
// three of four loads of a record (they hit L1 here) but made the warps of a
// tile wait for the one with the most hits in every batch.  Against that, with
// one pixel per lane and 8x4 blocks (B200): 1280x720 fit of 60000 splats at step
// 25 0.231 -> 0.119 ms, at step 400 0.359 -> 0.189; a million splats at
// 1920x1080 0.320 -> 0.235.  6 CTAs per SM and two hits at a time: 8 CTAs took
// 0.122 / 0.199 / 0.268, 5 CTAs and four hits 0.122 / 0.195 / 0.231.
//
// A pixel that is done (T <= 1e-4), outside the image or not reached by the
// splat composites alpha = 0, which changes neither its colour nor its T; only
// colours that are not finite and conics that are nearly singular (whose sigma may
// come out negative) need the guarded variant.  Without the sign test of the others,
// and with the two constants of exp folded into one packed product, the two scenes
// above went from 0.103 to 0.099 and from 0.217 to 0.209 ms.
constexpr int kFwdWarps = 4;

struct FwdShared {
  SplatRec hit[kFwdWarps][32 + kFwdGroup];
  float red[kFwdWarps];
  bool last;
};

template <int TS, bool kLoss, bool kCount, bool kBatch, bool kIds>
__global__ void __launch_bounds__(32 * kFwdWarps, DS_FWD_MIN_BLOCKS)
    composite_fwd_kernel(const float4* __restrict__ ra, const float4* __restrict__ rb,
                         const float4* __restrict__ rc, const uint32_t* __restrict__ sorted_splat,
                         const int2* __restrict__ ranges, const int32_t* __restrict__ order,
                         float* __restrict__ out_rgb, float* __restrict__ out_alpha,
                         int32_t* __restrict__ last_ids, int tiles, int W_, int H_, int ntx_,
                         const uint16_t* __restrict__ tile_inst, const InstGeom* __restrict__ geom,
                         const float* __restrict__ target, float* __restrict__ loss_partials,
                         DevScalars* __restrict__ sc) {
  pdl_wait();
  constexpr int kBlocks = (TS / 8) * (TS / 8);  // warp blocks of a tile
  constexpr int G = kFwdGroup;
  __shared__ FwdShared sm;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int at = blockIdx.x * kFwdWarps + w;
  const int blk = at % kBlocks;
  const bool real = at / kBlocks < tiles;  // 8-pixel tiles: the last CTA may be ragged
  const int slot = real ? at / kBlocks : 0;
  const int tile = order ? order[slot] : slot;
  const TileGeo tg = tile_geo<kBatch>(tile, W_, H_, ntx_, tile_inst, geom);
  const int W = tg.W, H = tg.H;
  const Pixels m = pixels<TS>(tg.local, tg.ntx, W, H, blk);
  const float4 box = make_float4(m.wx_lo, m.wx_hi, m.wy_lo, m.wy_hi);
  const int2 range = real ? ranges[tile] : make_int2(0, 0);
  const int end = range.y;
  const float2 npx = both(-m.px), npy = make_float2(-m.py[0], -m.py[1]);
  // T = 0: never composited
  float2 T = make_float2(m.inside[0] ? 1.f : 0.f, m.inside[1] ? 1.f : 0.f);
  float2 Cr = both(0.f), Cg = both(0.f), Cb = both(0.f);
  int cur0 = 0, cur1 = 0;
  uint32_t n_contrib = 0, n_tested = 0;
  SplatRec* const hit = sm.hit[w];

  auto composite = [&](auto guarded, int n) {
    for (int i = 0; i < n; i += G) {
      float2 al[G];
      bool ok0[G], ok1[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const SplatRec& r = hit[i + g];
        const float2 dx = add2(r.x(), npx);
        const float2 d2 = pair_dist2(dx, mul2(dx, dx), add2(r.y(), npy), r);
        al[g] = pair_opacity(d2, r);
        al[g] = make_float2(fminf(kMaxAlpha, al[g].x), fminf(kMaxAlpha, al[g].y));
        ok0[g] = !(al[g].x < kAlphaThres);
        ok1[g] = !(al[g].y < kAlphaThres);
        if (decltype(guarded)::value) {
          ok0[g] = ok0[g] && !(d2.x < 0.f);
          ok1[g] = ok1[g] && !(d2.y < 0.f);
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const SplatRec& r = hit[i + g];
        const float4 blue = r.blue;
        const int id = __float_as_int(blue.z);
        const bool p0 = ok0[g] && T.x > kTThres, p1 = ok1[g] && T.y > kTThres;
        if (kCount) {
          n_tested += (T.x > kTThres) + (T.y > kTThres);
          n_contrib += p0 + p1;
        }
        const float2 a = make_float2(p0 ? al[g].x : 0.f, p1 ? al[g].y : 0.f);
        if (kIds) {
          cur0 = p0 ? id : cur0;
          cur1 = p1 ? id : cur1;
        }
        const float2 vis = mul2(a, T);
        const float2 r1 = fma2(r.red(), vis, Cr);
        const float2 g1 = fma2(r.green(), vis, Cg);
        const float2 b1 = fma2(make_float2(blue.x, blue.y), vis, Cb);
        if (decltype(guarded)::value) {
          Cr = make_float2(p0 ? r1.x : Cr.x, p1 ? r1.y : Cr.y);
          Cg = make_float2(p0 ? g1.x : Cg.x, p1 ? g1.y : Cg.y);
          Cb = make_float2(p0 ? b1.x : Cb.x, p1 ? b1.y : Cb.y);
        } else {
          Cr = r1, Cg = g1, Cb = b1;
        }
        T = mul2(T, fma2(a, both(-1.f), both(1.f)));
      }
      if (!__any_sync(0xffffffffu, T.x > kTThres || T.y > kTThres)) return;
    }
  };

  // records of the first 32 splats, ids of the next 32
  Staged pf;
  uint32_t next = 0;
  pf.ok = range.x + lane < end;
  if (pf.ok) {
    const uint32_t g = sorted_splat[range.x + lane];
    pf.a = ra[g];
    pf.b = rb[g];
    pf.c = rc[g];
  }
  if (range.x + 32 + lane < end) next = sorted_splat[range.x + 32 + lane];
  for (int b0 = range.x; b0 < end; b0 += 32) {
    const bool mine = pf.ok && ellipse_hits(pf.a, pf.b, pf.c.w, box);
    const uint32_t word = __ballot_sync(0xffffffffu, mine);
    const int n = __popc(word);
    bool odd = false;  // a colour that is not finite, a conic that may go negative
    if (mine) {
      hit[__popc(word & ((1u << lane) - 1u))].set(pf.a, pf.b, pf.c, __int_as_float(b0 + lane));
      odd = !(finite3(pf.c.x, pf.c.y, pf.c.z) && definite(pf.b));
    }
    // the last group is filled with splats of opacity 0
    if (lane < G && n + lane < (n + G - 1) / G * G) hit[n + lane].set_none();
    pf.ok = b0 + 32 + lane < end;
    if (pf.ok) {
      pf.a = ra[next];
      pf.b = rb[next];
      pf.c = rc[next];
    }
    if (b0 + 64 + lane < end) next = sorted_splat[b0 + 64 + lane];
    odd = __any_sync(0xffffffffu, odd);
    __syncwarp();
    if (odd) composite(std::true_type{}, n);
    else composite(std::false_type{}, n);
    if (!__any_sync(0xffffffffu, T.x > kTThres || T.y > kTThres)) break;
    __syncwarp();
  }
  if (kCount) {
    n_contrib = warp_sum_u32(n_contrib);
    n_tested = warp_sum_u32(n_tested);
    if (lane == 0) {
      atomicAdd(&sc->pairs[0], (unsigned long long)n_contrib);
      atomicAdd(&sc->pairs[1], (unsigned long long)n_tested);
    }
  }
  float l = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!m.inside[k] || !real) continue;
    const int pix = tg.pix_off + m.i[k] * W + m.j;
    const float r = k ? Cr.y : Cr.x, g = k ? Cg.y : Cg.x, b = k ? Cb.y : Cb.x;
    out_rgb[pix * 3 + 0] = r;
    out_rgb[pix * 3 + 1] = g;
    out_rgb[pix * 3 + 2] = b;
    if (kIds) {
      out_alpha[pix] = 1.f - (k ? T.y : T.x);
      last_ids[pix] = k ? cur1 : cur0;
    }
    if (kLoss) {
      const float scale = 1.f / (float)(W * H);
      const float dR = r - target[pix * 3 + 0];
      const float dG = g - target[pix * 3 + 1];
      const float dB = b - target[pix * 3 + 2];
      l += (dR * dR + dG * dG + dB * dB) * scale;
    }
  }
  if (kLoss) {
    l = warp_sum(l);
    if (kBlocks < kFwdWarps) {  // 8-pixel tiles: one warp each
      if (lane == 0 && real) loss_partials[tile] = l;
      return;
    }
    // one partial per CTA: kBlocks / kFwdWarps of them per tile
    if (lane == 0) sm.red[w] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < kFwdWarps; ++k) s += sm.red[k];
      loss_partials[tile * (kBlocks / kFwdWarps) + blk / kFwdWarps] = s;
      if (!kBatch) {
        __threadfence();
        sm.last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
      }
    }
    // Batches sum their per-instance losses in batch_loss_kernel instead.
    if (kBatch) return;
    __syncthreads();
    if (sm.last) {
      // The last CTA to finish sums the per-tile partials in tile order.
      __threadfence();
      float s = 0.f;
      for (int k = threadIdx.x; k < (int)gridDim.x; k += 32 * kFwdWarps)
        s += ((volatile float*)loss_partials)[k];
      s = warp_sum(s);
      if (lane == 0) sm.red[w] = s;
      __syncthreads();
      if (threadIdx.x == 0) {
        float tot = 0.f;
        for (int k = 0; k < kFwdWarps; ++k) tot += sm.red[k];
        sc->loss = tot;
        sc->ticket = 0u;
      }
    }
  }
}

// Shared memory of one backward CTA (dynamic: up to 120 KB for 32-pixel tiles).
template <int TS, bool kLong>
struct BwdShared {
  using Lc = Lay<TS, kLong>;
  static constexpr int B = Lc::kBwdBatch, NW = Lc::kWarps;
  // Row of a hit's per-pixel values: 4 floats past the pixels of a warp, so
  // that the eight lanes of a 16-byte shared-memory phase (two hits, four
  // lanes each, 8 floats apart) fall on distinct banks.
  static constexpr int kPitch = 64 + 4;
  SplatRec splat[B + 1];       // the last one reaches nothing
  float4 box[NW];
  float4 gr[NW][16], gg[NW][16], gb[NW][16];  // per pixel of a warp: dL/dpixel
  float2 nx[NW][4];    // -x (NDC) of a warp's columns 2q and 2q + 1
  float2 ny[NW][4];    // -y of its rows r and r + 4
  float4 s[NW][kBwdHits * kPitch / 4];    // per (hit, pixel): opacity exp() dL/dalpha
  float4 fac[NW][kBwdHits * kPitch / 4];  // per (hit, pixel): alpha T
  float part[NW][B * 9];       // per-warp gradient of each batch splat
  uint32_t rec[B];             // record index of each batch splat
  uint32_t mask[B];            // warps whose block the splat can reach, kWild, kNotPlain
  uint32_t got[NW][B / 32];    // batch splats with a partial from the warp
  int2 list[NW][B / 2 + 1];    // the warp's hits of the batch
  int32_t final_id[NW];
  uint32_t spoilt[NW];         // a wild splat was among the warp's hits
};

// Slot of lane l's pixel pair (column l % 8, rows l / 8 and l / 8 + 4) in a hit's row
// of per-pixel values, in floats.  Row r's columns 2q and 2q + 1 are the 16-byte word
// at_word(r, q): for a fixed r, the four q of two hits fall on distinct banks.
__device__ __forceinline__ int at_word(int r, int q) { return (r >> 1) * 8 + q * 2 + (r & 1); }
__device__ __forceinline__ int pixel_slot(int lane) {
  return 4 * at_word(lane >> 3, (lane & 7) >> 1) + 2 * (lane & 1);
}

// The gradients of up to kBwdHits hits of a warp from their per-pixel values:
// four lanes per hit, each over two columns of the warp's block, the upper and the
// lower four rows in the halves of an instruction.  With u = a dx + b dy and
// w = b dx + c dy,
//   d dist2 / d(ndc x, ndc y) = (2u, 2w)
//   d dist2 / d(cov xx, xy, yy) = -u^2, -2uw, -w^2
// and s = -2 dL/d(dist2).  u and w are formed at every pixel, from its own dx and dy: sums of
// s u^2, s u w and s w^2 rebuilt from moments of s about a row cancel for splats thinner than
// a pixel, to a relative error of 3e-6 at sigma = 0.1 pixels and 1e-3 at 0.003, where this
// form stays at 1e-7, and saved little (1280x720 fit, step 4, 0.218 -> 0.214 ms; a million
// splats at 1920x1080 0.491 -> 0.484, B200).  kSafe also leaves out what s = 0 or fac = 0
// multiplies, as it may be infinite or NaN.
// The sum for cov xy takes u w as b dist2 + dx dy / det, the form that this gradient has always
// had: for long tilted splats either cancels, to as much as 1e-4 of a sum, and only the
// same products give the same values (u w would save 0.03 of 0.79 ms of that fit's step).
template <bool kSafe, class Sh>
__device__ __forceinline__ void reduce_hits(Sh& sm, int w, int lane, int count,
                                            int slot) {
  const int h = lane >> 2, q = lane & 3;
  const SplatRec& hit = sm.splat[slot];
  const float2 ca = hit.conic_a(), cb = mul2(hit.conic_2b(), both(0.5f)), cc = hit.conic_c();
  const float2 idet = both(hit.blue.z);
  const float2 dxs[2] = {add2(hit.x(), both(sm.nx[w][q].x)), add2(hit.x(), both(sm.nx[w][q].y))};
  float2 v[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) v[k] = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int at = at_word(r, q);
    const float4 f4 = sm.fac[w][h * (Sh::kPitch / 4) + at];
    const float4 r4 = sm.gr[w][at], g4 = sm.gg[w][at], b4 = sm.gb[w][at];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 f = e ? make_float2(f4.z, f4.w) : make_float2(f4.x, f4.y);
      float2 gr = e ? make_float2(r4.z, r4.w) : make_float2(r4.x, r4.y);
      float2 gg = e ? make_float2(g4.z, g4.w) : make_float2(g4.x, g4.y);
      float2 gb = e ? make_float2(b4.z, b4.w) : make_float2(b4.x, b4.y);
      if (kSafe) {
        gr.x = f.x != 0.f ? gr.x : 0.f, gr.y = f.y != 0.f ? gr.y : 0.f;
        gg.x = f.x != 0.f ? gg.x : 0.f, gg.y = f.y != 0.f ? gg.y : 0.f;
        gb.x = f.x != 0.f ? gb.x : 0.f, gb.y = f.y != 0.f ? gb.y : 0.f;
      }
      v[0] = fma2(f, gr, v[0]);
      v[1] = fma2(f, gg, v[1]);
      v[2] = fma2(f, gb, v[2]);
    }
    const float4 s4 = sm.s[w][h * (Sh::kPitch / 4) + at];
    const float2 dy = add2(hit.y(), sm.ny[w][r]);
    const float2 dyb = mul2(dy, cb), dyc = mul2(dy, cc), dyy = mul2(dy, dy);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 z = e ? make_float2(s4.z, s4.w) : make_float2(s4.x, s4.y);
      const float2 dx = dxs[e], xy = mul2(dx, dy);
      float2 u = fma2(dx, ca, dyb), t = fma2(dx, cb, dyc);
      const float2 dist2 = fma2(dyy, cc, fma2(mul2(dx, dx), ca, mul2(xy, hit.conic_2b())));
      float2 x = fma2(cb, dist2, mul2(xy, idet));
      if (kSafe) {
        u.x = z.x != 0.f ? u.x : 0.f, u.y = z.y != 0.f ? u.y : 0.f;
        t.x = z.x != 0.f ? t.x : 0.f, t.y = z.y != 0.f ? t.y : 0.f;
        x.x = z.x != 0.f ? x.x : 0.f, x.y = z.y != 0.f ? x.y : 0.f;
      }
      const float2 su = mul2(z, u), st = mul2(z, t);
      v[3] = add2(v[3], su);
      v[4] = add2(v[4], st);
      v[5] = fma2(su, u, v[5]);
      v[6] = fma2(z, x, v[6]);
      v[7] = fma2(st, t, v[7]);
      v[8] = add2(v[8], z);
    }
  }
  float r[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) r[k] = v[k].x + v[k].y;
  r[3] = -r[3];
  r[4] = -r[4];
  r[5] *= 0.5f;
  r[7] *= 0.5f;
  // sum over the hit's four lanes: lane q ends with values 4 (q & 1) + (q & 2) + {0, 1}
  const bool b0 = q & 1, b1 = q & 2;
  float t4[4], t2[2];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    t4[k] = (b0 ? r[k + 4] : r[k]) + __shfl_xor_sync(0xffffffffu, b0 ? r[k] : r[k + 4], 1);
#pragma unroll
  for (int k = 0; k < 2; ++k)
    t2[k] = (b1 ? t4[k + 2] : t4[k]) + __shfl_xor_sync(0xffffffffu, b1 ? t4[k] : t4[k + 2], 2);
  float o = r[8] + __shfl_xor_sync(0xffffffffu, r[8], 1);
  o += __shfl_xor_sync(0xffffffffu, o, 2);
  if (h < count) {
    float* dst = &sm.part[w][slot * 9];
    const int k = (b0 ? 4 : 0) + (b1 ? 2 : 0);
    dst[k] = t2[0];
    dst[k + 1] = t2[1];
    if (q == 0) dst[8] = o == 0.f ? 0.f : o / hit.opacity();  // s carries the opacity
  }
}

// Backward of one tile per CTA.  Bound by instruction issue.  Each (hit, pixel)
// yields two numbers, s (for position, covariance and opacity) and fac (for the
// colour); the nine gradients of a hit are sums of products of these with
// values that depend on the pixel or on the splat alone.  So the pixel loop
// (lane = pixel) only stores s and fac to shared memory, and for every
// kBwdHits hits (or one fewer, so that the loop has a single place to do it) the
// lanes regroup, four to a hit, and form the sums over the pixels (reduce_hits),
// which cost about 22 issue slots a hit where the nine-value butterfly over the
// warp took about 60 (counted before the sum for cov xy had its own products).  Against the butterfly (B200): 1280x720 fit of 60000 splats at
// step 25 0.366 -> 0.301 ms, at step 400 0.828 -> 0.504; a million splats at
// 1920x1080 0.656 -> 0.600.
//
// The pixel loop was next: of some 70 issue slots a hit, half went to tests and
// selects on the ALU pipe, which issues at half rate.  Splats that cannot reach alpha
// 0.99 and whose conic is not nearly singular ("plain", nearly all) need a test of alpha
// and one of the pixel's last contributor, and no other select.
// Step 4 of the 1280x720 fit 0.258 -> 0.218 ms; the million splats 0.525 -> 0.491, with
// batches staged ahead (there the warps of a tile wait for one another at every batch).
// With the sum for cov xy as it is now: 0.243 and 0.540.
template <int TS, bool kFusedLoss, bool kExact, bool kBatch, bool kLong>
__global__ void __launch_bounds__(Lay<TS, kLong>::kThreads, Lay<TS, kLong>::kMinBlocksBwd)
    composite_bwd_kernel(const float4* __restrict__ ra, const float4* __restrict__ rb,
                         const float4* __restrict__ rc, const float* __restrict__ ridet,
                         const uint32_t* __restrict__ sorted_splat,
                         const uint32_t* __restrict__ seg_start,
                         const ushort4* __restrict__ rect, const int2* __restrict__ ranges,
                         const int32_t* __restrict__ order, const float* __restrict__ alphas,
                         const int32_t* __restrict__ last_ids,
                         const float* __restrict__ grad_or_image, const float* __restrict__ target,
                         float* __restrict__ isect_grad, int W_, int H_, int ntx_,
                         const uint16_t* __restrict__ tile_inst,
                         const InstGeom* __restrict__ geom,
                         const uint32_t* __restrict__ depth_keys,
                         unsigned long long* __restrict__ tile_bound) {
  pdl_wait();
  using Lc = Lay<TS, kLong>;
  using Sh = BwdShared<TS, kLong>;
  constexpr int NT = Lc::kThreads;
  constexpr int NW = Lc::kWarps;
  constexpr int B = Lc::kBwdBatch;
  extern __shared__ __align__(16) unsigned char bwd_smem[];
  Sh& sm = *reinterpret_cast<Sh*>(bwd_smem);
  const int tile = order ? order[blockIdx.x] : (int)blockIdx.x;
  const int2 range = ranges[tile];
  const int start = range.x;
  if (range.y <= start) {
    if (threadIdx.x == 0) tile_bound[tile] = 0ull;
    return;
  }
  const TileGeo tg = tile_geo<kBatch>(tile, W_, H_, ntx_, tile_inst, geom);
  const int W = tg.W, H = tg.H;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const Pixels m = pixels<TS>(tg.local, tg.ntx, W, H, w);
  // the tile's row and column in its grid, for the record indices
  const int trow = tg.local / tg.ntx, tcol = tg.local - trow * tg.ntx;
  if (lane == 0) sm.box[w] = make_float4(m.wx_lo, m.wx_hi, m.wy_lo, m.wy_hi);
  // acc: over the splats behind (already visited), weight x (colour . dL/dpixel)
  float2 T, gr, gg, gb, acc = both(0.f);
  const float2 npx = both(-m.px), npy = make_float2(-m.py[0], -m.py[1]);
  int32_t fin[2];
  int32_t my_final = -1;
  bool finite = true;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int pix = tg.pix_off + min(m.i[k] * W + m.j, W * H - 1);
    const float t = 1.f - alphas[pix];
    fin[k] = m.inside[k] ? last_ids[pix] : -1;
    my_final = max(my_final, fin[k]);
    float r = 0.f, g = 0.f, b = 0.f;
    if (m.inside[k]) {
      if (kFusedLoss) {
        const float scale = 2.f / (float)(W * H);
        r = scale * (grad_or_image[pix * 3 + 0] - target[pix * 3 + 0]);
        g = scale * (grad_or_image[pix * 3 + 1] - target[pix * 3 + 1]);
        b = scale * (grad_or_image[pix * 3 + 2] - target[pix * 3 + 2]);
      } else {
        r = grad_or_image[pix * 3 + 0];
        g = grad_or_image[pix * 3 + 1];
        b = grad_or_image[pix * 3 + 2];
      }
      finite = finite && fabsf(r) <= 1e15f && fabsf(g) <= 1e15f && fabsf(b) <= 1e15f;
    }
    (k ? T.y : T.x) = t;
    (k ? gr.y : gr.x) = r;
    (k ? gg.y : gg.x) = g;
    (k ? gb.y : gb.x) = b;
  }
  reinterpret_cast<float2*>(sm.gr[w])[pixel_slot(lane) / 2] = gr;
  reinterpret_cast<float2*>(sm.gg[w])[pixel_slot(lane) / 2] = gg;
  reinterpret_cast<float2*>(sm.gb[w])[pixel_slot(lane) / 2] = gb;
  const bool safe_pixels = __all_sync(0xffffffffu, finite);
  if (lane < 8) reinterpret_cast<float*>(sm.nx[w])[lane] = -m.px;
  if ((lane & 7) == 0) sm.ny[w][lane >> 3] = make_float2(-m.py[0], -m.py[1]);
  const int32_t warp_final = warp_max(my_final);
  // Pairs after the tile's last contributing splat reach no pixel: the list
  // ends there for the backward, and no record is written for them (their
  // consumers skip them by tile_bound).
  if (lane == 0) sm.final_id[w] = warp_final, sm.spoilt[w] = 0u;
  __syncthreads();
  int32_t tile_final = sm.final_id[0];
#pragma unroll
  for (int k = 1; k < NW; ++k) tile_final = max(tile_final, sm.final_id[k]);
  const int end = min(range.y, tile_final + 1);
  if (threadIdx.x == 0) {
    unsigned long long bound = 0ull;
    if (end > start) {
      const uint32_t last = sorted_splat[end - 1];
      bound = (((unsigned long long)depth_keys[last] << 32) | last) + 1ull;
    }
    tile_bound[tile] = bound;
  }
  if (end <= start) return;
  const int nb = (end - start + B - 1) / B;
  // Threads per staged splat: with twice as many threads as batch slots, two
  // threads share a splat's warp-block tests and its cross-warp sum.
  constexpr int kSplit = NT >= 2 * B ? 2 : 1;
  constexpr int R = (B * kSplit + NT - 1) / NT;  // splats each thread stages
  Staged pf[R];
  uint32_t pf_rec[R];
  // batch bi holds sorted indices end - 1 - B bi down to end - B (bi + 1)
  auto prefetch = [&](int bi) {
    const int batch_end = end - 1 - B * bi;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int l = (threadIdx.x + r * NT) / kSplit, li = batch_end - l;
      pf[r].ok = l < B && li >= start;
      if (pf[r].ok) {
        const uint32_t g = sorted_splat[li];
        pf[r].a = ra[g];
        pf[r].b = rb[g];
        pf[r].c = rc[g];
        pf[r].idet = ridet[g];
        if ((threadIdx.x + r * NT) % kSplit == 0) {
          // the pair's emission index: the splat's first one plus the tile's
          // row-major index in the splat's tile rectangle
          const ushort4 t = rect[g];
          pf_rec[r] = seg_start[g] + (uint32_t)(trow - t.z) * (uint32_t)(t.y - t.x + 1) +
                      (uint32_t)(tcol - t.x);
        }
      }
    }
  };
  if (threadIdx.x == 0) sm.splat[B].set_none();
  float* const my_s = reinterpret_cast<float*>(sm.s[w]) + pixel_slot(lane);
  float* const my_f = reinterpret_cast<float*>(sm.fac[w]) + pixel_slot(lane);
  prefetch(0);
  for (int bi = 0; bi < nb; ++bi) {
    const int batch_end = end - 1 - B * bi;  // farthest splat of the batch
    const int bs = min(B, batch_end + 1 - start);
    // Stage the batch back to front: slot l holds sorted index batch_end - l.  Every warp
    // is past the previous batch's hits; its sums may still be read, but they lie
    // elsewhere, and a slot's record index is this warp's own.
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int slot = threadIdx.x + r * NT, l = slot / kSplit, h = slot % kSplit;
      uint32_t mk = 0u;
      if (l < B && pf[r].ok) {
        const float4 a = pf[r].a, b = pf[r].b, c = pf[r].c;
        if (kSplit == 1) {
          mk = warp_hits<NW>(a, b, c.w, sm.box);
        } else {
          // this thread tests half of the warp blocks
#pragma unroll
          for (int k = 0; k < NW / 2; ++k) {
            const int wb = h * (NW / 2) + k;
            mk |= ellipse_hits(a, b, c.w, sm.box[wb]) ? (1u << wb) : 0u;
          }
        }
        if (h == 0) {
          sm.splat[l].set(a, b, c, pf[r].idet);
          sm.rec[l] = pf_rec[r];
          // plain: cannot reach alpha 0.99, and nothing about it overflows
          const bool wild = !(fabsf(c.x) <= 1e15f && fabsf(c.y) <= 1e15f && fabsf(c.z) <= 1e15f);
          if (wild) mk |= kWild;
          if (wild || !(definite(b) && b.w <= kMaxAlpha)) mk |= kNotPlain;
        }
      }
      if (kSplit == 2) mk |= __shfl_xor_sync(0xffffffffu, mk, 1);  // pairs are adjacent lanes
      if (l < B && h == 0) sm.mask[l] = mk;
    }
    if (bi + 1 < nb) prefetch(bi + 1);
    __syncthreads();
    const int t_start = max(0, batch_end - warp_final);
    int* const list = reinterpret_cast<int*>(sm.list[w]);
    const int hits = list_hits(sm.mask, w, lane, t_start, bs, B, list, &sm.spoilt[w]);
    if (lane < B / 32) sm.got[w][lane] = 0u;
    __syncwarp();
    int count = 0, slot = 0;  // hits stored; the slot of this lane's hit (lane / 4)
    auto flush = [&] {
      __syncwarp();
      bool tame = true;
      if ((lane >> 2) < count) {
        const SplatRec& r = sm.splat[slot];
        tame = fabsf(r.conic_a().x) <= 1e15f && fabsf(r.conic_2b().x) <= 1e15f &&
               fabsf(r.conic_c().x) <= 1e15f;
        if ((lane & 3) == 0) atomicOr(&sm.got[w][slot >> 5], 1u << (slot & 31));
      }
      if (safe_pixels && __all_sync(0xffffffffu, tame))
        reduce_hits<false>(sm, w, lane, count, slot);
      else
        reduce_hits<true>(sm, w, lane, count, slot);
      count = 0;
      __syncwarp();
    };
    auto store = [&](float2 s, float2 fac, int t) {
      *reinterpret_cast<float2*>(my_s + count * Sh::kPitch) = s;
      *reinterpret_cast<float2*>(my_f + count * Sh::kPitch) = fac;
      if ((lane >> 2) == count) slot = t;
      ++count;
    };
    // lit: the splat's colour . dL/dpixel.  Reference recurrence
    // (tile_rasterize_layer.cu:518-521) weighs the colour behind (absolute weights
    // c_j alpha_j T_j) by T_before; the exact derivative divides it by T_after
    // instead.  The three colour channels enter only through their dot product with
    // dL/dpixel.
    auto lit_of = [&](const SplatRec& r) {
      const float2 blue = *reinterpret_cast<const float2*>(&r.blue);
      return fma2(blue, gb, fma2(r.red(), gr, mul2(r.green(), gg)));
    };
    auto weigh = [&](float2 lit) {
      const float2 nia = kExact ? make_float2(-1.f / T.x, -1.f / T.y) : both(-1.f);
      return fma2(acc, nia, lit);
    };
    // The hits two at a time: conic, exp and alpha of both first (independent of
    // T), then the recurrence back to front.
    for (int i = 0; i < hits; i += 2) {
      const int2 pair = sm.list[w][i >> 1];
      float2 oe[2], al[2];
      bool any[2];
      if (safe_pixels && (pair.x | pair.y) >= 0) {
        // Plain splats: alpha = opacity exp() where it passes, 0 elsewhere, which
        // leaves T and acc as they are, and s at 0 while acc is finite.
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int t = g ? pair.y : pair.x, id = batch_end - t;
          const SplatRec& r = sm.splat[t];
          const float2 dx = add2(r.x(), npx);
          oe[g] = pair_opacity(pair_dist2(dx, mul2(dx, dx), add2(r.y(), npy), r), r);
          const bool o0 = oe[g].x >= kAlphaThres && id <= fin[0];
          const bool o1 = oe[g].y >= kAlphaThres && id <= fin[1];
          al[g] = make_float2(o0 ? oe[g].x : 0.f, o1 ? oe[g].y : 0.f);
          any[g] = o0 || o1;
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (!__any_sync(0xffffffffu, any[g])) continue;
          const int t = g ? pair.y : pair.x;
          const float2 om = fma2(al[g], both(-1.f), both(1.f));  // >= 0.01
          const float2 lit = lit_of(sm.splat[t]);
          const float2 in = weigh(lit);
          T = mul2(T, make_float2(rcp(om.x), rcp(om.y)));
          const float2 fac = mul2(al[g], T);
          acc = fma2(lit, fac, acc);
          store(mul2(fac, in), fac, t);
        }
      } else {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int t = (g ? pair.y : pair.x) & 0x7fffffff, id = batch_end - t;
          const SplatRec& r = sm.splat[t];
          const float2 dx = add2(r.x(), npx);
          const float2 d2 = pair_dist2(dx, mul2(dx, dx), add2(r.y(), npy), r);
          oe[g] = pair_opacity(d2, r);
          const float a0 = fminf(kMaxAlpha, oe[g].x), a1 = fminf(kMaxAlpha, oe[g].y);
          const bool o0 = !(d2.x < 0.f) && id <= fin[0] && !(a0 < kAlphaThres);
          const bool o1 = !(d2.y < 0.f) && id <= fin[1] && !(a1 < kAlphaThres);
          // alpha 0: the splat is skipped at that pixel
          al[g] = make_float2(o0 ? a0 : 0.f, o1 ? a1 : 0.f);
          any[g] = o0 || o1;
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (!__any_sync(0xffffffffu, any[g])) continue;
          const int t = (g ? pair.y : pair.x) & 0x7fffffff;
          const bool o0 = al[g].x > 0.f, o1 = al[g].y > 0.f;
          const float2 om = fma2(al[g], both(-1.f), both(1.f));  // >= 0.01
          const float2 Tb = mul2(T, make_float2(rcp(om.x), rcp(om.y)));
          const float2 fac = mul2(al[g], Tb);
          const float2 lit = lit_of(sm.splat[t]);
          const float2 s2 = mul2(fac, weigh(lit));  // (fac as for a plain splat where it counts)
          const float2 next = fma2(lit, fac, acc);
          float2 s;
          s.x = o0 && oe[g].x <= kMaxAlpha ? s2.x : 0.f;
          s.y = o1 && oe[g].y <= kMaxAlpha ? s2.y : 0.f;
          acc = make_float2(o0 ? next.x : acc.x, o1 ? next.y : acc.y);
          T = make_float2(o0 ? Tb.x : T.x, o1 ? Tb.y : T.y);
          store(s, fac, t);
        }
      }
      if (count >= kBwdHits - 1 || (i + 2 >= hits && count > 0)) flush();
    }
    __syncthreads();
    for (int slot2 = threadIdx.x; slot2 < bs * kSplit; slot2 += NT) {
      const int l = slot2 / kSplit, h = slot2 % kSplit;
      float* dst = isect_grad + (size_t)sm.rec[l] * 9;
      float v[(9 + kSplit - 1) / kSplit];
#pragma unroll
      for (int q = 0; q < (9 + kSplit - 1) / kSplit; ++q) v[q] = 0.f;
#pragma unroll
      for (int ww = 0; ww < NW; ++ww) {
        if (!(sm.got[ww][l >> 5] >> (l & 31) & 1u)) continue;
#pragma unroll
        for (int q = h; q < 9; q += kSplit) v[q / kSplit] += sm.part[ww][l * 9 + q];
      }
#pragma unroll
      for (int q = h; q < 9; q += kSplit) dst[q] = v[q / kSplit];
    }
  }
}

const int32_t* schedule(const RasterBuffers& rb) {
  return rb.schedule == DS_SCHEDULE_LONGEST_FIRST ? rb.tile_order : nullptr;
}

template <int TS, bool kBatch>
void launch_fwd(RasterBuffers& rb, float* out_rgb, const float* target, bool count,
                cudaStream_t s) {
  constexpr int kBlocks = (TS / 8) * (TS / 8);
  const int32_t* order = schedule(rb);
  const dim3 grid((unsigned)(((int64_t)rb.tiles * kBlocks + kFwdWarps - 1) / kFwdWarps));
#define DS_FWD(L, C, I)                                                                      \
  launch_pdl(composite_fwd_kernel<TS, L, C, kBatch, I>, grid, dim3(32 * kFwdWarps), 0, s,    \
             rb.rec_a, rb.rec_b, rb.rec_c, rb.sorted_splat, rb.ranges, order, out_rgb,        \
             rb.alphas, rb.last_ids, rb.tiles, rb.width, rb.height, rb.ntx, rb.tile_inst,     \
             rb.geom, L ? target : nullptr, L ? rb.loss_partials : nullptr, rb.scalars)
  if (count) DS_FWD(false, true, true);
  else if (target) DS_FWD(true, false, true);
  else if (kBatch || !rb.image_only) DS_FWD(false, false, true);
  else DS_FWD(false, false, false);
#undef DS_FWD
}

template <int TS, bool kBatch, bool kLong = false>
void launch_bwd(RasterBuffers& rb, const float* image, const float* grad_rgb, const float* target,
                cudaStream_t s) {
  constexpr int NT = Lay<TS, kLong>::kThreads;
  const float* g = grad_rgb ? grad_rgb : image;
  const float* t = grad_rgb ? nullptr : target;
  const bool exact = rb.grad_mode == DS_GRAD_EXACT;
  const int32_t* order = schedule(rb);
  constexpr int smem = (int)sizeof(BwdShared<TS, kLong>);
#define DS_BWD(F, E)                                                                         \
  do {                                                                                       \
    static std::atomic<uint64_t> set{0};                                                     \
    allow_smem(composite_bwd_kernel<TS, F, E, kBatch, kLong>, smem, set);                     \
    launch_pdl(composite_bwd_kernel<TS, F, E, kBatch, kLong>, dim3(rb.tiles), dim3(NT), smem, \
               s,                                                                            \
               rb.rec_a, rb.rec_b, rb.rec_c, rb.rec_idet, rb.sorted_splat, rb.seg_start,     \
               rb.rect, rb.ranges, order, rb.alphas, rb.last_ids, g, t, rb.isect_grad, rb.width,      \
               rb.height, rb.ntx, rb.tile_inst, rb.geom, rb.depth_keys, rb.tile_bound);      \
  } while (0)
  if (grad_rgb) {
    if (exact) DS_BWD(false, true);
    else DS_BWD(false, false);
  } else {
    if (exact) DS_BWD(true, true);
    else DS_BWD(true, false);
  }
#undef DS_BWD
}

// Whether the backward takes its lists in batches of 256 splats, 2 CTAs per SM, not of 64,
// 5 CTAs.  The warps of a tile meet twice a batch, which counts where few warps
// share an SM: in grids whose tiles are all on the chip at once, and where most splats
// lie in few tiles, as with more than 65536 of them (surfaces).  Elsewhere the other CTAs
// are worth more.  Kernel in ms, 64 / 256 (B200): random splats, 60000 at 256x256 (256 tiles)
// 0.073 / 0.066, 433x341 (616) 0.070 / 0.094, 1280x720 (3600) 0.221 / 0.333; surfaces, 94000 at
// 184x144 0.501 / 0.435, 433x341 0.549 / 0.463, 1280x720 0.201 / 0.164, 500000 at 1280x720 0.569 /
// 0.490.  128 splats and 4 CTAs lie between (94000 at 433x341 0.502).
bool long_batches(const RasterBuffers& rb) {
  return rb.tiles <= (rb.max_splats > kSmallSort ? 4096 : 2 * 148);
}

// Single instance: 16-pixel tiles.  Batch: tiles of 8, 16 or 32 pixels.
void forward(RasterBuffers& rb, float* out_rgb, const float* target, bool count,
             cudaStream_t s) {
  if (!rb.geom) launch_fwd<16, false>(rb, out_rgb, target, count, s);
  else if (rb.tile_size == 8) launch_fwd<8, true>(rb, out_rgb, target, count, s);
  else if (rb.tile_size == 32) launch_fwd<32, true>(rb, out_rgb, target, count, s);
  else launch_fwd<16, true>(rb, out_rgb, target, count, s);
}

}  // namespace

bool composite_longest_first() {
  static const bool on = [] {
    const char* e = getenv("DS_TILE_SCHEDULE");
    return !(e && strcmp(e, "raster") == 0);
  }();
  return on;
}

int raster_composite_forward(RasterBuffers& rb, float* out_rgb, const float* target,
                             cudaStream_t s) {
  forward(rb, out_rgb, target, false, s);
  return cuda_status(cudaGetLastError());
}

int raster_composite_count(RasterBuffers& rb, float* out_rgb, cudaStream_t s) {
  DS_CUDA(cudaMemsetAsync(rb.scalars->pairs, 0, sizeof(rb.scalars->pairs), s));
  forward(rb, out_rgb, nullptr, true, s);
  return cuda_status(cudaGetLastError());
}

int raster_composite_backward(RasterBuffers& rb, const float* image, const float* grad_rgb,
                              const float* target, cudaStream_t s) {
  if (!rb.geom && long_batches(rb))
    launch_bwd<16, false, true>(rb, image, grad_rgb, target, s);
  else if (!rb.geom) launch_bwd<16, false>(rb, image, grad_rgb, target, s);
  else if (rb.tile_size == 8) launch_bwd<8, true>(rb, image, grad_rgb, target, s);
  else if (rb.tile_size == 32) launch_bwd<32, true>(rb, image, grad_rgb, target, s);
  else launch_bwd<16, true>(rb, image, grad_rgb, target, s);
  return cuda_status(cudaGetLastError());
}

}  // namespace ds
