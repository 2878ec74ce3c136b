// Tile lists from the depth-ordered tile rectangles: for every tile the ids of the
// splats whose rectangle covers it, in depth order with equal depths by id -- the
// reference's sorted (tile << 32 | depth) order (tile_rasterize_layer.cu:52-162).
//
// The depth-ordered splats are cut into chunks, the tile grid into bins of 8 x 8 tiles:
//   tile_bins_kernel<false>  per chunk, splats per tile -> hist[chunk][tile]
//   tile_offsets_kernel      per tile, exclusive prefix of hist over the chunks (in
//                            place) and the total; the last CTA to finish scans the
//                            totals into the tile ranges and orders the tiles for the
//                            composite (longest first)
//   tile_bins_kernel<true>   per chunk, the ids to range start + prefix + rank
// A warp takes a bin of a chunk: it picks the splats that reach the bin (one
// comparison of packed bytes each), gives 32 of them a lane each and a 64-bit mask of
// the bin's tiles that they cover, and transposes the masks (five shuffles per half),
// after which lane t holds the splats of tiles t and 32 + t as bits in depth order.
// Counting is a popcount, a splat's rank in a tile the bits below it.  No (tile,
// splat) pair exists before it is written to its place.
//
// Batches: the splats are ordered by instance first, a chunk holds splats of one
// instance, and only that instance's bins are walked.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ds_common.cuh"
#include "ds_internal.h"
#include "ds_warp_gather.cuh"

namespace ds {

namespace {

constexpr int kBinThreads = 256;
constexpr int kBinWarps = kBinThreads / 32;
constexpr int kBin = 8;             // tiles per bin edge
constexpr int kBinMaxAxis = 127;    // bins per axis that the packed comparison holds
constexpr int kChunkMin = 64, kChunkMax = 1024;  // splats per chunk
constexpr int kBinSplats = 65536;   // most splats of a single instance
constexpr uint32_t kFew = 4;        // splats of 32 that a lane appends to its tile by itself

struct BinArgs {
  const ushort4* rect;     // depth order; x0 > x1 for a splat in no tile
  const uint32_t* perm;    // splat ids in depth order
  int n, per;              // splats, splats per chunk
  int ntx, nty;
  const int4* chunks;      // batch: {first, end, instance, first of hist}
  const InstGeom* geom;
  uint32_t* hist;
  const int2* ranges;
  uint32_t* out;
  const DevScalars* sc;
};

// 32 x 32 bits: lane t's bit i becomes lane i's bit t.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu
                     : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? (x & ~m) | ((y & ~m) >> j) : (x & m) | ((y & m) << j);
  }
  return x;
}

// The bin's tiles that rectangle r covers: bit 8 y + x of {lo, hi} for tile (X0 + x, Y0 +
// y).  limit: only the first `limit` tiles of the rectangle, row by row (the pairs
// that still fit the buffers).
__device__ __forceinline__ void tile_mask(const ushort4& r, int X0, int Y0, uint32_t limit,
                                          uint32_t& lo, uint32_t& hi) {
  const int x0 = max((int)r.x - X0, 0), x1 = min((int)r.y - X0, kBin - 1);
  const int y0 = max((int)r.z - Y0, 0), y1 = min((int)r.w - Y0, kBin - 1);
  const uint32_t cols = (0xffu >> (kBin - 1 - x1)) & (0xffu << x0);
  const unsigned long long rows = (~0ull >> (8 * (kBin - 1 - y1))) & (~0ull << (8 * y0));
  lo = (cols * 0x01010101u) & (uint32_t)rows;
  hi = (cols * 0x01010101u) & (uint32_t)(rows >> 32);
  if (limit != 0xffffffffu) {
    const uint32_t w = (uint32_t)(r.y - r.x + 1);
    for (int y = y0; y <= y1; ++y)
      for (int x = x0; x <= x1; ++x) {
        const uint32_t k = (uint32_t)(Y0 + y - r.z) * w + (uint32_t)(X0 + x - r.x);
        if (k >= limit) (y < 4 ? lo : hi) &= ~(1u << ((y & 3) * 8 + x));
      }
  }
}

// Bins that a rectangle reaches as bytes {x0, y0, 127 - x1, 127 - y1}: it reaches bin
// (x, y) when none is above {x, y, 127 - x, 127 - y}, i.e. when subtracting them from
// the latter with the high bits set borrows from none of these.
__device__ __forceinline__ uint32_t bin_bytes(int x0, int y0, int x1, int y1) {
  return (uint32_t)x0 | (uint32_t)y0 << 8 | (uint32_t)(kBinMaxAxis - x1) << 16 |
         (uint32_t)(kBinMaxAxis - y1) << 24;
}
__device__ __forceinline__ bool reaches(uint32_t splat, uint32_t bin_high) {
  return ((bin_high - splat) & 0x80808080u) == 0x80808080u;
}

// Shared memory of a chunk of `per` splats; the packed bins are padded to whole steps.
constexpr int padded(int per) { return (per + 127) & ~127; }
constexpr size_t bin_smem(int per) { return (size_t)per * 12 + (size_t)padded(per) * 4; }

template <bool kWrite>
__global__ void __launch_bounds__(kBinThreads) tile_bins_kernel(const BinArgs g) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smem[];
  ushort4* srect = reinterpret_cast<ushort4*>(smem);           // [per]
  uint32_t* sid = reinterpret_cast<uint32_t*>(srect + g.per);  // [per]
  uint32_t* sbin = sid + g.per;                                // [padded] packed bins
  __shared__ uint16_t sbuf[kBinWarps][64];                      // a warp's picked splats
  __shared__ uint2 stile[kBinWarps][kWrite ? 64 : 1];           // {splats, next place} per tile
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  int lo, hi, ntx = g.ntx, nty = g.nty;
  size_t row;  // first value of the chunk's histogram row
  int tile_off = 0;
  if (g.chunks) {
    const int4 c = g.chunks[blockIdx.x];
    const InstGeom geo = g.geom[c.z];
    lo = c.x, hi = c.y;
    ntx = geo.ntx, nty = geo.nty, tile_off = geo.tile_off;
    row = (size_t)c.w;
  } else {
    lo = min(g.n, (int)blockIdx.x * g.per);
    hi = min(g.n, lo + g.per);
    row = (size_t)blockIdx.x * ntx * nty;
  }
  const int nbx = (ntx + kBin - 1) / kBin, bins = nbx * ((nty + kBin - 1) / kBin);
  if ((int)blockIdx.y * kBinWarps >= bins) return;  // uniform
  const int count = hi - lo;
  // Pairs past the capacity are dropped in depth order: last_p is the splat whose
  // pairs fill it, with last_m of them kept.  (Batches: its position in their order; what
  // is behind it has an empty rectangle.)
  const uint32_t last_p = g.sc->last_p, last_m = g.sc->last_m;
  for (int k = threadIdx.x; k < ((count + 127) & ~127); k += kBinThreads) {
    uint32_t b = 0x7f7f7f7fu;  // reaches no bin
    if (k < count) {
      const ushort4 r = g.rect[lo + k];
      srect[k] = r;
      if (r.x <= r.y && (g.chunks || (uint32_t)(lo + k) <= last_p))
        b = bin_bytes(r.x / kBin, r.z / kBin, r.y / kBin, r.w / kBin);
      if (kWrite) sid[k] = g.perm[lo + k];
    }
    sbin[k] = b;
  }
  __syncthreads();
  for (int b = blockIdx.y * kBinWarps + w; b < bins; b += gridDim.y * kBinWarps) {
    const int BX = b % nbx, BY = b / nbx, X0 = BX * kBin, Y0 = BY * kBin;
    const uint32_t key = bin_bytes(BX, BY, BX, BY) | 0x80808080u;
    // lane t has tiles (X0 + t % 8, Y0 + t / 8) and the one four rows below
    const int tx = X0 + (lane & 7), ty = Y0 + (lane >> 3);
    const bool in0 = tx < ntx && ty < nty, in1 = tx < ntx && ty + 4 < nty;
    const int t0 = ty * ntx + tx, t1 = t0 + 4 * ntx;
    uint32_t at0 = 0, at1 = 0;  // counts, or the next place in the tile's list
    if (kWrite) {
      if (in0) at0 = (uint32_t)g.ranges[tile_off + t0].x + g.hist[row + t0];
      if (in1) at1 = (uint32_t)g.ranges[tile_off + t1].x + g.hist[row + t1];
    }
    auto place = [&](int k) {  // the first k splats of the warp's buffer
      uint32_t m0 = 0, m1 = 0, id = 0;
      if (lane < k) {
        const int q = sbuf[w][lane];
        tile_mask(srect[q], X0, Y0, (uint32_t)(lo + q) == last_p ? last_m : 0xffffffffu, m0, m1);
        if (kWrite) id = sid[q];
      }
      uint32_t w0 = transpose32(m0, lane), w1 = transpose32(m1, lane);
      const uint32_t c0 = __popc(w0), c1 = __popc(w1);
      if (kWrite) {
        // Tiles with few of the splats: their lanes append one each in turn.  With many:
        // the splats of one tile are written together, side by side.
        uint32_t big0 = __ballot_sync(0xffffffffu, c0 > kFew);
        uint32_t big1 = __ballot_sync(0xffffffffu, c1 > kFew);
        if (__popc(big0) + __popc(big1) > 24) {
          stile[w][lane] = make_uint2(w0, at0);
          stile[w][32 + lane] = make_uint2(w1, at1);
          __syncwarp();
#pragma unroll 16
          for (int t = 0; t < 64; ++t) {
            const uint2 v = stile[w][t];
            if (v.x >> lane & 1u) g.out[v.y + __popc(v.x & lt)] = id;
          }
          __syncwarp();
        } else {
          for (; big0; big0 &= big0 - 1u) {
            const int t = __ffs(big0) - 1;
            const uint32_t word = __shfl_sync(0xffffffffu, w0, t);
            const uint32_t p = __shfl_sync(0xffffffffu, at0, t);
            if (word >> lane & 1u) g.out[p + __popc(word & lt)] = id;
          }
          for (; big1; big1 &= big1 - 1u) {
            const int t = __ffs(big1) - 1;
            const uint32_t word = __shfl_sync(0xffffffffu, w1, t);
            const uint32_t p = __shfl_sync(0xffffffffu, at1, t);
            if (word >> lane & 1u) g.out[p + __popc(word & lt)] = id;
          }
          uint32_t p0 = at0, p1 = at1;
          if (c0 > kFew) w0 = 0u;
          if (c1 > kFew) w1 = 0u;
          while (__any_sync(0xffffffffu, (w0 | w1) != 0u)) {
            const uint32_t v0 = __shfl_sync(0xffffffffu, id, w0 ? __ffs(w0) - 1 : 0);
            const uint32_t v1 = __shfl_sync(0xffffffffu, id, w1 ? __ffs(w1) - 1 : 0);
            if (w0) g.out[p0++] = v0;
            if (w1) g.out[p1++] = v1;
            w0 &= w0 - 1u;
            w1 &= w1 - 1u;
          }
        }
      }
      at0 += c0;
      at1 += c1;
    };
    int pend = 0;
    for (int k = 0; k < count; k += 128) {
      uint32_t word[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        word[u] = __ballot_sync(0xffffffffu, reaches(sbin[k + 32 * u + lane], key));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!word[u]) continue;
        pend = warp_gather(sbuf[w], pend, word[u], k + 32 * u, lane, place);
      }
    }
    __syncwarp();
    if (pend > 0) place(pend);
    __syncwarp();
    if (!kWrite) {
      if (in0) g.hist[row + t0] = at0;
      if (in1) g.hist[row + t1] = at1;
    }
  }
}

__global__ void __launch_bounds__(kBinThreads)
    gather_rects_kernel(const ushort4* __restrict__ rect, const uint32_t* __restrict__ perm,
                        const uint32_t* __restrict__ seg_start, int n, uint32_t cap,
                        ushort4* __restrict__ rect_sorted, DevScalars* __restrict__ sc) {
  pdl_wait();
  const int p = blockIdx.x * kBinThreads + threadIdx.x;
  if (p >= n) return;
  const uint32_t id = perm[p];
  ushort4 r = rect[id];
  const uint32_t area = (uint32_t)((int)r.y - (int)r.x + 1) * (uint32_t)((int)r.w - (int)r.z + 1);
  const uint32_t room = area ? cap - seg_start[id] : 0u;  // (seg_start stops at cap)
  if (area > room) {
    if (room == 0u) {
      r = make_ushort4(1, 0, 1, 0);
    } else {  // at most one splat
      sc->last_p = (uint32_t)p;
      sc->last_m = room;
    }
  }
  rect_sorted[p] = r;
}

// Longest-first schedule of the composite CTAs: tiles bucketed by their list
// length (quarter-octave buckets), buckets in descending order.  The heaviest
// tiles start in the first wave, so they no longer set the kernel's tail.  The
// order inside a bucket is arbitrary (plain shared atomics hand out the
// slots); every tile's result is independent of it.
constexpr int kOrderBuckets = 128;

__device__ __forceinline__ int work_bucket(int2 r) {
  const uint32_t len = (uint32_t)max(r.y - r.x, 0);
  if (len == 0) return 0;
  const int l = 31 - __clz(len);
  const uint32_t sub = l >= 2 ? (len >> (l - 2)) & 3u : (len << (2 - l)) & 3u;
  return min(kOrderBuckets - 1, 1 + 4 * l + (int)sub);
}

// The schedule of tiles [0, tiles) from their ranges, by one 1024-thread CTA.
__device__ void order_tiles(const int2* __restrict__ ranges, int tiles, int32_t* __restrict__ order) {
  __shared__ uint32_t cnt[kOrderBuckets];
  __shared__ uint32_t off[kOrderBuckets];
  for (int b = threadIdx.x; b < kOrderBuckets; b += blockDim.x) cnt[b] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int rounds = (tiles + (int)blockDim.x - 1) / (int)blockDim.x;
  for (int r = 0; r < rounds; ++r) {
    const int t = r * blockDim.x + threadIdx.x;
    if (t < tiles) atomicAdd(&cnt[work_bucket(ranges[t])], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // lane l owns buckets 127-4l .. 124-4l (descending); exclusive scan over lanes
    uint32_t v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = cnt[kOrderBuckets - 1 - 4 * lane - k];
      s += v[k];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    uint32_t run = incl - s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      off[kOrderBuckets - 1 - 4 * lane - k] = run;
      run += v[k];
    }
  }
  __syncthreads();
  for (int r = 0; r < rounds; ++r) {
    const int t = r * blockDim.x + threadIdx.x;
    if (t < tiles) order[atomicAdd(&off[work_bucket(ranges[t])], 1u)] = t;
  }
}

__global__ void __launch_bounds__(1024)
    tile_order_kernel(const int2* __restrict__ ranges, int tiles, int32_t* __restrict__ order) {
  pdl_wait();
  order_tiles(ranges, tiles, order);
}

constexpr int kOffsetThreads = 1024;  // 32 tiles x 32 slices of the chunk column

__global__ void __launch_bounds__(kOffsetThreads)
    tile_offsets_kernel(uint32_t* __restrict__ hist, int chunks, int tiles,
                        const uint16_t* __restrict__ tile_inst,
                        const InstGeom* __restrict__ geom, const int2* __restrict__ inst_hist,
                        uint32_t* __restrict__ totals, int2* __restrict__ ranges,
                        DevScalars* __restrict__ sc, int32_t* __restrict__ order) {
  pdl_wait();
  constexpr int kSlices = kOffsetThreads / 32;
  __shared__ uint32_t part[kSlices][33];
  __shared__ uint32_t wsum[kSlices];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
  const int t = blockIdx.x * 32 + lane;
  // the tile's column: hist[col + r * pitch], one row per chunk (of its instance)
  size_t col = (size_t)t;
  int pitch = tiles, rows = chunks;
  if (geom && t < tiles) {
    const int k = tile_inst[t];
    const InstGeom g = geom[k];
    const int2 h = inst_hist[k];  // {first of hist, chunks}
    pitch = g.ntx * g.nty;
    col = (size_t)h.x + (t - g.tile_off);
    rows = h.y;
  }
  const int r0 = s * rows / kSlices, r1 = (s + 1) * rows / kSlices;
  uint32_t sum = 0;
  if (t < tiles) {
#pragma unroll 4
    for (int r = r0; r < r1; ++r) sum += hist[col + (size_t)r * pitch];
  }
  part[s][lane] = sum;
  __syncthreads();
  uint32_t run = 0;
  for (int k = 0; k < s; ++k) run += part[k][lane];
  if (t < tiles) {
    for (int r = r0; r < r1; ++r) {
      const size_t q = col + (size_t)r * pitch;
      const uint32_t v = hist[q];
      hist[q] = run;
      run += v;
    }
    if (s == kSlices - 1) totals[t] = run;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&sc->sort_ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // Last CTA: exclusive scan of the totals into the ranges; each thread takes
  // a contiguous run of tiles.
  const int per = (tiles + kOffsetThreads - 1) / kOffsetThreads;
  const int a = min(tiles, threadIdx.x * per), b = min(tiles, a + per);
  uint32_t mine = 0;
  for (int k = a; k < b; ++k) mine += ((volatile uint32_t*)totals)[k];
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[s] = incl;
  __syncthreads();
  if (s == 0) {
    const uint32_t w = wsum[lane];
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += v;
    }
    wsum[lane] = wi - w;  // exclusive over the warps
  }
  __syncthreads();
  uint32_t base = incl - mine + wsum[s];
  for (int k = a; k < b; ++k) {
    const uint32_t c = ((volatile uint32_t*)totals)[k];
    ranges[k] = c ? make_int2((int)base, (int)(base + c)) : make_int2(0, 0);
    base += c;
  }
  if (threadIdx.x == 0) sc->sort_ticket = 0u;
  if (order) {
    // the longest-first composite schedule from the ranges just written
    __syncthreads();
    order_tiles(ranges, tiles, order);
  }
}

int bins_of(int ntx, int nty) {
  return ((ntx + kBin - 1) / kBin) * ((nty + kBin - 1) / kBin);
}

// Splats per chunk: a (chunk, bin) task per warp and four waves of 8 warps on 148 SMs.
int chunk_of(double tests) {
  const int64_t want = (int64_t)std::ceil(tests / (148 * 32));
  return (int)std::min<int64_t>(kChunkMax, std::max<int64_t>(kChunkMin, (want + 31) / 32 * 32));
}

int offsets(RasterBuffers& rb, int chunks, const int2* inst_hist, cudaStream_t s) {
  int32_t* order =
      (rb.tile_order && rb.schedule == DS_SCHEDULE_LONGEST_FIRST) ? rb.tile_order : nullptr;
  DS_CUDA(launch_pdl(tile_offsets_kernel, dim3((rb.tiles + 31) / 32), dim3(kOffsetThreads), 0, s,
                     rb.tile_hist, chunks, rb.tiles, rb.tile_inst, inst_hist ? rb.geom : nullptr,
                     inst_hist, rb.tile_totals, rb.ranges, rb.scalars, order));
  return DS_OK;
}

}  // namespace

// The cost by bins follows the splats per bin (and the fullest bin, which one warp of a
// chunk walks alone), that of sorting pairs the pairs.  B200, depth sort and list
// build, by bins / by pairs:
//   random splats over the image: 4096 at 256x256 0.070 / 0.070 ms, 30011 at 797x531
//   0.080 / 0.087, 60000 at 1280x720 (47 tiles each) 0.093 / 0.118, 60000 at 1920x1080
//   0.112 / 0.189; 16 uneven batched fits, whole step 1.84 / 2.61
//   surfaces seen from a distance (2 tiles each, most in few bins): 5000 at 512x512
//   0.071 / 0.073, 60000 at 1280x720 0.100 / 0.083, 300000 0.144 / 0.098, a million at
//   1920x1080 0.327 / 0.206
// What decides is the splats per bin, which the host does not know; their number stands
// in for it.  A fit of many splats comes with small ones, so those sort pairs, and batches
// are of many small fits.  It is a guess either way: surfaces of 60000 splats would be
// 0.02 ms faster by pairs, and 300000 splats over a whole image (29 million pairs) 1.9 ms
// faster by bins.
bool tile_bins_pay(const RasterBuffers& rb, const InstGeom* inst) {
  const int k = inst ? rb.instances : 1;
  double hist = 0;
  for (int i = 0; i < k; ++i) {
    const int ntx = inst ? inst[i].ntx : rb.ntx, nty = inst ? inst[i].nty : rb.nty;
    if (std::max(ntx, nty) > kBin * kBinMaxAxis) return false;
    const double n = inst ? inst[i].count : rb.max_splats;
    hist += (n / kChunkMin + 1) * ntx * nty;
  }
  return hist <= 2e9 && (inst || rb.max_splats <= kBinSplats);
}

int tile_bins_alloc(RasterBuffers& rb, const InstGeom* inst) {
  size_t values = 0;
  if (!inst) {
    // more splats, longer chunks: the rows of n splats are bounded by those of the
    // shortest chunk up to where it grows, and by those of max_splats
    const double bins = bins_of(rb.ntx, rb.nty);
    const int64_t short_rows = std::min<int64_t>((rb.max_splats + kChunkMin - 1) / kChunkMin,
                                                 (int64_t)(148 * 32 / bins) + 2);
    const int per = chunk_of(bins * rb.max_splats);
    values = (size_t)std::max<int64_t>(short_rows, (rb.max_splats + per - 1) / per + 1) * rb.tiles;
  } else {
    double tests = 0;
    for (int k = 0; k < rb.instances; ++k)
      tests += (double)inst[k].count * bins_of(inst[k].ntx, inst[k].nty);
    rb.bin_per = chunk_of(tests);
    rb.bin_most = 0;
    std::vector<int4> chunks;
    std::vector<int2> first(rb.instances);
    for (int k = 0; k < rb.instances; ++k) {
      const InstGeom& g = inst[k];
      rb.bin_most = std::max(rb.bin_most, bins_of(g.ntx, g.nty));
      const int rows = (g.count + rb.bin_per - 1) / rb.bin_per;
      first[k] = make_int2((int)values, rows);
      for (int r = 0; r < rows; ++r) {
        const int lo = g.splat_off + r * rb.bin_per;
        chunks.push_back(make_int4(lo, std::min(lo + rb.bin_per, g.splat_off + g.count), k,
                                   (int)values));
        values += (size_t)g.ntx * g.nty;
      }
      if (values > INT32_MAX) return DS_ERR_OOM;
    }
    rb.bin_chunk_count = (int)chunks.size();
    DS_CUDA(device_alloc(&rb.bin_chunks, chunks.size() * sizeof(int4)));
    DS_CUDA(device_alloc(&rb.inst_hist, first.size() * sizeof(int2)));
    DS_CUDA(cudaMemcpy(rb.bin_chunks, chunks.data(), chunks.size() * sizeof(int4),
                       cudaMemcpyHostToDevice));
    DS_CUDA(cudaMemcpy(rb.inst_hist, first.data(), first.size() * sizeof(int2),
                       cudaMemcpyHostToDevice));
  }
  DS_CUDA(device_alloc(&rb.tile_hist, std::max<size_t>(1, values) * 4));
  DS_CUDA(device_alloc(&rb.tile_totals, (size_t)std::max(1, rb.tiles) * 4));
  return DS_OK;
}

int gather_rects(RasterBuffers& rb, int n, cudaStream_t s) {
  DS_CUDA(launch_pdl(gather_rects_kernel, dim3((n + kBinThreads - 1) / kBinThreads),
                     dim3(kBinThreads), 0, s, rb.rect, rb.depth_perm, rb.seg_start, n,
                     (uint32_t)rb.cap, rb.rect_sorted, rb.scalars));
  return DS_OK;
}

int tile_bins(RasterBuffers& rb, int n, cudaStream_t s) {
  const bool batch = rb.bin_chunks != nullptr;
  const int bins = batch ? rb.bin_most : bins_of(rb.ntx, rb.nty);
  BinArgs g;
  g.rect = rb.rect_sorted;
  g.perm = rb.depth_perm;
  g.n = n;
  g.per = batch ? rb.bin_per : chunk_of((double)bins * n);
  g.ntx = rb.ntx;
  g.nty = rb.nty;
  g.chunks = rb.bin_chunks;
  g.geom = rb.geom;
  g.hist = rb.tile_hist;
  g.ranges = rb.ranges;
  g.out = rb.sorted_splat;
  g.sc = rb.scalars;
  const int chunks = batch ? rb.bin_chunk_count : (n + g.per - 1) / g.per;
  // the bins of a chunk go to several CTAs while there are few chunks
  const int split = std::max(1, std::min((bins + kBinWarps - 1) / kBinWarps, 148 * 16 / chunks));
  const dim3 grid(chunks, split);
  DS_CUDA(launch_pdl(tile_bins_kernel<false>, grid, dim3(kBinThreads), bin_smem(g.per), s, g));
  DS_TRY(offsets(rb, chunks, rb.inst_hist, s));
  DS_CUDA(launch_pdl(tile_bins_kernel<true>, grid, dim3(kBinThreads), bin_smem(g.per), s, g));
  return cuda_status(cudaGetLastError());
}

int tile_offsets(RasterBuffers& rb, int chunks, cudaStream_t s) {
  return offsets(rb, chunks, nullptr, s);
}

int tile_order(RasterBuffers& rb, cudaStream_t s) {
  if (rb.tile_order && rb.schedule == DS_SCHEDULE_LONGEST_FIRST)
    DS_CUDA(launch_pdl(tile_order_kernel, dim3(1), dim3(1024), 0, s, rb.ranges, rb.tiles,
                       rb.tile_order));
  return DS_OK;
}

}  // namespace ds
