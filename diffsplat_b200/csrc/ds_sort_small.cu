// Depth order of up to 65536 splats of a single instance: the stable sort of (depth
// bits, id) that the radix passes of ds_sort.cu do in twelve launches, each of which
// has less than a microsecond's work at these sizes (0.045 ms together, of the 0.105
// ms step of a 256x256 fit).
//
// Up to kRankSort splats every splat counts those before it: n^2 comparisons spread
// over all SMs.  The same pass adds up their tiles, so the offsets of
// scan_counts_permuted come with it: 7 us for 4096 splats where sort and scan took 53 (256x256
// fit 105 -> 77 us a step), 15 us for 8192; it grows with n^2, so the line lies there.
//
// Above that, one thread-block cluster sorts in its shared memory: 21 us for 16384
// splats, 27 for 30011, 39 for 60000.  Per 8-bit digit in which the keys differ at all,
// each warp ranks its items (by ballots: a match instruction takes 60 cycles of its SM
// here, eight ballots a quarter of that), the CTA groups them by digit, and the runs go
// to their places in the CTAs that hold those parts of the order, by coalesced stores to
// distributed shared memory (item by item they took twice the time).
#include <cooperative_groups.h>

#include "ds_common.cuh"
#include "ds_internal.h"

namespace cg = cooperative_groups;

namespace ds {

namespace {

// ---- by counting ----------------------------------------------------------------

constexpr int kRankThreads = 256;
constexpr int kRankChunk = 256;  // splats that a CTA compares its 256 with

__device__ __forceinline__ uint32_t area_of(const ushort4& r) {
  return (uint32_t)((int)r.y - (int)r.x + 1) * (uint32_t)((int)r.w - (int)r.z + 1);
}

// Adds to rank[i] and before[i] the splats of a chunk ahead of splat i, and their tiles.
__global__ void __launch_bounds__(kRankThreads)
    rank_kernel(const uint32_t* __restrict__ keys, const ushort4* __restrict__ rect, int n,
                uint32_t* __restrict__ rank, uint32_t* __restrict__ before,
                DevScalars* __restrict__ sc) {
  pdl_wait();
  __shared__ __align__(16) uint2 other[kRankChunk];  // {key, tiles}
  const int i = blockIdx.x * kRankThreads + threadIdx.x;
  const int j0 = blockIdx.y * kRankChunk, m = min(kRankChunk, n - j0);
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) sc->n_long = 0u;
  if ((int)threadIdx.x < m)
    other[threadIdx.x] = make_uint2(keys[j0 + threadIdx.x], area_of(rect[j0 + threadIdx.x]));
  else
    other[threadIdx.x] = make_uint2(0xffffffffu, 0u);  // ahead of none (and of no id below)
  __syncthreads();
  const uint32_t key = i < n ? keys[i] : 0u;
  uint32_t r = 0, o = 0;
  auto count = [&](auto ahead) {
#pragma unroll 8
    for (int j = 0; j < kRankChunk; j += 2) {
      const uint4 two = *reinterpret_cast<const uint4*>(&other[j]);
      if (ahead(two.x, j0 + j)) r += 1u, o += two.y;
      if (ahead(two.z, j0 + j + 1)) r += 1u, o += two.w;
    }
  };
  if (blockIdx.y > blockIdx.x) count([&](uint32_t k, int) { return k < key; });
  else if (blockIdx.y < blockIdx.x) count([&](uint32_t k, int) { return k <= key; });
  else count([&](uint32_t k, int j) { return k < key || (k == key && j < i); });
  if (i < n) {
    if (r) atomicAdd(&rank[i], r);
    if (o) atomicAdd(&before[i], o);
  }
}

// Everything in its place in the order; rank and before are left zero for the next call.
__global__ void __launch_bounds__(kRankThreads)
    place_kernel(const ushort4* __restrict__ rect, int n, uint32_t cap,
                 uint32_t* __restrict__ rank, uint32_t* __restrict__ before,
                 uint32_t* __restrict__ perm, ushort4* __restrict__ rect_sorted,
                 unsigned long long* __restrict__ offsets, uint32_t* __restrict__ seg_start,
                 uint4* __restrict__ long_list, DevScalars* __restrict__ sc) {
  pdl_wait();
  const int i = blockIdx.x * kRankThreads + threadIdx.x;
  if (i >= n) return;
  const uint32_t p = rank[i], s0 = before[i];
  rank[i] = 0u;
  before[i] = 0u;
  const ushort4 r = rect[i];
  const uint32_t area = area_of(r), s1 = s0 + area;  // < 2^32: see small_sort
  perm[p] = (uint32_t)i;
  rect_sorted[p] = r;
  offsets[p] = s0;
  if (area) {
    seg_start[i] = min(s0, cap);
    if (s0 < cap && s1 >= cap) {
      sc->last_p = p;
      sc->last_m = cap - s0;
    }
    if (long_list && area > kSerialRecords)
      long_list[atomicAdd(&sc->n_long, 1u)] =
          make_uint4((uint32_t)i, min(s0, cap), min(s1, cap), 0u);
  }
  if (p == (uint32_t)n - 1u) {  // s1 is the number of pairs
    sc->n_isects_raw = s1;
    sc->n_isects = min(s1, cap);
    if (s1 > cap) atomicOr(&sc->status, kStatusIsectOverflow);
    if (s1 < cap) sc->last_p = 0xffffffffu;  // else the splat that fills it writes
  }
}

// ---- by one cluster ---------------------------------------------------------------

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;       // most items per thread
constexpr int kClusterMax = 8;  // CTAs, the portable most
static_assert(kSmallSort == kThreads * kItems * kClusterMax, "items of a full cluster");

struct SortShared {
  uint2 group[kThreads * kItems];    // {key, id}: this CTA's items by digit
  uint2 order[kThreads * kItems];    // its part of the order (written by the cluster)
  uint16_t cnt[kWarps][256];         // a warp's digit counts, then its offsets in the quarter
  uint32_t part[4][256];             // digit counts of 8 warps each, then their local starts
  uint32_t total[256];               // digit counts of this CTA (read by the cluster)
  uint32_t shift_to[256];            // place in the order minus place in the CTA, per digit
  uint2 wsum[8];
  uint32_t wand[kWarps], wor[kWarps];
  uint32_t all_and, all_or;          // of this CTA's keys (read by the cluster)
};

__global__ void __launch_bounds__(kThreads, 1)
    cluster_sort_kernel(const uint32_t* __restrict__ keys, int n, int log_seg,
                        uint32_t* __restrict__ perm) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smem[];
  SortShared& sm = *reinterpret_cast<SortShared*>(smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const int seg = 1 << log_seg, items = seg / kThreads;  // items per thread
  const int first = w * items * 32 + lane;               // this thread's first item
  const int valid = min(seg, max(0, n - rank * seg));    // items of this CTA
  uint2 item[kItems];
  uint32_t band = 0xffffffffu, bor = 0u;
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int q = first + 32 * it;
    item[it] = make_uint2(0u, 0u);
    if (it < items && q < valid) {
      item[it] = make_uint2(keys[rank * seg + q], (uint32_t)(rank * seg + q));
      band &= item[it].x;
      bor |= item[it].x;
    }
  }
  band = __reduce_and_sync(0xffffffffu, band);
  bor = __reduce_or_sync(0xffffffffu, bor);
  if (lane == 0) {
    sm.wand[w] = band;
    sm.wor[w] = bor;
  }
  __syncthreads();
  if (w == 0) {
    band = __reduce_and_sync(0xffffffffu, sm.wand[lane]);
    bor = __reduce_or_sync(0xffffffffu, sm.wor[lane]);
    if (lane == 0) {
      sm.all_and = band;
      sm.all_or = bor;
    }
  }
  cluster.sync();
  band = 0xffffffffu, bor = 0u;
  for (int c = 0; c < ctas; ++c) {
    band &= *cluster.map_shared_rank(&sm.all_and, c);
    bor |= *cluster.map_shared_rank(&sm.all_or, c);
  }
  const uint32_t varying = band ^ bor;
  for (int shift = 0; shift < 32; shift += 8) {
    if (!(varying >> shift & 255u)) continue;
    uint32_t* zero = reinterpret_cast<uint32_t*>(sm.cnt[w]);
#pragma unroll
    for (int k = 0; k < 4; ++k) zero[32 * k + lane] = 0u;
    __syncwarp();
    uint32_t rnk[kItems];
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      if (it >= items) continue;
      const bool ok = first + 32 * it < valid;
      const uint32_t d = (item[it].x >> shift) & 255u;
      uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool bit = d >> b & 1u;
        const uint32_t vote = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? vote : ~vote;
      }
      const uint32_t pre = sm.cnt[w][d];
      __syncwarp();
      if (ok && (peers & lt) == 0u) sm.cnt[w][d] = (uint16_t)(pre + __popc(peers));
      __syncwarp();
      rnk[it] = pre + __popc(peers & lt);
    }
    __syncthreads();
    const int d = threadIdx.x & 255, q = threadIdx.x >> 8;
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t c = sm.cnt[8 * q + k][d];
      sm.cnt[8 * q + k][d] = (uint16_t)run;
      run += c;
    }
    sm.part[q][d] = run;
    __syncthreads();
    uint32_t own = 0;
    if (q == 0) {
      own = sm.part[0][d] + sm.part[1][d] + sm.part[2][d] + sm.part[3][d];
      sm.total[d] = own;
    }
    cluster.sync();
    uint32_t all = 0, before = 0;
    uint2 incl = make_uint2(0u, 0u);  // over the digits: of the cluster, of this CTA
    if (q == 0) {
#pragma unroll
      for (int c = 0; c < kClusterMax; ++c) {
        if (c >= ctas) continue;
        const uint32_t v = cluster.map_shared_rank(sm.total, c)[d];
        all += v;
        before += c < rank ? v : 0u;
      }
      incl = make_uint2(all, own);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, incl.x, o);
        const uint32_t b = __shfl_up_sync(0xffffffffu, incl.y, o);
        if (lane >= o) incl.x += a, incl.y += b;
      }
      if (lane == 31) sm.wsum[w] = incl;
    }
    __syncthreads();
    if (q == 0) {
      uint32_t place = incl.x - all + before, local = incl.y - own;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint2 s = sm.wsum[k];
        if (k < w) place += s.x, local += s.y;
      }
      sm.shift_to[d] = place - local;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t c = sm.part[k][d];
        sm.part[k][d] = local;
        local += c;
      }
    }
    __syncthreads();
    // group the CTA's items by digit, then send the runs to their places
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      if (it >= items || first + 32 * it >= valid) continue;
      const uint32_t dd = (item[it].x >> shift) & 255u;
      sm.group[sm.part[w >> 3][dd] + sm.cnt[w][dd] + rnk[it]] = item[it];
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      const int j = it * kThreads + threadIdx.x;
      if (it >= items || j >= valid) continue;
      const uint2 v = sm.group[j];
      const uint32_t p = sm.shift_to[(v.x >> shift) & 255u] + (uint32_t)j;
      cluster.map_shared_rank(&sm.order[0], p >> log_seg)[p & (seg - 1)] = v;
    }
    cluster.sync();
#pragma unroll
    for (int it = 0; it < kItems; ++it)
      if (it < items && first + 32 * it < valid) item[it] = sm.order[first + 32 * it];
    // (the cluster writes `order` again only past the next digit's barrier)
  }
#pragma unroll
  for (int it = 0; it < kItems; ++it)
    if (it < items && first + 32 * it < valid) perm[rank * seg + first + 32 * it] = item[it].y;
  cluster.sync();  // no CTA leaves while another reads its shared memory
}

}  // namespace

int small_sort_setup() {
  static std::atomic<uint64_t> set{0};
  return cuda_status(allow_smem(cluster_sort_kernel, sizeof(SortShared), set));
}

bool rank_sort_fits(const RasterBuffers& rb, int n) {
  return n <= kRankSort && (int64_t)n * rb.tiles < ((int64_t)1 << 32);  // 32-bit pair offsets
}

int rank_sort(RasterBuffers& rb, int n, bool with_long_list, cudaStream_t s) {
  const unsigned blocks = (unsigned)((n + kRankThreads - 1) / kRankThreads);
  static_assert(kRankThreads == kRankChunk, "blocks of ids and chunks coincide");
  rb.depth_perm = rb.depth_v0;
  DS_CUDA(launch_pdl(rank_kernel, dim3(blocks, blocks), dim3(kRankThreads), 0, s, rb.depth_keys,
                     rb.rect, n, rb.rank, rb.rank + kRankSort, rb.scalars));
  DS_CUDA(launch_pdl(place_kernel, dim3(blocks), dim3(kRankThreads), 0, s, rb.rect, n,
                     (uint32_t)rb.cap, rb.rank, rb.rank + kRankSort, rb.depth_perm,
                     rb.rect_sorted, rb.emit_offsets, rb.seg_start,
                     with_long_list ? rb.long_list : nullptr, rb.scalars));
  return DS_OK;
}

int cluster_sort(RasterBuffers& rb, int n, cudaStream_t s) {
  if (n <= 0 || n > kSmallSort) return DS_ERR_ARG;
  // two items per thread while the cluster can grow, then up to kItems
  int ctas = 1;
  while (ctas < kClusterMax && ctas * kThreads * 2 < n) ctas *= 2;
  int log_seg = 10;
  while (((int64_t)ctas << log_seg) < n) ++log_seg;
  rb.depth_perm = rb.depth_v0;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)ctas;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(SortShared);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  DS_CUDA(cudaLaunchKernelEx(&cfg, cluster_sort_kernel, (const uint32_t*)rb.depth_keys, n, log_seg,
                             rb.depth_perm));
  return DS_OK;
}

}  // namespace ds
