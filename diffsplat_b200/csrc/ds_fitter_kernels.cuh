// Kernels of the fused training step shared by the single fitter
// (ds_fitter.cu) and the batched fitter (ds_batch.cu): step begin (Adam bias
// corrections), and per-splat projection backward -> activation backward ->
// Adam on every field.
#pragma once
#include <float.h>
#include <math.h>

#include <vector>

#include "ds_common.cuh"
#include "ds_internal.h"
#include "ds_preprocess.cuh"

namespace ds {

namespace {

constexpr int kThreads = 256;
constexpr int kBcTableMax = 1 << 20;
#ifndef DS_ADAM_BLOCKS
#define DS_ADAM_BLOCKS 3
#endif

struct Lrs {
  float pos, scale, rot, sh_dc, sh_rest, opacity;
};

__global__ void step_begin_kernel(DevScalars* sc, const float2* __restrict__ bc_table,
                                  int table_len, float2* __restrict__ bc_out) {
  pdl_wait();
  uint32_t t = sc->step + 1u;
  sc->step = t;
  sc->visible = 0u;
  sc->ticket = 0u;
  sc->n_splats = sc->n_splats;  // set once at creation
  float2 bc = make_float2(1.f, 1.f);
  if ((int)t <= table_len) bc = bc_table[t - 1];
  *bc_out = bc;
}

__device__ __forceinline__ void adam1(float& p, float& m, float& v, float g, float lr, float b1,
                                      float b2, float eps, float bc1, float bc2) {
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  float m_hat = m * bc1;
  float v_hat = v * bc2;
  p -= lr * m_hat / (sqrtf(v_hat) + eps);
}

// Integer hash "lowbias32" (C. Wellons, 2018): the random bits of the
// stochastic rounding of BF16 Adam moments, from (element, field, step).
__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// FP32 -> BF16 with stochastic rounding: adds 16 random bits below the kept
// mantissa and truncates, so E[result] = x.  An Adam moment updated by
// (1 - beta2) = 1e-3 of itself per step would otherwise round back to its old
// value forever under round-to-nearest (BF16 keeps 8 significant bits).
__device__ __forceinline__ __nv_bfloat16 bf16_stochastic(float x, uint32_t r) {
  uint32_t u = __float_as_uint(x);
  if ((u & 0x7f800000u) == 0x7f800000u) return __float2bfloat16_rn(x);
  u += r & 0xffffu;
  return __ushort_as_bfloat16((unsigned short)(u >> 16));
}

struct AdamHyper {
  float b1, b2, eps;
};

// dL/dCov3D -> dL/d(log-scale, raw quaternion); identical to the layer
// backward in ds_activ_project.cu (gauss_activ_layer.cu:259-329).
__device__ __forceinline__ void cov_backward(float rw, float rx, float ry, float rz, float lsx,
                                             float lsy, float lsz, float g_xx, float g_xy,
                                             float g_xz, float g_yy, float g_yz, float g_zz,
                                             float* d) {
  UnitQuat nq = unit_quat(rw, rx, ry, rz);
  Rot3 R = rot_from_quat(nq.w, nq.x, nq.y, nq.z);
  float sx = expf(lsx), sy = expf(lsy), sz = expf(lsz);
  float m00 = R.r00 * sx, m01 = R.r01 * sy, m02 = R.r02 * sz;
  float m10 = R.r10 * sx, m11 = R.r11 * sy, m12 = R.r12 * sz;
  float m20 = R.r20 * sx, m21 = R.r21 * sy, m22 = R.r22 * sz;
  float dm00 = 2.f * (g_xx * m00 + g_xy * m10 + g_xz * m20);
  float dm01 = 2.f * (g_xx * m01 + g_xy * m11 + g_xz * m21);
  float dm02 = 2.f * (g_xx * m02 + g_xy * m12 + g_xz * m22);
  float dm10 = 2.f * (g_xy * m00 + g_yy * m10 + g_yz * m20);
  float dm11 = 2.f * (g_xy * m01 + g_yy * m11 + g_yz * m21);
  float dm12 = 2.f * (g_xy * m02 + g_yy * m12 + g_yz * m22);
  float dm20 = 2.f * (g_xz * m00 + g_yz * m10 + g_zz * m20);
  float dm21 = 2.f * (g_xz * m01 + g_yz * m11 + g_zz * m21);
  float dm22 = 2.f * (g_xz * m02 + g_yz * m12 + g_zz * m22);
  d[0] = (dm00 * R.r00 + dm10 * R.r10 + dm20 * R.r20) * sx;
  d[1] = (dm01 * R.r01 + dm11 * R.r11 + dm21 * R.r21) * sy;
  d[2] = (dm02 * R.r02 + dm12 * R.r12 + dm22 * R.r22) * sz;
  float dr00 = dm00 * sx, dr10 = dm10 * sx, dr20 = dm20 * sx;
  float dr01 = dm01 * sy, dr11 = dm11 * sy, dr21 = dm21 * sy;
  float dr02 = dm02 * sz, dr12 = dm12 * sz, dr22 = dm22 * sz;
  float dqw = 2.f * (dr10 * nq.z - dr20 * nq.y + dr01 * (-nq.z) + dr21 * nq.x + dr02 * nq.y +
                     dr12 * (-nq.x));
  float dqx = 2.f * (dr10 * nq.y + dr20 * nq.z + dr01 * nq.y + dr11 * (-2.f * nq.x) + dr21 * nq.w +
                     dr02 * nq.z + dr12 * (-nq.w) + dr22 * (-2.f * nq.x));
  float dqy = 2.f * (dr00 * (-2.f * nq.y) + dr10 * nq.x + dr20 * (-nq.w) + dr01 * nq.x +
                     dr12 * nq.z + dr21 * nq.z + dr22 * (-2.f * nq.y) + dr02 * nq.w);
  float dqz = 2.f * (dr00 * (-2.f * nq.z) + dr10 * nq.w + dr20 * nq.x + dr01 * (-nq.w) +
                     dr11 * (-2.f * nq.z) + dr12 * nq.y + dr21 * nq.y + dr02 * nq.x);
  float dot = dqw * nq.w + dqx * nq.x + dqy * nq.y + dqz * nq.z;
  d[3] = nq.inv_norm * (dqw - dot * nq.w);
  d[4] = nq.inv_norm * (dqx - dot * nq.x);
  d[5] = nq.inv_norm * (dqy - dot * nq.y);
  d[6] = nq.inv_norm * (dqz - dot * nq.z);
}

// VEC consecutive values of a row, loaded and stored as one (VEC x sizeof(T) bytes,
// aligned to that).
template <int VEC>
__device__ __forceinline__ void load_row(const float* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
    v[0] = *p;
  }
}
template <int VEC>
__device__ __forceinline__ void load_row(const __nv_bfloat16* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(q.x << 16), v[1] = __uint_as_float(q.x & 0xffff0000u);
    v[2] = __uint_as_float(q.y << 16), v[3] = __uint_as_float(q.y & 0xffff0000u);
  } else {
    v[0] = __bfloat162float(*p);
  }
}
template <int VEC>
__device__ __forceinline__ void store_row(float* p, const float (&v)[VEC]) {
  if constexpr (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else *p = v[0];
}
template <int VEC>
__device__ __forceinline__ void store_row(__nv_bfloat16* p, const __nv_bfloat16 (&v)[VEC]) {
  if constexpr (VEC == 4) {
    auto pair = [](__nv_bfloat16 a, __nv_bfloat16 b) {
      return (uint32_t)__bfloat16_as_ushort(a) | (uint32_t)__bfloat16_as_ushort(b) << 16;
    };
    *reinterpret_cast<uint2*>(p) = make_uint2(pair(v[0], v[1]), pair(v[2], v[3]));
  } else {
    *p = v[0];
  }
}
__device__ __forceinline__ float moment_of(const float*, float x, uint32_t) { return x; }
__device__ __forceinline__ __nv_bfloat16 moment_of(const __nv_bfloat16*, float x, uint32_t r) {
  return bf16_stochastic(x, r);
}

// Gradients of a CTA's splats (read four at a time): of the 14 scalar fields, and the
// factors of the SH rest rows.
template <bool kSh>
struct __align__(16) GradRows {
  float g[14][kThreads];
  float dc[kSh ? 3 : 1][kThreads];  // dL/d(colour), gated by the clamp
  float y[kSh ? 15 : 1][kThreads];  // basis values
};

// Adam on every field of the CTA's splats [first, first + count) (adam.cu:12-37; group
// learning rates of registerGaussian3DGroups, gaussian3d_adam.h:27-55).  The SoA is one
// [14 + 3 nb][n] array: a row is `count` consecutive values, of which the threads
// take VEC each, with several rows in flight.  Bound by HBM: a thread that walked
// the rows of its own splat with four-byte accesses and one band ahead reached 3.3
// TB/s on a million SH-3 splats (0.464 ms).  In BF16 storage the render copy of every
// field but the position follows its master.
template <typename T, bool kSh, int VEC>
__device__ __forceinline__ void adam_rows(float* __restrict__ P, T* __restrict__ R,
                                          T* __restrict__ M, T* __restrict__ V,
                                          float* __restrict__ G, const GradRows<kSh>& sg, int nb,
                                          int n, int first, int count, uint32_t salt,
                                          const Lrs& lr, float b1, float b2, float eps, float bc1,
                                          float bc2) {
  constexpr bool kBf16 = sizeof(T) == 2;
  constexpr int kGroups = kThreads / VEC;       // groups of VEC splats in a row
  constexpr int kStep = kThreads / kGroups;     // rows the CTA works on at a time
  constexpr int kRows = VEC == 4 ? (kSh ? 3 : 4) : 5;  // rows of a thread in flight
  const int l = (threadIdx.x % kGroups) * VEC;  // first splat of this thread's group
  if (l >= count) return;                       // count is a multiple of VEC
  const int rows = 14 + (kSh ? 3 * nb : 0);
  for (int r0 = threadIdx.x / kGroups; r0 < rows; r0 += kStep * kRows) {
    float p[kRows][VEC], m[kRows][VEC], v[kRows][VEC];
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int r = r0 + u * kStep;
      if (r >= rows) continue;
      const int64_t at = (int64_t)r * n + first + l;
      load_row<VEC>(P + at, p[u]);
      load_row<VEC>(M + at, m[u]);
      load_row<VEC>(V + at, v[u]);
    }
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
      const int r = r0 + u * kStep;
      if (r >= rows) continue;
      const int64_t at = (int64_t)r * n + first + l;
      float g[VEC];
      float rate;
      uint32_t field = (uint32_t)r, k = (uint32_t)(first + l);  // element k of the field
      if (!kSh || r < 14) {
        load_row<VEC>(&sg.g[r][l], g);
        rate = r < 3 ? lr.pos : r < 6 ? lr.scale : r < 10 ? lr.rot : r < 13 ? lr.sh_dc
                                                                           : lr.opacity;
      } else {
        const int c = (r - 14) / nb, b = r - 14 - c * nb;
        float dc[VEC];
        load_row<VEC>(&sg.dc[c][l], dc);
        load_row<VEC>(&sg.y[b][l], g);
#pragma unroll
        for (int e = 0; e < VEC; ++e) g[e] *= dc[e];
        rate = lr.sh_rest;
        field = 16u + 3u * (uint32_t)b + (uint32_t)c;
        k += (uint32_t)b * (uint32_t)n;
      }
      T mo[VEC], vo[VEC], ro[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        adam1(p[u][e], m[u][e], v[u][e], g[e], rate, b1, b2, eps, bc1, bc2);
        // one hash per element: its low 16 bits round m, its high 16 bits round v
        const uint32_t hs =
            kBf16 ? mix32((k + e) * 0x9e3779b1u ^ salt ^ field * 0xc2b2ae35u) : 0u;
        mo[e] = moment_of((const T*)nullptr, m[u][e], hs);
        vo[e] = moment_of((const T*)nullptr, v[u][e], hs >> 16);
        if constexpr (kBf16) ro[e] = __float2bfloat16_rn(p[u][e]);
      }
      store_row<VEC>(P + at, p[u]);
      store_row<VEC>(M + at, mo);
      store_row<VEC>(V + at, vo);
      if constexpr (kBf16) {
        if (r >= 3) store_row<VEC>(R + at, ro);
      }
      if (G) store_row<VEC>(G + at, g);
    }
  }
}

// Backward of one step and Adam.  P holds the FP32 masters (updated in
// place), R the attributes the forward rendered (P itself in FP32 storage; in
// BF16 storage the render copy, rewritten from the updated masters), M and V
// the moments in the storage type; each is one [14 + 3 nb][n] array.  kSh: the splats
// have SH rest rows.
template <typename T, bool kSh, bool kBatch = false>
__global__ void __launch_bounds__(kThreads, DS_ADAM_BLOCKS)
    fit_backward_adam_kernel(ds_gaussian3d P, Soa<T> R, Soa<T> M, Soa<T> V, ds_gaussian3d G,
                             int keep_grads, int exact, int degree, const Camera* __restrict__ camp,
                             const float* __restrict__ g2sum, GradSegments seg,
                             const float4* __restrict__ rec_c,
                             const float2* __restrict__ bcp,
                             const DevScalars* __restrict__ sc, Lrs lr, AdamHyper h,
                             const uint16_t* __restrict__ inst_of_splat = nullptr,
                             const uint32_t* __restrict__ visible = nullptr,
                             float* __restrict__ grad_accum = nullptr,
                             uint32_t* __restrict__ grad_count = nullptr) {
  pdl_wait();
  constexpr bool kBf16 = sizeof(T) == 2;
  __shared__ Mat4 sP;
  __shared__ float sCam[3];
  if (!kBatch) {
    if (threadIdx.x < 16) sP.m[threadIdx.x] = camp->pv[threadIdx.x];
    if (threadIdx.x < 3) sCam[threadIdx.x] = camp->cam[threadIdx.x];
  }
  __syncthreads();
  const int n = P.count;
  const int first = blockIdx.x * kThreads;
  const int i = first + threadIdx.x;
  const float2 bc = *bcp;
  const uint32_t salt = kBf16 ? sc->step * 0x85ebca6bu : 0u;
  __shared__ GradRows<kSh> sg;
  if (i < n) {
    const Camera* cam_i = kBatch ? camp + inst_of_splat[i] : camp;
    const Mat4& PV = kBatch ? *reinterpret_cast<const Mat4*>(cam_i->pv) : sP;
    const float* eye = kBatch ? cam_i->cam : sCam;

    // 1) Splat2D gradient = sum of this splat's per-tile records: summed here in
    // record order when it has at most kSerialRecords tiles, else read from the
    // long-segment reduction (segment_reduce_long_kernel).
    float g2[9];
    {
      const uint32_t c = seg.counts[i];
      unsigned long long s0 = 0, e0 = 0;
      if (c) {
        s0 = seg.start[i];
        e0 = s0 + c;
        if (e0 > seg.cap) e0 = seg.cap;
      }
      if (c > kSerialRecords) {
#pragma unroll
        for (int k = 0; k < 9; ++k) g2[k] = g2sum[(size_t)k * n + i];
      } else {
#pragma unroll
        for (int k = 0; k < 9; ++k) g2[k] = 0.f;
        if (e0 > s0) {
          // records of the tiles whose list ends (for compositing) before this
          // splat were not written: skip them
          const ushort4 rc = seg.rect[i];
          const uint32_t w = (uint32_t)(rc.y - rc.x + 1);
          uint32_t row0, pitch;
          seg_origin(seg, (uint32_t)i, rc, row0, pitch);
          const unsigned long long key = seg_key(seg, (uint32_t)i);
          uint32_t tx = 0, trow = row0;
          for (unsigned long long q = s0; q < e0; ++q) {
            if (key < seg.tile_bound[trow + tx]) {
              const float* r = seg.rec + q * 9;
#pragma unroll
              for (int k = 0; k < 9; ++k) g2[k] += r[k];
            }
            if (++tx == w) {
              tx = 0;
              trow += pitch;
            }
          }
        }
      }
    }
    // g2 = {color r, g, b, ndc x, ndc y, cov2 xx, xy, yy, opacity}
    if (grad_accum && visible[i] > 0u) {
      // densification statistics: norm of the NDC position gradient, steps visible
      grad_accum[i] += sqrtf(g2[3] * g2[3] + g2[4] * g2[4]);
      grad_count[i] += 1u;
    }

    // 2) projection backward (persp_project_layer.cu:173-267)
    const float px = P.pos_x[i], py = P.pos_y[i], pz = P.pos_z[i];
    const float rw = ldv(R.rot_w[i]), rx = ldv(R.rot_x[i]), ry = ldv(R.rot_y[i]),
                rz = ldv(R.rot_z[i]);
    const float lsx = ldv(R.scale_x[i]), lsy = ldv(R.scale_y[i]), lsz = ldv(R.scale_z[i]);
    float clip_x, clip_y, clip_z, clip_w;
    project_jacobian(PV, px, py, pz, clip_x, clip_y, clip_z, clip_w);
    float gpos[3] = {0.f, 0.f, 0.f};
    float gcov[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float gcol[3] = {0.f, 0.f, 0.f};
    float gop = 0.f;
    if (clip_w > 0.f) {
      const float inv_w = 1.f / clip_w;
      const float inv_w2 = inv_w * inv_w;
      Jac2 J = jacobian(PV, clip_x, clip_y, clip_w, inv_w2);
      const float j00 = J.j00, j01 = J.j01, j02 = J.j02, j10 = J.j10, j11 = J.j11, j12 = J.j12;
      const float dcxx = g2[5], dcxy = g2[6], dcyy = g2[7];
      const float hdxy = 0.5f * dcxy;
      gcov[0] = j00 * j00 * dcxx + j00 * j10 * dcxy + j10 * j10 * dcyy;
      gcov[1] = j00 * j01 * dcxx + hdxy * (j00 * j11 + j10 * j01) + j10 * j11 * dcyy;
      gcov[2] = j00 * j02 * dcxx + hdxy * (j00 * j12 + j10 * j02) + j10 * j12 * dcyy;
      gcov[3] = j01 * j01 * dcxx + j01 * j11 * dcxy + j11 * j11 * dcyy;
      gcov[4] = j01 * j02 * dcxx + hdxy * (j01 * j12 + j11 * j02) + j11 * j12 * dcyy;
      gcov[5] = j02 * j02 * dcxx + j02 * j12 * dcxy + j12 * j12 * dcyy;
      gpos[0] = g2[3] * j00 + g2[4] * j10;
      gpos[1] = g2[3] * j01 + g2[4] * j11;
      gpos[2] = g2[3] * j02 + g2[4] * j12;
      gcol[0] = g2[0];
      gcol[1] = g2[1];
      gcol[2] = g2[2];
      gop = g2[8];
      if (exact) {
        UnitQuat q = unit_quat(rw, rx, ry, rz);
        Rot3 Rm = rot_from_quat(q.w, q.x, q.y, q.z);
        Cov3 c3 = cov3_from(Rm, expf(lsx), expf(lsy), expf(lsz));
        float3 e = jacobian_position_grad(PV, J, clip_w, dcxx, hdxy, dcyy, c3.xx, c3.xy, c3.xz,
                                          c3.yy, c3.yz, c3.zz);
        gpos[0] += e.x;
        gpos[1] += e.y;
        gpos[2] += e.z;
      }
    }

    // 3) activation backward (gauss_activ_layer.cu:254-406)
    float d[7];
    cov_backward(rw, rx, ry, rz, lsx, lsy, lsz, gcov[0], gcov[1], gcov[2], gcov[3], gcov[4],
                 gcov[5], d);
    // The forward's colours decide the clamp's gate; a splat in no tile has none, and
    // no gradient.
    const bool seen = seg.counts[i] > 0u;
    const float4 col = seen ? rec_c[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float dR = (col.x > 0.f && col.x < 1.f) ? gcol[0] : 0.f;
    const float dG = (col.y > 0.f && col.y < 1.f) ? gcol[1] : 0.f;
    const float dB = (col.z > 0.f && col.z < 1.f) ? gcol[2] : 0.f;
    if constexpr (kSh) {
      float y[15];
#pragma unroll
      for (int b = 0; b < 15; ++b) y[b] = 0.f;
      sh_basis(degree, dir_to_camera(eye[0], eye[1], eye[2], px, py, pz), y);
#pragma unroll
      for (int b = 0; b < 15; ++b) sg.y[b][threadIdx.x] = y[b];
      sg.dc[0][threadIdx.x] = dR;
      sg.dc[1][threadIdx.x] = dG;
      sg.dc[2][threadIdx.x] = dB;
    }
    const float logit = ldv(R.logit_opacity[i]);
    const float s = 1.f / (1.f + expf(-logit));
    const float glogit = gop * s * (1.f - s);

    const float g[14] = {gpos[0], gpos[1], gpos[2], d[0],     d[1],     d[2],     d[3],
                         d[4],    d[5],    d[6],    dR * kC0, dG * kC0, dB * kC0, glogit};
#pragma unroll
    for (int k = 0; k < 14; ++k) sg.g[k][threadIdx.x] = g[k];
  }
  __syncthreads();

  // 4) Adam.  Rows of n values: groups of four stay aligned when n is a multiple of 4.
  const int count = min(kThreads, n - first), nb = P.sh_num_bands;
  float* grads = keep_grads ? G.pos_x : nullptr;
  if ((n & 3) == 0)
    adam_rows<T, kSh, 4>(P.pos_x, R.pos_x, M.pos_x, V.pos_x, grads, sg, nb, n, first, count, salt,
                         lr, h.b1, h.b2, h.eps, bc.x, bc.y);
  else
    adam_rows<T, kSh, 1>(P.pos_x, R.pos_x, M.pos_x, V.pos_x, grads, sg, nb, n, first, count, salt,
                         lr, h.b1, h.b2, h.eps, bc.x, bc.y);
}

// Bias-correction table on the device: bc_k(t) = 1 / (1 - powf(beta_k, t)),
// computed on the host like the reference (adam.cu:61-62), up to the step at
// which both corrections reach 1.0f (step_begin_kernel uses 1.0f past it).
inline int make_bc_table(float beta1, float beta2, float2** table, int* len) {
  std::vector<float2> tab;
  for (int t = 1; t <= kBcTableMax; ++t) {
    const float p1 = powf(beta1, (float)t), p2 = powf(beta2, (float)t);
    const float bc1 = 1.f / (1.f - p1), bc2 = 1.f / (1.f - p2);
    tab.push_back(make_float2(bc1, bc2));
    if (bc1 == 1.f && bc2 == 1.f) break;
  }
  *len = (int)tab.size();
  DS_CUDA(cudaMalloc(table, tab.size() * sizeof(float2)));
  DS_CUDA(cudaMemcpy(*table, tab.data(), tab.size() * sizeof(float2), cudaMemcpyHostToDevice));
  return DS_OK;
}

}  // namespace

}  // namespace ds
