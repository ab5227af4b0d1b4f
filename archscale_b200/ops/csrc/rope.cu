// Fused per-head RMSNorm (QK-norm) + rotary embedding (NeoX halves) for q:[N,H,D] and k:[N,G,D], bf16.
// One warp per token (all its heads, two at a time); D ∈ {64, 128}.  Statistics and rotation in fp32.
// Backward undoes the rotation (conjugate), then applies the RMSNorm backward; the weight gradient
// is accumulated per warp in registers, per CTA in shared memory (warps in a fixed order) and written as per-CTA partials
// (deterministic two-stage reduction).
#include "sm100.cuh"
#include "api.h"

namespace b200 {

template <int EPL> __device__ __forceinline__ void ld_row(const __nv_bfloat16* p, float (&v)[EPL]);
template <> __device__ __forceinline__ void ld_row<4>(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <> __device__ __forceinline__ void ld_row<2>(const __nv_bfloat16* p, float (&v)[2]) {
  const float2 a = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p));
  v[0] = a.x; v[1] = a.y;
}
template <int EPL> __device__ __forceinline__ void st_row(__nv_bfloat16* p, const float (&v)[EPL]);
template <> __device__ __forceinline__ void st_row<4>(__nv_bfloat16* p, const float (&v)[4]) {
  uint2 u; u.x = pack_bf16x2(v[0], v[1]); u.y = pack_bf16x2(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = u;
}
template <> __device__ __forceinline__ void st_row<2>(__nv_bfloat16* p, const float (&v)[2]) {
  *reinterpret_cast<uint32_t*>(p) = pack_bf16x2(v[0], v[1]);
}
// EPL packed elements as loaded (half the registers of their fp32 values), and the conversion
template <int EPL> struct Raw { uint32_t w[EPL / 2]; };
__device__ __forceinline__ void ld_raw(const __nv_bfloat16* p, Raw<4>& r) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  r.w[0] = u.x; r.w[1] = u.y;
}
__device__ __forceinline__ void ld_raw(const __nv_bfloat16* p, Raw<2>& r) { r.w[0] = *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ void st_raw(__nv_bfloat16* p, const Raw<4>& r) { *reinterpret_cast<uint2*>(p) = make_uint2(r.w[0], r.w[1]); }
__device__ __forceinline__ void st_raw(__nv_bfloat16* p, const Raw<2>& r) { *reinterpret_cast<uint32_t*>(p) = r.w[0]; }
template <int EPL> __device__ __forceinline__ void expand(const Raw<EPL>& r, float (&v)[EPL]) {
#pragma unroll
  for (int i = 0; i < EPL / 2; ++i) { const float2 f = unpack_bf16x2(r.w[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
template <typename TW> __device__ __forceinline__ float ldw(const TW* w, int i);
template <> __device__ __forceinline__ float ldw<float>(const float* w, int i) { return w[i]; }
template <> __device__ __forceinline__ float ldw<__nv_bfloat16>(const __nv_bfloat16* w, int i) { return __bfloat162float(w[i]); }

// Sum over the 16 lanes of a half warp.
__device__ __forceinline__ float half_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per TOKEN, half a warp per head: a lane owns EPL elements of the head's first half and the EPL elements they are
// rotated with, so the rotation needs no exchange and a row sum takes four shuffles for two heads.  (With a row over the whole
// warp, five shuffles for the sum and EPL for the rotation per head kept the kernels at a third of the copy bandwidth: B8 T4096
// H16 G4 D128 forward + value copy 0.105 -> 0.081 ms, backward 0.241 -> 0.138; B1 T8192 H40 G20 D64 0.064 / 0.126 -> 0.050 /
// 0.083.)  cos / sin and the norm gains are loaded once and serve all heads of the token, which are walked 2·ROPE_U at a time so
// that as many rows are in flight per warp (ROPE_U 4 needs 128 registers backward: 0.138 ms too, 0.099 against 0.091 at H8 G2).
constexpr int ROPE_U = 2;

// Where the heads of a token sit.  Dense rows [tokens, heads, D] are q_hpg = H, k_gs = D; the output of a fused QKV projection
// laid out per key/value group as [group][q_per_kv query heads, key head, value head][D] is q_hpg = q_per_kv and
// q_gs = k_gs = (q_per_kv + 2)·D with the key / value base pointers advanced to their slot of group 0.
struct QKLayout {
  long long q_ts, k_ts;      // token strides (elements)
  long long q_gs, k_gs;      // stride between groups of query heads / between key (value) heads
  int q_hpg;                 // query heads per group
};

// Copies the G value rows of every token between two layouts (token and head strides): a pass of its own after the loop over
// tokens, eight rows in flight per warp (inside that loop it is one more load-to-store wait per token: backward 0.171 against
// 0.126 ms without any copy at B8 T4096 H16 G4 D128).
template <int EPL>
__device__ __forceinline__ void copy_value_rows(const __nv_bfloat16* __restrict__ src, long long s_ts, long long s_hs,
                                                __nv_bfloat16* __restrict__ dst, long long d_ts, long long d_hs, int64_t n_tokens, int G,
                                                int64_t warp_global, int64_t n_warps, int lane) {
  const int64_t rows = n_tokens * G;
  for (int64_t r0 = warp_global * 8; r0 < rows; r0 += n_warps * 8) {
    Raw<EPL> x[8];
    int64_t tok = r0 / G;
    int g = static_cast<int>(r0 - tok * G);
    const int64_t tok0 = tok;
    const int g0 = g;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (r0 + u < rows) ld_raw(src + tok * s_ts + g * s_hs + lane * EPL, x[u]);
      if (++g == G) { g = 0; ++tok; }
    }
    tok = tok0; g = g0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (r0 + u < rows) st_raw(dst + tok * d_ts + g * d_hs + lane * EPL, x[u]);
      if (++g == G) { g = 0; ++tok; }
    }
  }
}

// The `per` head rows at src (stride hstride), normalised (w: the gains of this lane's elements, first half then second, or
// has_w false) and rotated (rot), to dense rows at dst.  src / dst point at this lane's first element of head 0.
template <int EPL>
__device__ __forceinline__ void fwd_heads(const __nv_bfloat16* src, long long hstride, __nv_bfloat16* dst, float* rstd, int per,
                                          const float (&w)[2 * EPL], bool has_w, bool rot, const float (&cs)[EPL], const float (&sn)[EPL],
                                          int lane, float eps) {
  constexpr int D = EPL * 32;
  const int sub = lane >> 4;
  for (int h0 = 0; h0 < per; h0 += 2 * ROPE_U) {
    Raw<EPL> rlo[ROPE_U], rhi[ROPE_U];
#pragma unroll
    for (int u = 0; u < ROPE_U; ++u) {
      const int h = min(h0 + 2 * u + sub, per - 1);            // past the last head: loaded again, not stored
      ld_raw(src + h * hstride, rlo[u]);
      ld_raw(src + h * hstride + D / 2, rhi[u]);
    }
#pragma unroll
    for (int u = 0; u < ROPE_U; ++u) {
      const int h = h0 + 2 * u + sub;
      float lo[EPL], hi[EPL];
      expand<EPL>(rlo[u], lo);
      expand<EPL>(rhi[u], hi);
      if (has_w) {
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < EPL; ++e) ss += lo[e] * lo[e] + hi[e] * hi[e];
        ss = half_sum(ss);
        const float rs = rsqrtf(ss / D + eps);
        if ((lane & 15) == 0 && h < per) rstd[h] = rs;
#pragma unroll
        for (int e = 0; e < EPL; ++e) { lo[e] = lo[e] * rs * w[e]; hi[e] = hi[e] * rs * w[EPL + e]; }
      }
      if (rot) {
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          const float a = lo[e], b = hi[e];
          lo[e] = a * cs[e] - b * sn[e];
          hi[e] = a * sn[e] + b * cs[e];
        }
      }
      if (h < per) {
        st_row<EPL>(dst + h * D, lo);
        st_row<EPL>(dst + h * D + D / 2, hi);
      }
    }
  }
}

// GROUPED: the per-group layout (else every head of a part is D elements after the previous one: dense rows or the blocked
// fused projection, for which the loops below reduce to the plain walk over heads).  WITH_V: also copy the value heads.
template <int EPL, typename TW, bool GROUPED, bool WITH_V>
__global__ void __launch_bounds__(256, 4) qknorm_rope_fwd_kernel(
    const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const TW* __restrict__ qw,
    const TW* __restrict__ kw, const __nv_bfloat16* __restrict__ cosb, const __nv_bfloat16* __restrict__ sinb,
    __nv_bfloat16* __restrict__ qo, __nv_bfloat16* __restrict__ ko, float* __restrict__ q_rstd,
    float* __restrict__ k_rstd, int64_t n_tokens, int T, int H, int G, float eps, const QKLayout L,
    const __nv_bfloat16* __restrict__ v, __nv_bfloat16* __restrict__ vo) {
  constexpr int D = EPL * 32;
  const int lane = threadIdx.x & 31;
  const int64_t warp_global = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int ci = (lane & 15) * EPL;                 // this lane's first element of a head row
  float wq[2 * EPL], wk[2 * EPL];
#pragma unroll
  for (int e = 0; e < 2 * EPL; ++e) {
    const int c = ci + (e % EPL) + (e / EPL) * (D / 2);
    wq[e] = qw ? ldw<TW>(qw, c) : 1.f;
    wk[e] = kw ? ldw<TW>(kw, c) : 1.f;
  }
  for (int64_t tok = warp_global; tok < n_tokens; tok += n_warps) {
    float cs[EPL], sn[EPL];
    if (cosb) {
      const size_t co = static_cast<size_t>(tok % T) * (D / 2) + ci;
      ld_row<EPL>(cosb + co, cs);
      ld_row<EPL>(sinb + co, sn);
    }
    // inputs may be column slices of a wider (fused projection) matrix, dense or interleaved per group: see QKLayout.
    // Query heads are walked group by group (one group of H heads for dense rows), so no head index is ever divided.
    const int per = GROUPED ? L.q_hpg : H, n_groups = GROUPED ? H / L.q_hpg : 1;
    for (int grp = 0; grp < n_groups; ++grp)
      fwd_heads<EPL>(q + tok * L.q_ts + (GROUPED ? grp * L.q_gs : 0) + ci, D, qo + (tok * H + grp * per) * D + ci,
                     q_rstd + tok * H + grp * per, per, wq, qw != nullptr, cosb != nullptr, cs, sn, lane, eps);
    fwd_heads<EPL>(k + tok * L.k_ts + ci, GROUPED ? L.k_gs : D, ko + tok * G * D + ci, k_rstd + tok * G, G, wk, kw != nullptr,
                   cosb != nullptr, cs, sn, lane, eps);
  }
  if (WITH_V)                                       // the value heads, copied out of the fused projection into dense rows
    copy_value_rows<EPL>(v, L.k_ts, GROUPED ? L.k_gs : D, vo, static_cast<long long>(G) * D, D, n_tokens, G, warp_global, n_warps, lane);
}

// Backward of fwd_heads: rotate back, then the RMSNorm backward; the gain gradient is added into dw.
template <int EPL>
__device__ __forceinline__ void bwd_heads(const __nv_bfloat16* gsrc, const __nv_bfloat16* xsrc, long long hstride, __nv_bfloat16* gdst,
                                          long long o_hstride, const float* rstd, int per, const float (&w)[2 * EPL],
                                          float (&dw)[2 * EPL], bool has_w, bool rot, const float (&cs)[EPL], const float (&sn)[EPL],
                                          int lane) {
  constexpr int D = EPL * 32;
  const int sub = lane >> 4;
  for (int h0 = 0; h0 < per; h0 += 2 * ROPE_U) {
    Raw<EPL> rgl[ROPE_U], rgh[ROPE_U], rxl[ROPE_U], rxh[ROPE_U];
    float rsv[ROPE_U];
#pragma unroll
    for (int u = 0; u < ROPE_U; ++u) {
      const int h = h0 + 2 * u + sub;
      rgl[u] = rgh[u] = rxl[u] = rxh[u] = Raw<EPL>{};            // past the last head: zeros, which add nothing to the gain gradient
      rsv[u] = 0.f;
      if (h < per) {
        ld_raw(gsrc + h * D, rgl[u]);
        ld_raw(gsrc + h * D + D / 2, rgh[u]);
        if (has_w) {
          ld_raw(xsrc + h * hstride, rxl[u]);
          ld_raw(xsrc + h * hstride + D / 2, rxh[u]);
          rsv[u] = rstd[h];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < ROPE_U; ++u) {
      const int h = h0 + 2 * u + sub;
      float glo[EPL], ghi[EPL];
      expand<EPL>(rgl[u], glo);
      expand<EPL>(rgh[u], ghi);
      if (rot) {
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          const float a = glo[e], b = ghi[e];
          glo[e] = a * cs[e] + b * sn[e];
          ghi[e] = b * cs[e] - a * sn[e];
        }
      }
      if (has_w) {
        float xlo[EPL], xhi[EPL], dot = 0.f;
        expand<EPL>(rxl[u], xlo);
        expand<EPL>(rxh[u], xhi);
        const float rs = rsv[u];
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          dw[e] += glo[e] * xlo[e] * rs;
          dw[EPL + e] += ghi[e] * xhi[e] * rs;
          glo[e] *= w[e];
          ghi[e] *= w[EPL + e];
          dot += glo[e] * xlo[e] + ghi[e] * xhi[e];
        }
        dot = half_sum(dot);
        const float c1 = dot * rs * rs * rs / D;
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
          glo[e] = glo[e] * rs - xlo[e] * c1;
          ghi[e] = ghi[e] * rs - xhi[e] * c1;
        }
      }
      if (h < per) {
        st_row<EPL>(gdst + h * o_hstride, glo);
        st_row<EPL>(gdst + h * o_hstride + D / 2, ghi);
      }
    }
  }
}

template <int EPL, typename TW, bool GROUPED, bool WITH_V>
__global__ void __launch_bounds__(256, 3) qknorm_rope_bwd_kernel(
    const __nv_bfloat16* __restrict__ dqo, const __nv_bfloat16* __restrict__ dko, const __nv_bfloat16* __restrict__ q,
    const __nv_bfloat16* __restrict__ k, const TW* __restrict__ qw, const TW* __restrict__ kw,
    const __nv_bfloat16* __restrict__ cosb, const __nv_bfloat16* __restrict__ sinb, const float* __restrict__ q_rstd,
    const float* __restrict__ k_rstd, __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk,
    float* __restrict__ dw_partial /* [grid, 2, D] */, int64_t n_tokens, int T, int H, int G, const QKLayout L,
    const QKLayout LO /* layout of dq, dk (and dv_dst) */, const __nv_bfloat16* __restrict__ dvo, __nv_bfloat16* __restrict__ dv_dst) {
  constexpr int D = EPL * 32;
  __shared__ float dw_s[8][2][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t warp_global = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int ci = (lane & 15) * EPL;
  float dwq[2 * EPL], dwk[2 * EPL], wq[2 * EPL], wk[2 * EPL];
#pragma unroll
  for (int e = 0; e < 2 * EPL; ++e) {
    const int c = ci + (e % EPL) + (e / EPL) * (D / 2);
    dwq[e] = dwk[e] = 0.f;
    wq[e] = qw ? ldw<TW>(qw, c) : 1.f;
    wk[e] = kw ? ldw<TW>(kw, c) : 1.f;
  }
  for (int64_t tok = warp_global; tok < n_tokens; tok += n_warps) {
    float cs[EPL], sn[EPL];
    if (cosb) {
      const size_t co = static_cast<size_t>(tok % T) * (D / 2) + ci;
      ld_row<EPL>(cosb + co, cs);
      ld_row<EPL>(sinb + co, sn);
    }
    const int per = GROUPED ? L.q_hpg : H, n_groups = GROUPED ? H / L.q_hpg : 1;      // LO: same grouping
    for (int grp = 0; grp < n_groups; ++grp)
      bwd_heads<EPL>(dqo + (tok * H + grp * per) * D + ci, q + tok * L.q_ts + (GROUPED ? grp * L.q_gs : 0) + ci, D,
                     dq + tok * LO.q_ts + (GROUPED ? grp * LO.q_gs : 0) + ci, D, q_rstd + tok * H + grp * per, per, wq, dwq,
                     qw != nullptr, cosb != nullptr, cs, sn, lane);
    bwd_heads<EPL>(dko + tok * G * D + ci, k + tok * L.k_ts + ci, GROUPED ? L.k_gs : D, dk + tok * LO.k_ts + ci, GROUPED ? LO.k_gs : D,
                   k_rstd + tok * G, G, wk, dwk, kw != nullptr, cosb != nullptr, cs, sn, lane);
  }
  if (WITH_V)                                       // the value gradient takes its slot of the fused-projection gradient
    copy_value_rows<EPL>(dvo, static_cast<long long>(G) * D, D, dv_dst, LO.k_ts, GROUPED ? LO.k_gs : D, n_tokens, G, warp_global,
                         n_warps, lane);
  if (qw) {                                         // the two halves of a warp, then the warps in order
#pragma unroll
    for (int e = 0; e < 2 * EPL; ++e) {
      const float a = dwq[e] + __shfl_xor_sync(0xffffffffu, dwq[e], 16), b = dwk[e] + __shfl_xor_sync(0xffffffffu, dwk[e], 16);
      const int c = ci + (e % EPL) + (e / EPL) * (D / 2);
      if (lane < 16) { dw_s[warp][0][c] = a; dw_s[warp][1][c] = b; }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += (&dw_s[w][0][0])[i];
      dw_partial[static_cast<size_t>(blockIdx.x) * 2 * D + i] = t;
    }
  }
}

// partials are [n, 2·D]: columns 0..D−1 belong to dqw, D..2D−1 to dkw
__global__ void __launch_bounds__(1024) qk_dw_reduce_kernel(const float* __restrict__ part, float* __restrict__ dqw, float* __restrict__ dkw, int n, int D) {
  const float t = column_sum_block(part, n, 2 * D);
  const int c = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x < 32 && c < 2 * D) { if (c < D) dqw[c] = t; else dkw[c - D] = t; }
}

constexpr int kRopeGrid = 148 * 8;

}  // namespace b200

using namespace b200;
typedef __nv_bfloat16 bf16;

extern "C" int b200_qknorm_rope_grid() { return kRopeGrid; }

// q_hpg / gs: see QKLayout (q_hpg = H, gs = D for dense rows).  v / vo: optional value heads (k's layout) copied to dense rows.
extern "C" int b200_qknorm_rope_fwd_ex(const void* q, const void* k, const void* v, const void* qw, const void* kw, int w_dtype,
                                       const void* cos, const void* sin, void* qo, void* ko, void* vo, float* q_rstd, float* k_rstd,
                                       int64_t n_tokens, int T, int H, int G, int D, float eps, int64_t q_ts, int64_t k_ts,
                                       int q_hpg, int64_t q_gs, int64_t k_gs, cudaStream_t st) {
  if (n_tokens == 0) return 0;
  if (q_hpg <= 0 || H % q_hpg) return -1;
  const QKLayout L{q_ts, k_ts, q_gs, k_gs, q_hpg};
  const bool grouped = q_hpg != H, with_v = v != nullptr;
  if (!grouped && k_gs != D) return -1;
#define LAUNCH2(EPL, TW, GR, WV)                                                                                      \
  qknorm_rope_fwd_kernel<EPL, TW, GR, WV><<<kRopeGrid, 256, 0, st>>>((const bf16*)q, (const bf16*)k, (const TW*)qw, (const TW*)kw, \
                                                             (const bf16*)cos, (const bf16*)sin, (bf16*)qo, (bf16*)ko,  \
                                                             q_rstd, k_rstd, n_tokens, T, H, G, eps, L, (const bf16*)v, (bf16*)vo)
#define LAUNCH(EPL, TW)                                                        \
  do {                                                                         \
    if (grouped) { if (with_v) LAUNCH2(EPL, TW, true, true); else LAUNCH2(EPL, TW, true, false); } \
    else { if (with_v) LAUNCH2(EPL, TW, false, true); else LAUNCH2(EPL, TW, false, false); }       \
  } while (0)
  if (D == 128) { if (w_dtype == 1) LAUNCH(4, bf16); else LAUNCH(4, float); }
  else if (D == 64) { if (w_dtype == 1) LAUNCH(2, bf16); else LAUNCH(2, float); }
  else return -1;
#undef LAUNCH
#undef LAUNCH2
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

extern "C" int b200_qknorm_rope_fwd(const void* q, const void* k, const void* qw, const void* kw, int w_dtype,
                                    const void* cos, const void* sin, void* qo, void* ko, float* q_rstd, float* k_rstd,
                                    int64_t n_tokens, int T, int H, int G, int D, float eps, int64_t q_ts, int64_t k_ts, cudaStream_t st) {
  return b200_qknorm_rope_fwd_ex(q, k, nullptr, qw, kw, w_dtype, cos, sin, qo, ko, nullptr, q_rstd, k_rstd, n_tokens, T, H, G, D, eps,
                                 q_ts, k_ts, H, 0, D, st);
}

// dq / dk are written with the layout (o_q_ts, o_k_ts, o_q_hpg, o_q_gs, o_k_gs); dvo (dense) is copied to dv_dst in k's output layout.
extern "C" int b200_qknorm_rope_bwd_ex(const void* dqo, const void* dko, const void* dvo, const void* q, const void* k, const void* qw,
                                       const void* kw, int w_dtype, const void* cos, const void* sin, const float* q_rstd,
                                       const float* k_rstd, void* dq, void* dk, void* dv_dst, float* dqw, float* dkw,
                                       float* dw_partial, int64_t n_tokens, int T, int H, int G, int D, int64_t q_ts, int64_t k_ts,
                                       int q_hpg, int64_t q_gs, int64_t k_gs, int64_t o_q_ts, int64_t o_k_ts, int o_q_hpg,
                                       int64_t o_q_gs, int64_t o_k_gs, cudaStream_t st) {
  if (n_tokens == 0) return 0;
  if (q_hpg <= 0 || o_q_hpg != q_hpg || H % q_hpg) return -1;       // input and output share one grouping
  const QKLayout L{q_ts, k_ts, q_gs, k_gs, q_hpg}, LO{o_q_ts, o_k_ts, o_q_gs, o_k_gs, o_q_hpg};
  const bool grouped = q_hpg != H, with_v = dvo != nullptr;
  if (!grouped && (k_gs != D || o_k_gs != D)) return -1;
#define LAUNCH2(EPL, TW, GR, WV)                                                                                       \
  qknorm_rope_bwd_kernel<EPL, TW, GR, WV><<<kRopeGrid, 256, 0, st>>>((const bf16*)dqo, (const bf16*)dko, (const bf16*)q, (const bf16*)k, \
                                                             (const TW*)qw, (const TW*)kw, (const bf16*)cos, (const bf16*)sin,  \
                                                             q_rstd, k_rstd, (bf16*)dq, (bf16*)dk, dw_partial, n_tokens, T, H, G, L, LO, \
                                                             (const bf16*)dvo, (bf16*)dv_dst)
#define LAUNCH(EPL, TW)                                                        \
  do {                                                                         \
    if (grouped) { if (with_v) LAUNCH2(EPL, TW, true, true); else LAUNCH2(EPL, TW, true, false); } \
    else { if (with_v) LAUNCH2(EPL, TW, false, true); else LAUNCH2(EPL, TW, false, false); }       \
  } while (0)
  if (D == 128) { if (w_dtype == 1) LAUNCH(4, bf16); else LAUNCH(4, float); }
  else if (D == 64) { if (w_dtype == 1) LAUNCH(2, bf16); else LAUNCH(2, float); }
  else return -1;
#undef LAUNCH
#undef LAUNCH2
  if (qw) qk_dw_reduce_kernel<<<(2 * D + 31) / 32, 1024, 0, st>>>(dw_partial, dqw, dkw, kRopeGrid, D);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

extern "C" int b200_qknorm_rope_bwd(const void* dqo, const void* dko, const void* q, const void* k, const void* qw,
                                     const void* kw, int w_dtype, const void* cos, const void* sin, const float* q_rstd,
                                     const float* k_rstd, void* dq, void* dk, float* dqw, float* dkw, float* dw_partial,
                                     int64_t n_tokens, int T, int H, int G, int D, int64_t q_ts, int64_t k_ts, cudaStream_t st) {
  return b200_qknorm_rope_bwd_ex(dqo, dko, nullptr, q, k, qw, kw, w_dtype, cos, sin, q_rstd, k_rstd, dq, dk, nullptr, dqw, dkw,
                                 dw_partial, n_tokens, T, H, G, D, q_ts, k_ts, H, 0, D, static_cast<int64_t>(H) * D,
                                 static_cast<int64_t>(G) * D, H, 0, D, st);
}
