// Mamba-1 selective scan, forward and backward, on token-major activations (rows = tokens, channels contiguous).
//   dt_t = softplus(delta_t + bias),  h_t = exp(dt_t·A)·h_{t-1} + dt_t·B_t·u_t,  y_t = C_t·h_t + D·u_t  (·silu(z_t))
// with N = 16 states per channel and an optional per-token reset flag (start of a packed document: h_{t-1} := 0).
//
// Work decomposition: NS (2 or 4) states per thread, 16/NS threads per channel, 16 channels per CTA, time sequential inside
// the thread.  What bounds it is one exponential per (step, channel, state) on MUFU (B4 L4096 Di3968: 1.04e9 of them, 0.23 ms):
// everything else has to stay below that.  With one state per thread (what this file did before) every step cost four
// shared-memory loads, fifteen sixteenths of a shuffle and its selects per state.  Several states per thread share the loads of dt and dt·u, read B and C as vectors, do two states per instruction
// (fma.rn.f32x2) and add most of the sum over states in registers; the remaining 16/NS lanes use a reduce-scatter over 16/NS
// steps (lane q ends up with the total of step q).  Measured (L2 flushed, both trees on one box), one state -> several per thread, ms:
//   B4 L4096 Di3968   forward 1.17 -> 0.59   backward 3.89 -> 2.28        B1 L32768 Di3968  forward 4.05 -> 1.66   backward 8.44 -> 5.78
//   B8 L4096 Di4096   forward 2.07 -> 1.06   backward 7.29 -> 4.48        B1 L8192 Di5120   forward 1.15 -> 0.55   backward 3.70 -> 2.09
// (the B1 forwards with the time axis split, see b200_selective_scan_parts).
//
// The forward stages tiles of 64 steps through shared memory (the next tile's loads are in flight during the steps) and
// stores the state entering every 32-step half tile (fp32, L/32 × Di × 16).  The backward walks 32-step tiles in reverse,
// recomputes the 32 states from their checkpoint into registers (two states per thread: 64 registers) and runs the adjoint
//   G_t = C_t·dy'_t + a_{t+1}·G_{t+1}
// dB/dC (sums over channels) are reduced over the warp's 4 channels by shuffles and over the CTA's 4 warps in shared memory,
// written as per-CTA partial sums and summed over channel blocks by a second kernel (deterministic, no atomics).
#include <type_traits>
#include "sm100.cuh"
#include "api.h"

namespace b200 {

constexpr int SS_T = 64;    // steps per forward tile
constexpr int SS_TB = 32;   // steps per backward tile (= checkpoint interval)
constexpr int SS_C = 16;    // channels per CTA
constexpr int SS_N = 16;    // states per channel
constexpr int SS_YP = 24;   // row pitch of the per-step sums: 8-channel rows of neighbouring steps fall into different banks
constexpr float SS_LOG2E = 1.4426950408889634f;

template <typename T> __device__ __forceinline__ void st1(T* p, float v);
template <> __device__ __forceinline__ void st1<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void st1<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

// four neighbouring elements as they lie in memory; `vec`: the address is a multiple of their size
template <typename T> struct Raw4;
template <> struct Raw4<float> {
  float4 v;
  __device__ __forceinline__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void load(const float* p, bool vec) {
    if (vec) v = *reinterpret_cast<const float4*>(p);
    else v = make_float4(p[0], p[1], p[2], p[3]);
  }
  __device__ __forceinline__ float4 get() const { return v; }
};
template <> struct Raw4<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void zero() { v = make_uint2(0u, 0u); }
  __device__ __forceinline__ void load(const __nv_bfloat16* p, bool vec) {
    if (vec) { v = *reinterpret_cast<const uint2*>(p); return; }
    const unsigned short* s = reinterpret_cast<const unsigned short*>(p);
    v.x = s[0] | (static_cast<uint32_t>(s[1]) << 16);
    v.y = s[2] | (static_cast<uint32_t>(s[3]) << 16);
  }
  __device__ __forceinline__ float4 get() const {
    const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y);
    return make_float4(a.x, a.y, b.x, b.y);
  }
};
__device__ __forceinline__ void put4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void put4(__nv_bfloat16* p, float4 v) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}
// row stride and base of a [rows, 16·k] operand allow vector loads of four elements
template <typename T> __host__ __device__ __forceinline__ bool rows_vec4(const T* p, int stride) {
  return p == nullptr || (reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T)) == 0 && stride % 4 == 0);
}

__device__ __forceinline__ float ss_softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }
__device__ __forceinline__ float ss_sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }

// 2^x · h as (2^(x − cap) · h) · cap with cap = 2^min(x, 126): growing states (A·dt > 0) may gain more than the largest float over
// a part, and the product is still what the steps give: zero stays zero (not 0·inf), a small state stays finite.  For x ≤ 126
// the first factor is exactly one.
__device__ __forceinline__ float2 ss_exp2_cap(float2 x) { return make_float2(exp2f(fminf(x.x, 126.f)), exp2f(fminf(x.y, 126.f))); }
__device__ __forceinline__ float2 ss_exp2_mul(float2 x, float2 h) {
  return make_float2(exp2f(fminf(fmaxf(x.x - 126.f, 0.f), 126.f)) * h.x, exp2f(fminf(fmaxf(x.y - 126.f, 0.f), 126.f)) * h.y);
}

// v[s] (s = 0..W-1) summed over W neighbouring lanes (lane index q inside the group); lane q returns the total of step q.
template <int W>
__device__ __forceinline__ float lane_scatter_sum(float (&v)[W], int q) {
#pragma unroll
  for (int w = W / 2; w >= 1; w >>= 1) {
    const bool hi = (q & w) != 0;
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const float send = hi ? v[k] : v[k + w];
      const float keep = hi ? v[k + w] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return v[0];
}

// Time may be split into gridDim.z parts of `part` steps (a multiple of 64): a first launch (END) runs every part from h = 0 and
// leaves its final states, the sum of its dt and whether it holds a reset; the second folds the parts before its own into its
// initial state (their decay is exp(A·Σdt)) and computes the outputs.
template <typename T, int NS, bool RESET, bool END>
__global__ void __launch_bounds__(SS_C * SS_N / NS)
sscan_fwd_kernel(const T* __restrict__ u, int su, const T* __restrict__ delta, int sd, const float* __restrict__ A,
                 const T* __restrict__ Bm, int sB, const T* __restrict__ Cm, int sC, const float* __restrict__ Dp,
                 const T* __restrict__ z, int sz, const float* __restrict__ dbias, const int* __restrict__ reset,
                 T* __restrict__ y, float* __restrict__ ckpt, int L, int Di, int softplus, int part, float* __restrict__ p_h,
                 float* __restrict__ p_dt, int* __restrict__ p_reset) {
  constexpr int TPC = SS_N / NS;                     // threads per channel
  constexpr int NT = SS_C * TPC;
  constexpr int PPT = SS_T * SS_C / 4 / NT;          // 4-element pieces of a [64, 16] tile per thread
  __shared__ __align__(16) float2 s_d[SS_T][SS_C];   // (dt, dt·u)
  __shared__ __align__(16) float s_B[SS_T][SS_N], s_C[SS_T][SS_N], s_y[SS_T][SS_YP];
  __shared__ unsigned s_reset[SS_T / 32];            // one bit per step
  const int tid = threadIdx.x;
  const int cl = tid / TPC, q = tid % TPC;
  const int d0 = blockIdx.x * SS_C, b = blockIdx.y, d = d0 + cl;
  const int pr = tid >> 2, pc = (tid & 3) * 4;       // staging: rows pr + k·NT/4, columns pc .. pc + 3
  const bool vu = rows_vec4(u, su), vd = rows_vec4(delta, sd), vB = rows_vec4(Bm, sB), vC = rows_vec4(Cm, sC), vz = rows_vec4(z, sz);
  float2 A2[NS / 2], h[NS / 2];
#pragma unroll
  for (int j = 0; j < NS / 2; ++j) {
    A2[j] = make_float2(A[d * SS_N + q * NS + 2 * j] * SS_LOG2E, A[d * SS_N + q * NS + 2 * j + 1] * SS_LOG2E);
    h[j] = make_float2(0.f, 0.f);
  }
  float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f), D4 = bias4;
  if (dbias) bias4 = make_float4(dbias[d0 + pc], dbias[d0 + pc + 1], dbias[d0 + pc + 2], dbias[d0 + pc + 3]);
  if (Dp) D4 = make_float4(Dp[d0 + pc], Dp[d0 + pc + 1], Dp[d0 + pc + 2], Dp[d0 + pc + 3]);
  const int nseg = (L + SS_T - 1) / SS_T;
  const size_t row0 = static_cast<size_t>(b) * L;
  const int z0 = blockIdx.z, parts = gridDim.z;
  const int seg_lo = z0 * (part / SS_T), seg_hi = min(nseg, seg_lo + part / SS_T);
  float sum_dt = 0.f, sum_lost = 0.f;                // Σdt and what its additions rounded off
  int any_reset = 0;
  if (!END) {
    for (int k = 0; k < z0; ++k) {
      const size_t pi = (static_cast<size_t>(b) * parts + k) * Di + d;
      const bool cut = RESET && p_reset[b * parts + k] != 0;
      const float sdt = p_dt[pi];
#pragma unroll
      for (int j = 0; j < NS / 2; ++j) {
        const float2 e = *reinterpret_cast<const float2*>(&p_h[pi * SS_N + q * NS + 2 * j]);
        const float2 x = make_float2(sdt * A2[j].x, sdt * A2[j].y);
        // selected, not multiplied by zero: a state that is not finite ends with its document
        h[j] = cut ? e : fma_f32x2(ss_exp2_mul(x, h[j]), ss_exp2_cap(x), e);
      }
    }
  }
  Raw4<T> ru[PPT], rd[PPT], rB[PPT], rC[PPT];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int t = t0 + pr + k * (NT / 4);
      ru[k].zero(); rd[k].zero(); rB[k].zero(); rC[k].zero();
      if (t < L) {
        const size_t r = row0 + t;
        ru[k].load(u + r * su + d0 + pc, vu);
        rd[k].load(delta + r * sd + d0 + pc, vd);
        rB[k].load(Bm + r * sB + pc, vB);
        if (!END) rC[k].load(Cm + r * sC + pc, vC);
      }
    }
  };
  fetch(seg_lo * SS_T);
  for (int seg = seg_lo; seg < seg_hi; ++seg) {
    const int t0 = seg * SS_T;
    Raw4<T> cu[PPT], cz[PPT];
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int i = pr + k * (NT / 4);
      cu[k] = ru[k];
      float4 dt = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t0 + i < L) {
        const float4 x = rd[k].get();
        dt = make_float4(x.x + bias4.x, x.y + bias4.y, x.z + bias4.z, x.w + bias4.w);
        if (softplus) dt = make_float4(ss_softplus(dt.x), ss_softplus(dt.y), ss_softplus(dt.z), ss_softplus(dt.w));
      }
      const float4 uu = ru[k].get();
      float4* o = reinterpret_cast<float4*>(&s_d[i][pc]);
      o[0] = make_float4(dt.x, dt.x * uu.x, dt.y, dt.y * uu.y);
      o[1] = make_float4(dt.z, dt.z * uu.z, dt.w, dt.w * uu.w);
      *reinterpret_cast<float4*>(&s_B[i][pc]) = rB[k].get();
      if (!END) *reinterpret_cast<float4*>(&s_C[i][pc]) = rC[k].get();
    }
    if (RESET && tid < SS_T) {
      const unsigned m = __ballot_sync(0xffffffffu, t0 + tid < L && reset[row0 + t0 + tid] != 0);
      if ((tid & 31) == 0) s_reset[tid >> 5] = m;
    }
    __syncthreads();
    if (seg + 1 < seg_hi) fetch(t0 + SS_T);
    if (!END && z) {
#pragma unroll
      for (int k = 0; k < PPT; ++k) {
        const int t = t0 + pr + k * (NT / 4);
        cz[k].zero();
        if (t < L) cz[k].load(z + (row0 + t) * sz + d0 + pc, vz);
      }
    }
#pragma unroll 1
    for (int sb = 0; sb < SS_T / 8; ++sb) {
      if (!END && (sb & 3) == 0 && ckpt) {
        float* cp = ckpt + ((static_cast<size_t>(b) * nseg * 2 + seg * 2 + (sb >> 2)) * Di + d) * SS_N + q * NS;
        if constexpr (NS == 4) *reinterpret_cast<float4*>(cp) = make_float4(h[0].x, h[0].y, h[1].x, h[1].y);
        else *reinterpret_cast<float2*>(cp) = h[0];
      }
      float p[8];
      // eight steps; the ones that clear the state first are marked in `bits` (CLEAR: there are any)
      auto steps = [&](auto CLEAR, unsigned bits) {
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const int i = sb * 8 + s;
          const float2 dd = s_d[i][cl];
          float2 Bv[NS / 2], Cv[NS / 2];
          if constexpr (NS == 4) {
            const float4 b4 = *reinterpret_cast<const float4*>(&s_B[i][q * 4]);
            Bv[0] = make_float2(b4.x, b4.y); Bv[1] = make_float2(b4.z, b4.w);
            if (!END) {
              const float4 c4 = *reinterpret_cast<const float4*>(&s_C[i][q * 4]);
              Cv[0] = make_float2(c4.x, c4.y); Cv[1] = make_float2(c4.z, c4.w);
            }
          } else {
            Bv[0] = *reinterpret_cast<const float2*>(&s_B[i][q * 2]);
            if (!END) Cv[0] = *reinterpret_cast<const float2*>(&s_C[i][q * 2]);
          }
          if (decltype(CLEAR)::value && (bits >> s & 1)) {
#pragma unroll
            for (int j = 0; j < NS / 2; ++j) h[j] = make_float2(0.f, 0.f);
          }
          if (END) p[s] = dd.x;
          const float2 dt2 = make_float2(dd.x, dd.x), du2 = make_float2(dd.y, dd.y);
          float2 acc;
#pragma unroll
          for (int j = 0; j < NS / 2; ++j) {
            const float2 e = mul_f32x2(dt2, A2[j]);
            const float2 a = make_float2(exp2f(e.x), exp2f(e.y));
            h[j] = fma_f32x2(a, h[j], mul_f32x2(du2, Bv[j]));
            if (!END) acc = j == 0 ? mul_f32x2(h[j], Cv[j]) : fma_f32x2(h[j], Cv[j], acc);
          }
          if (!END) p[s] = acc.x + acc.y;
        }
      };
      const unsigned bits = RESET ? s_reset[sb >> 2] >> (sb & 3) * 8 & 0xff : 0;
      if (RESET && bits) {
        any_reset = 1;
        steps(std::true_type(), bits);
      } else {
        steps(std::false_type(), 0);
      }
      if (END) {
        // a plain chain of equal steps rounds the same way every time: 6e-4 of a state that grows by e^115 over a part
        const float g = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7])), t = __fadd_rn(sum_dt, g);
        sum_lost = __fadd_rn(sum_lost, __fsub_rn(g, __fsub_rn(t, sum_dt)));
        sum_dt = t;
        continue;
      }
#pragma unroll
      for (int s0 = 0; s0 < 8; s0 += TPC) {
        float v[TPC];
#pragma unroll
        for (int s = 0; s < TPC; ++s) v[s] = p[s0 + s];
        const float tot = lane_scatter_sum<TPC>(v, q);
        s_y[sb * 8 + s0 + q][cl] = tot;
      }
    }
    __syncthreads();
    if (END) continue;
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int i = pr + k * (NT / 4), t = t0 + i;
      if (t < L) {
        const float4 sv = *reinterpret_cast<const float4*>(&s_y[i][pc]), uu = cu[k].get();
        float4 yv = make_float4(sv.x + D4.x * uu.x, sv.y + D4.y * uu.y, sv.z + D4.z * uu.z, sv.w + D4.w * uu.w);
        if (z) {
          const float4 zz = cz[k].get();
          yv.x *= zz.x * ss_sigmoid(zz.x); yv.y *= zz.y * ss_sigmoid(zz.y);
          yv.z *= zz.z * ss_sigmoid(zz.z); yv.w *= zz.w * ss_sigmoid(zz.w);
        }
        put4(y + (row0 + t) * Di + d0 + pc, yv);
      }
    }
  }
  if (END) {
    const size_t pi = (static_cast<size_t>(b) * parts + z0) * Di + d;
#pragma unroll
    for (int j = 0; j < NS / 2; ++j) *reinterpret_cast<float2*>(&p_h[pi * SS_N + q * NS + 2 * j]) = h[j];
    const float sum = sum_dt + sum_lost;
    if (q == 0) p_dt[pi] = sum == sum ? sum : sum_dt;    // an infinite Σdt has no remainder
    if (RESET && blockIdx.x == 0 && tid == 0) p_reset[b * parts + z0] = any_reset;
  }
}

// MINB: resident CTAs per SM the registers are limited for.  2 (255 registers, hardly any spill) where the grid leaves no more
// to an SM anyway, else 4 (128 registers).  ms with 2 / 3 / 4: B4 L4096 Di3968 (992 CTAs) 2.72 / 2.80 / 2.27, B8 L4096 Di4096
// 5.04 / 4.91 / 4.47, B2 L4096 Di4096 (512) 1.46 / 1.80 / 1.27, B1 L8192 Di5120 (320) 2.54 / 2.04 / 2.09, B1 L32768 Di3968 (248)
// 5.77 / 6.69 / 7.01.
template <typename T, bool RESET, bool GATE, int MINB>
__global__ void __launch_bounds__(128, MINB)
sscan_bwd_kernel(const T* __restrict__ dy, int sdy, const T* __restrict__ u, int su, const T* __restrict__ delta, int sd,
                 const float* __restrict__ A, const T* __restrict__ Bm, int sB, const T* __restrict__ Cm, int sC,
                 const float* __restrict__ Dp, const T* __restrict__ z, int sz, const float* __restrict__ dbias,
                 const int* __restrict__ reset, const float* __restrict__ ckpt, T* __restrict__ du, T* __restrict__ ddelta,
                 T* __restrict__ dz, float* __restrict__ dA, float* __restrict__ dBf, float* __restrict__ dCf,
                 float* __restrict__ dD, float* __restrict__ ddbias, int L, int Di, int softplus) {
  __shared__ __align__(16) float4 s_d[SS_TB][SS_C];                    // (dt, dt·u, dy', u)
  __shared__ __align__(16) float s_B[SS_TB][SS_N], s_C[SS_TB][SS_N];
  __shared__ __align__(16) float s_y[SS_TB][SS_YP], s_gb[SS_TB][SS_YP], s_da[SS_TB][SS_YP];   // Σ_n of h·C, g·B, g·a·h₋·A
  __shared__ __align__(16) float s_bc[4][SS_TB][32];                   // per warp: dB (columns 0..15) and dC (16..31) of its 4 channels
  __shared__ int s_reset[SS_TB];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int cl = tid >> 3, q = tid & 7;
  const int d0 = blockIdx.x * SS_C, b = blockIdx.y, d = d0 + cl;
  const int pr = tid >> 2, pc = (tid & 3) * 4;       // staging: row pr, columns pc .. pc + 3
  const bool vu = rows_vec4(u, su), vd = rows_vec4(delta, sd), vB = rows_vec4(Bm, sB), vC = rows_vec4(Cm, sC), vz = rows_vec4(z, sz),
             vy = rows_vec4(dy, sdy);
  const float2 Ar = make_float2(A[d * SS_N + q * 2], A[d * SS_N + q * 2 + 1]);
  const float2 A2 = make_float2(Ar.x * SS_LOG2E, Ar.y * SS_LOG2E);
  float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f), D4 = bias4;
  if (dbias) bias4 = make_float4(dbias[d0 + pc], dbias[d0 + pc + 1], dbias[d0 + pc + 2], dbias[d0 + pc + 3]);
  if (Dp) D4 = make_float4(Dp[d0 + pc], Dp[d0 + pc + 1], Dp[d0 + pc + 2], Dp[d0 + pc + 3]);
  const int nseg = (L + SS_TB - 1) / SS_TB, nck = 2 * ((L + SS_T - 1) / SS_T);
  const size_t row0 = static_cast<size_t>(b) * L;
  float2 G = make_float2(0.f, 0.f);                  // a_{t+1}·G_{t+1}: adjoint arriving from later steps
  float2 dA_acc = make_float2(0.f, 0.f);
  float4 dD_acc = make_float4(0.f, 0.f, 0.f, 0.f), db_acc = dD_acc;
  Raw4<T> ru, rd, ry, rz, rB, rC;
  float2 h0;
  auto fetch = [&](int seg) {
    const int t = seg * SS_TB + pr;
    ru.zero(); rd.zero(); ry.zero(); rz.zero(); rB.zero(); rC.zero();
    if (t < L) {
      const size_t r = row0 + t;
      ru.load(u + r * su + d0 + pc, vu);
      rd.load(delta + r * sd + d0 + pc, vd);
      ry.load(dy + r * sdy + d0 + pc, vy);
      if (GATE) rz.load(z + r * sz + d0 + pc, vz);
      rB.load(Bm + r * sB + pc, vB);
      rC.load(Cm + r * sC + pc, vC);
    }
    h0 = *reinterpret_cast<const float2*>(&ckpt[((static_cast<size_t>(b) * nck + seg) * Di + d) * SS_N + q * 2]);
  };
  fetch(nseg - 1);
#pragma unroll 1
  for (int seg = nseg - 1; seg >= 0; --seg) {
    const int t = seg * SS_TB + pr;
    const float4 uu = ru.get(), yy = ry.get(), zz = rz.get();
    float4 dt = make_float4(0.f, 0.f, 0.f, 0.f), sg = make_float4(1.f, 1.f, 1.f, 1.f), sz4, dyp = yy;
    {
      if (t < L) {
        const float4 x = rd.get();
        dt = make_float4(x.x + bias4.x, x.y + bias4.y, x.z + bias4.z, x.w + bias4.w);
        if (softplus) {
          sg = make_float4(ss_sigmoid(dt.x), ss_sigmoid(dt.y), ss_sigmoid(dt.z), ss_sigmoid(dt.w));
          dt = make_float4(ss_softplus(dt.x), ss_softplus(dt.y), ss_softplus(dt.z), ss_softplus(dt.w));
        }
      }
      if (GATE) {
        sz4 = make_float4(ss_sigmoid(zz.x), ss_sigmoid(zz.y), ss_sigmoid(zz.z), ss_sigmoid(zz.w));
        dyp = make_float4(yy.x * zz.x * sz4.x, yy.y * zz.y * sz4.y, yy.z * zz.z * sz4.z, yy.w * zz.w * sz4.w);
      }
      s_d[pr][pc] = make_float4(dt.x, dt.x * uu.x, dyp.x, uu.x);
      s_d[pr][pc + 1] = make_float4(dt.y, dt.y * uu.y, dyp.y, uu.y);
      s_d[pr][pc + 2] = make_float4(dt.z, dt.z * uu.z, dyp.z, uu.z);
      s_d[pr][pc + 3] = make_float4(dt.w, dt.w * uu.w, dyp.w, uu.w);
      *reinterpret_cast<float4*>(&s_B[pr][pc]) = rB.get();
      *reinterpret_cast<float4*>(&s_C[pr][pc]) = rC.get();
    }
    if (RESET && tid < SS_TB) s_reset[tid] = seg * SS_TB + tid < L ? reset[row0 + seg * SS_TB + tid] : 0;
    const float2 hin = h0;
    __syncthreads();
    if (seg > 0) fetch(seg - 1);
    // ---- states after every step of the tile
    float2 hs[SS_TB];
    {
      float2 h = hin;
#pragma unroll
      for (int s0 = 0; s0 < SS_TB; s0 += 8) {
        float p[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          const int i = s0 + s;
          const float2 dd = *reinterpret_cast<const float2*>(&s_d[i][cl]);
          const float2 Bv = *reinterpret_cast<const float2*>(&s_B[i][q * 2]);
          if (RESET && s_reset[i]) h = make_float2(0.f, 0.f);
          const float2 e = mul_f32x2(make_float2(dd.x, dd.x), A2);
          h = fma_f32x2(make_float2(exp2f(e.x), exp2f(e.y)), h, mul_f32x2(make_float2(dd.y, dd.y), Bv));
          hs[i] = h;
          if (GATE) {
            const float2 c = mul_f32x2(h, *reinterpret_cast<const float2*>(&s_C[i][q * 2]));
            p[s] = c.x + c.y;
          }
        }
        if (GATE) s_y[s0 + q][cl] = lane_scatter_sum<8>(p, q);
        __syncwarp();                                // keeps the loads of the next steps from being moved up here (registers)
      }
    }
    // ---- adjoint, last step first
#pragma unroll
    for (int s0 = SS_TB - 8; s0 >= 0; s0 -= 8) {
      float vgb[8], vda[8];
#pragma unroll
      for (int s = 7; s >= 0; --s) {
        const int i = s0 + s;
        const float4 dd = s_d[i][cl];
        const float2 Bv = *reinterpret_cast<const float2*>(&s_B[i][q * 2]), Cv = *reinterpret_cast<const float2*>(&s_C[i][q * 2]);
        const float2 e = mul_f32x2(make_float2(dd.x, dd.x), A2);
        float2 a = make_float2(exp2f(e.x), exp2f(e.y));
        float2 hp = i > 0 ? hs[i > 0 ? i - 1 : 0] : hin;
        if (RESET && s_reset[i]) { a = make_float2(0.f, 0.f); hp = a; }
        const float2 g = fma_f32x2(Cv, make_float2(dd.z, dd.z), G);
        G = mul_f32x2(g, a);
        const float2 daa = mul_f32x2(G, hp);
        dA_acc = fma_f32x2(daa, make_float2(dd.x, dd.x), dA_acc);
        const float2 gb = mul_f32x2(g, Bv), da = mul_f32x2(daa, Ar);
        vgb[s] = gb.x + gb.y;
        vda[s] = da.x + da.y;
        const float2 vB2 = mul_f32x2(g, make_float2(dd.y, dd.y)), vC2 = mul_f32x2(hs[i], make_float2(dd.z, dd.z));
        // four values over the warp's four channels: lane bit 4 keeps dB or dC, lane bit 3 the first or the second state
        const bool hi = (lane & 16) != 0, odd = (lane & 8) != 0;
        const float s0v = hi ? vB2.x : vC2.x, s1v = hi ? vB2.y : vC2.y;
        const float k0 = (hi ? vC2.x : vB2.x) + __shfl_xor_sync(0xffffffffu, s0v, 16);
        const float k1 = (hi ? vC2.y : vB2.y) + __shfl_xor_sync(0xffffffffu, s1v, 16);
        const float kk = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 8);
        s_bc[w][i][(hi ? 16 : 0) + 2 * q + (odd ? 1 : 0)] = kk;
        if (s == 4) __syncwarp();
      }
      s_gb[s0 + q][cl] = lane_scatter_sum<8>(vgb, q);
      s_da[s0 + q][cl] = lane_scatter_sum<8>(vda, q);
      __syncwarp();
    }
    __syncthreads();
    if (t < L) {
      const size_t r = row0 + t;
      const float4 gb = *reinterpret_cast<const float4*>(&s_gb[pr][pc]), da = *reinterpret_cast<const float4*>(&s_da[pr][pc]);
      const float4 dd = make_float4((da.x + gb.x * uu.x) * sg.x, (da.y + gb.y * uu.y) * sg.y, (da.z + gb.z * uu.z) * sg.z,
                                    (da.w + gb.w * uu.w) * sg.w);
      put4(ddelta + r * Di + d0 + pc, dd);
      db_acc.x += dd.x; db_acc.y += dd.y; db_acc.z += dd.z; db_acc.w += dd.w;
      put4(du + r * Di + d0 + pc, make_float4(gb.x * dt.x + dyp.x * D4.x, gb.y * dt.y + dyp.y * D4.y, gb.z * dt.z + dyp.z * D4.z,
                                              gb.w * dt.w + dyp.w * D4.w));
      dD_acc.x += dyp.x * uu.x; dD_acc.y += dyp.y * uu.y; dD_acc.z += dyp.z * uu.z; dD_acc.w += dyp.w * uu.w;
      if (GATE) {
        const float4 sv = *reinterpret_cast<const float4*>(&s_y[pr][pc]);
        put4(dz + r * Di + d0 + pc,
             make_float4(yy.x * (sv.x + D4.x * uu.x) * sz4.x * (1.f + zz.x * (1.f - sz4.x)),
                         yy.y * (sv.y + D4.y * uu.y) * sz4.y * (1.f + zz.y * (1.f - sz4.y)),
                         yy.z * (sv.z + D4.z * uu.z) * sz4.z * (1.f + zz.z * (1.f - sz4.z)),
                         yy.w * (sv.w + D4.w * uu.w) * sz4.w * (1.f + zz.w * (1.f - sz4.w))));
      }
      // partial sums of this 16-channel block; summed over blocks by sscan_reduce_bc_kernel
      const size_t po = (static_cast<size_t>(blockIdx.x) * gridDim.y * L + r) * SS_N + pc;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float4 a = *reinterpret_cast<const float4*>(&s_bc[0][pr][half * 16 + pc]);
#pragma unroll
        for (int ww = 1; ww < 4; ++ww) {
          const float4 o = *reinterpret_cast<const float4*>(&s_bc[ww][pr][half * 16 + pc]);
          a.x += o.x; a.y += o.y; a.z += o.z; a.w += o.w;
        }
        *reinterpret_cast<float4*>((half ? dCf : dBf) + po) = a;
      }
    }
    // the next tile's staging writes s_d / s_B / s_C only (nobody reads them here any more); its sums are written after its barrier
  }
  atomicAdd(&dA[d * SS_N + q * 2], dA_acc.x);
  atomicAdd(&dA[d * SS_N + q * 2 + 1], dA_acc.y);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {                 // the 8 rows of a warp
    dD_acc.x += __shfl_xor_sync(0xffffffffu, dD_acc.x, o); dD_acc.y += __shfl_xor_sync(0xffffffffu, dD_acc.y, o);
    dD_acc.z += __shfl_xor_sync(0xffffffffu, dD_acc.z, o); dD_acc.w += __shfl_xor_sync(0xffffffffu, dD_acc.w, o);
    db_acc.x += __shfl_xor_sync(0xffffffffu, db_acc.x, o); db_acc.y += __shfl_xor_sync(0xffffffffu, db_acc.y, o);
    db_acc.z += __shfl_xor_sync(0xffffffffu, db_acc.z, o); db_acc.w += __shfl_xor_sync(0xffffffffu, db_acc.w, o);
  }
  if (lane < 4) {
    if (dD) {
      atomicAdd(&dD[d0 + pc], dD_acc.x); atomicAdd(&dD[d0 + pc + 1], dD_acc.y);
      atomicAdd(&dD[d0 + pc + 2], dD_acc.z); atomicAdd(&dD[d0 + pc + 3], dD_acc.w);
    }
    if (ddbias) {
      atomicAdd(&ddbias[d0 + pc], db_acc.x); atomicAdd(&ddbias[d0 + pc + 1], db_acc.y);
      atomicAdd(&ddbias[d0 + pc + 2], db_acc.z); atomicAdd(&ddbias[d0 + pc + 3], db_acc.w);
    }
  }
}

// dB / dC [rows, 16] = Σ over channel blocks of the partial sums [nblk, rows, 16] written by the backward.
template <typename T>
__global__ void __launch_bounds__(256) sscan_reduce_bc_kernel(const float* __restrict__ pB, const float* __restrict__ pC,
                                                             T* __restrict__ dB, T* __restrict__ dC, size_t n, int nblk) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float sb = 0.f, sc = 0.f;
#pragma unroll 4
  for (int k = 0; k < nblk; ++k) { sb += pB[k * n + i]; sc += pC[k * n + i]; }
  st1(dB + i, sb);
  st1(dC + i, sc);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_selective_scan_channel_blocks(int Di) { return Di / SS_C; }

extern "C" int b200_selective_scan_ckpt_segments(int L) { return 2 * ((L + SS_T - 1) / SS_T); }

template <typename T, int NS>
static void launch_sscan_fwd(const void* u, int su, const void* delta, int sd, const float* A, const void* Bm, int sB, const void* Cm,
                             int sC, const float* D, const void* z, int sz, const float* dbias, const int* reset, void* y, float* ckpt,
                             int B, int L, int Di, int softplus, int parts, float* scratch, cudaStream_t st) {
  const int part = ((L + parts - 1) / parts + SS_T - 1) / SS_T * SS_T;
  parts = (L + part - 1) / part;                       // no empty part
  float* p_h = scratch;
  float* p_dt = scratch + static_cast<size_t>(B) * parts * Di * SS_N;
  int* p_reset = reinterpret_cast<int*>(p_dt + static_cast<size_t>(B) * parts * Di);
  auto run = [&](auto kern, int nz) {
    kern<<<dim3(Di / SS_C, B, nz), SS_C * SS_N / NS, 0, st>>>((const T*)u, su, (const T*)delta, sd, A, (const T*)Bm, sB, (const T*)Cm, sC, D,
                                                             (const T*)z, sz, dbias, reset, (T*)y, ckpt, L, Di, softplus, part, p_h, p_dt,
                                                             p_reset);
  };
  if (parts > 1) {
    if constexpr (NS == 4) {
      if (reset) run(sscan_fwd_kernel<T, 4, true, true>, parts); else run(sscan_fwd_kernel<T, 4, false, true>, parts);
    }
  }
  if (reset) run(sscan_fwd_kernel<T, NS, true, false>, parts); else run(sscan_fwd_kernel<T, NS, false, false>, parts);
}

// Parts of the sequence that the forward scan runs side by side.  With few channels the steps cost their latency: splitting the
// time costs a second pass over the exponentials but multiplies the warps.  Parts are kept at 512 steps or more.  Whole -> split,
// ms: B·Di 4096: L1536 0.112 -> 0.106, L1600 0.116 -> 0.119, L2048 0.153 -> 0.130, L4096 0.310 -> 0.228; B·Di 7936: L1536 0.156 -> 0.198,
// L2048 0.207 -> 0.226, L4096 0.413 -> 0.432, L8192 0.825 -> 0.821; B·Di 8192: L4096 0.412 -> 0.447, L32768 3.30 -> 3.52; B1 L32768 Di3968
// 2.73 -> 1.66.  The line lies at B·Di = 8192; short sequences just below it would be better off whole (every one of these is ahead of
// one state per thread: 0.239 for B·Di 7936 L1536).
extern "C" int b200_selective_scan_parts(int B, int L, int Di) {
  const long long width = static_cast<long long>(B) * Di;
  if (width <= 0 || width >= 8192) return 1;
  int parts = static_cast<int>((49152 + width - 1) / width);
  if (parts > L / 512) parts = L / 512;
  return parts > 2 ? parts : 1;                        // two parts would only pay back the second pass
}
// floats of scratch for that many parts
extern "C" long long b200_selective_scan_scratch(int B, int Di, int parts) {
  return parts > 1 ? static_cast<long long>(B) * parts * (Di * (SS_N + 1LL) + 1) : 0;
}

// u, delta, z: rows of `su`, `sd`, `sz` elements; Bm, Cm: [B·L, 16] with row strides sB, sC; y: dense [B, L, Di].
// reset: int32 per token (1 = h is cleared before this step) or null.  ckpt: fp32 [B, 2·ceil(L/64), Di, 16] or null.
// parts, scratch: see b200_selective_scan_parts / _scratch (1, null: one pass).
extern "C" int b200_selective_scan_fwd(const void* u, int su, const void* delta, int sd, const float* A, const void* Bm, int sB,
                                       const void* Cm, int sC, const float* D, const void* z, int sz, const float* dbias,
                                       const int* reset, void* y, float* ckpt, int dtype, int B, int L, int Di, int softplus, int parts,
                                       float* scratch, cudaStream_t st) {
  if (Di % SS_C || parts < 1 || (parts > 1 && !scratch)) return -1;
  if (B * L == 0) return 0;
  // four states per thread leave B·Di/8 warps for 592 schedulers; with fewer than about two and a half each, two states per thread.
  // ms, two / four: B·Di 6144 L1000 0.086 / 0.094, 8192 L4096 0.412 / 0.382, 10240 L1000 0.120 / 0.120, 11904 L4096 0.542 / 0.478,
  // 12288 L1000 0.139 / 0.124, 15872 L4096 0.627 / 0.581: the true crossing is nearer to 8192 than to 12288.
  const bool ns4 = parts > 1 || static_cast<long long>(B) * Di >= 12288;
  auto run = dtype == 1 ? (ns4 ? launch_sscan_fwd<__nv_bfloat16, 4> : launch_sscan_fwd<__nv_bfloat16, 2>)
                        : (ns4 ? launch_sscan_fwd<float, 4> : launch_sscan_fwd<float, 2>);
  run(u, su, delta, sd, A, Bm, sB, Cm, sC, D, z, sz, dbias, reset, y, ckpt, B, L, Di, softplus, parts, scratch, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

template <typename T>
static void launch_sscan_bwd(const void* dy, int sdy, const void* u, int su, const void* delta, int sd, const float* A, const void* Bm,
                             int sB, const void* Cm, int sC, const float* D, const void* z, int sz, const float* dbias, const int* reset,
                             const float* ckpt, void* du, void* ddelta, void* dz, float* dA, float* partB, float* partC, void* dB,
                             void* dC, float* dD, float* ddbias, int B, int L, int Di, int softplus, cudaStream_t st) {
  const bool few = static_cast<long long>(B) * (Di / SS_C) <= 2 * 148;
  auto kern = reset ? (z ? (few ? sscan_bwd_kernel<T, true, true, 2> : sscan_bwd_kernel<T, true, true, 4>)
                         : (few ? sscan_bwd_kernel<T, true, false, 2> : sscan_bwd_kernel<T, true, false, 4>))
                    : (z ? (few ? sscan_bwd_kernel<T, false, true, 2> : sscan_bwd_kernel<T, false, true, 4>)
                         : (few ? sscan_bwd_kernel<T, false, false, 2> : sscan_bwd_kernel<T, false, false, 4>));
  kern<<<dim3(Di / SS_C, B), 128, 0, st>>>((const T*)dy, sdy, (const T*)u, su, (const T*)delta, sd, A, (const T*)Bm, sB, (const T*)Cm, sC,
                                           D, (const T*)z, sz, dbias, reset, ckpt, (T*)du, (T*)ddelta, (T*)dz, dA, partB, partC, dD,
                                           ddbias, L, Di, softplus);
  const size_t n = static_cast<size_t>(B) * L * SS_N;
  sscan_reduce_bc_kernel<T><<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(partB, partC, (T*)dB, (T*)dC, n, Di / SS_C);
}

extern "C" int b200_selective_scan_bwd(const void* dy, int sdy, const void* u, int su, const void* delta, int sd, const float* A,
                                       const void* Bm, int sB, const void* Cm, int sC, const float* D, const void* z, int sz,
                                       const float* dbias, const int* reset, const float* ckpt, void* du, void* ddelta, void* dz,
                                       float* dA, float* partB, float* partC, void* dB, void* dC, float* dD, float* ddbias,
                                       int dtype, int B, int L, int Di, int softplus, cudaStream_t st) {
  if (Di % SS_C) return -1;
  if (B * L == 0) return 0;
  auto run = dtype == 1 ? launch_sscan_bwd<__nv_bfloat16> : launch_sscan_bwd<float>;
  run(dy, sdy, u, su, delta, sd, A, Bm, sB, Cm, sC, D, z, sz, dbias, reset, ckpt, du, ddelta, dz, dA, partB, partC, dB, dC, dD, ddbias, B,
      L, Di, softplus, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
