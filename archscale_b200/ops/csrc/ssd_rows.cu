// Element-wise passes around the chunked SSD (Mamba-2) products, one launch each.  A row is one (token, head): P contiguous
// channels (P a multiple of 64), taken by 16 lanes with four channels each; per-row factors and row sums are [rows].
//   scale     xw = x · w_row                                                        (operand of the chunk summaries)
//   combine   out = y + y2 · carry_row + x · D_head                                 (intra-chunk + state read-out + skip)
//   dprep     dy2 = dout · carry_row,  dcarry_row = Σ_p dout·y2,  dD_row = Σ_p dout·x
//   dfinish   dx = dx_i + dxw · w_row + dout · D_head,  dw_row = Σ_p dxw·x
// x, out, dout are bf16 or fp32 (T), everything else fp32.  All four are bound by memory: at B4 L4096 H62 P64 (65 M elements)
// they move 0.39 / 0.78 / 0.78 / 0.91 GB.  As PyTorch expressions the same work was about thirty passes over fp32 tensors of
// 260 MB each per layer (widening copies of x, broadcast products, their reductions and gradient sums): with the new intra-chunk
// backward the whole op went from 1.75 to 0.98 ms forward and from 5.54 to 1.80 ms backward at that size with N = 128 (batched matmuls
// in TF32, as the trainer sets them; in fp32 2.33 -> 1.73 and 6.53 -> 2.75).
#include "sm100.cuh"
#include "api.h"

namespace b200 {

__device__ __forceinline__ float4 sr_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 sr_ld4(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void sr_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void sr_st4(__nv_bfloat16* p, float4 v) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}
__device__ __forceinline__ float sr_dot(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ float sr_sum16(float v) {
#pragma unroll
  for (int o = 8; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, 16);
  return v;
}

constexpr int SR_THREADS = 256, SR_ROWS = SR_THREADS / 16;

template <typename T>
__global__ void __launch_bounds__(SR_THREADS) ssd_scale_kernel(const T* __restrict__ x, const float* __restrict__ w, float* __restrict__ xw,
                                                              long long rows, int P) {
  const long long r = static_cast<long long>(blockIdx.x) * SR_ROWS + (threadIdx.x >> 4);
  if (r >= rows) return;
  const float s = w[r];
  for (int p = (threadIdx.x & 15) * 4; p < P; p += 64) {
    const float4 v = sr_ld4(x + r * P + p);
    sr_st4(xw + r * P + p, make_float4(v.x * s, v.y * s, v.z * s, v.w * s));
  }
}

template <typename T>
__global__ void __launch_bounds__(SR_THREADS) ssd_combine_kernel(const float* __restrict__ y, const float* __restrict__ y2,
                                                                const float* __restrict__ carry, const T* __restrict__ x,
                                                                const float* __restrict__ D, T* __restrict__ out, long long rows, int H, int P) {
  const long long r = static_cast<long long>(blockIdx.x) * SR_ROWS + (threadIdx.x >> 4);
  if (r >= rows) return;
  const float c = carry[r], d = D ? D[r % H] : 0.f;
  for (int p = (threadIdx.x & 15) * 4; p < P; p += 64) {
    const float4 a = sr_ld4(y + r * P + p), b = sr_ld4(y2 + r * P + p);
    float4 o = make_float4(a.x + b.x * c, a.y + b.y * c, a.z + b.z * c, a.w + b.w * c);
    if (D) {
      const float4 v = sr_ld4(x + r * P + p);
      o = make_float4(o.x + v.x * d, o.y + v.y * d, o.z + v.z * d, o.w + v.w * d);
    }
    sr_st4(out + r * P + p, o);
  }
}

template <typename T>
__global__ void __launch_bounds__(SR_THREADS) ssd_dprep_kernel(const T* __restrict__ dout, const float* __restrict__ y2,
                                                              const float* __restrict__ carry, const T* __restrict__ x,
                                                              float* __restrict__ dy2, float* __restrict__ dcarry, float* __restrict__ dD,
                                                              long long rows, int P) {
  const long long r = static_cast<long long>(blockIdx.x) * SR_ROWS + (threadIdx.x >> 4);
  const bool on = r < rows;
  const float c = on ? carry[r] : 0.f;
  float s2 = 0.f, sx = 0.f;
  if (on) {
    for (int p = (threadIdx.x & 15) * 4; p < P; p += 64) {
      const float4 g = sr_ld4(dout + r * P + p);
      s2 += sr_dot(g, sr_ld4(y2 + r * P + p));
      sx += sr_dot(g, sr_ld4(x + r * P + p));
      sr_st4(dy2 + r * P + p, make_float4(g.x * c, g.y * c, g.z * c, g.w * c));
    }
  }
  s2 = sr_sum16(s2);
  sx = sr_sum16(sx);
  if (on && (threadIdx.x & 15) == 0) { dcarry[r] = s2; dD[r] = sx; }
}

template <typename T>
__global__ void __launch_bounds__(SR_THREADS) ssd_dfinish_kernel(const float* __restrict__ dxi, const float* __restrict__ dxw,
                                                                const float* __restrict__ w, const T* __restrict__ dout,
                                                                const T* __restrict__ x, const float* __restrict__ D, T* __restrict__ dx,
                                                                float* __restrict__ dw, long long rows, int H, int P) {
  const long long r = static_cast<long long>(blockIdx.x) * SR_ROWS + (threadIdx.x >> 4);
  const bool on = r < rows;
  const float s = on ? w[r] : 0.f, d = on && D ? D[r % H] : 0.f;
  float sw = 0.f;
  if (on) {
    for (int p = (threadIdx.x & 15) * 4; p < P; p += 64) {
      const float4 a = sr_ld4(dxi + r * P + p), b = sr_ld4(dxw + r * P + p);
      sw += sr_dot(b, sr_ld4(x + r * P + p));
      float4 o = make_float4(a.x + b.x * s, a.y + b.y * s, a.z + b.z * s, a.w + b.w * s);
      if (D) {
        const float4 g = sr_ld4(dout + r * P + p);
        o = make_float4(o.x + g.x * d, o.y + g.y * d, o.z + g.z * d, o.w + g.w * d);
      }
      sr_st4(dx + r * P + p, o);
    }
  }
  sw = sr_sum16(sw);
  if (on && (threadIdx.x & 15) == 0) dw[r] = sw;
}

static unsigned sr_grid(long long rows) { return static_cast<unsigned>((rows + SR_ROWS - 1) / SR_ROWS); }

}  // namespace b200

using namespace b200;
using sr_bf16 = __nv_bfloat16;

// dtype: 0 fp32, 1 bf16 (x, out, dout, dx).  rows = tokens · H; P a multiple of 64.  D may be null.
extern "C" int b200_ssd_scale(const void* x, int dtype, const float* w, float* xw, long long rows, int P, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (P % 64 || (rows + SR_ROWS - 1) / SR_ROWS > 0x7fffffffLL) return -1;
  if (dtype == 1) ssd_scale_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(static_cast<const sr_bf16*>(x), w, xw, rows, P);
  else ssd_scale_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(static_cast<const float*>(x), w, xw, rows, P);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
extern "C" int b200_ssd_combine(const float* y, const float* y2, const float* carry, const void* x, int dtype, const float* D, void* out,
                                long long rows, int H, int P, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (P % 64 || (rows + SR_ROWS - 1) / SR_ROWS > 0x7fffffffLL) return -1;
  if (dtype == 1)
    ssd_combine_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(y, y2, carry, static_cast<const sr_bf16*>(x), D, static_cast<sr_bf16*>(out), rows, H, P);
  else
    ssd_combine_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(y, y2, carry, static_cast<const float*>(x), D, static_cast<float*>(out), rows, H, P);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
extern "C" int b200_ssd_dprep(const void* dout, int dtype, const float* y2, const float* carry, const void* x, float* dy2, float* dcarry,
                              float* dD, long long rows, int P, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (P % 64 || (rows + SR_ROWS - 1) / SR_ROWS > 0x7fffffffLL) return -1;
  if (dtype == 1)
    ssd_dprep_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(static_cast<const sr_bf16*>(dout), y2, carry, static_cast<const sr_bf16*>(x), dy2,
                                                           dcarry, dD, rows, P);
  else
    ssd_dprep_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(static_cast<const float*>(dout), y2, carry, static_cast<const float*>(x), dy2, dcarry,
                                                           dD, rows, P);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
extern "C" int b200_ssd_dfinish(const float* dxi, const float* dxw, const float* w, const void* dout, const void* x, int dtype,
                                const float* D, void* dx, float* dw, long long rows, int H, int P, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (P % 64 || (rows + SR_ROWS - 1) / SR_ROWS > 0x7fffffffLL) return -1;
  if (dtype == 1)
    ssd_dfinish_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(dxi, dxw, w, static_cast<const sr_bf16*>(dout), static_cast<const sr_bf16*>(x), D,
                                                             static_cast<sr_bf16*>(dx), dw, rows, H, P);
  else
    ssd_dfinish_kernel<<<sr_grid(rows), SR_THREADS, 0, st>>>(dxi, dxw, w, static_cast<const float*>(dout), static_cast<const float*>(x), D,
                                                             static_cast<float*>(dx), dw, rows, H, P);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
