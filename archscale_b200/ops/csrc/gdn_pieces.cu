// The 64×64 pieces of the chunked gated delta rule, one block per (batch, head, chunk): what lies between the Gram products, the
// triangular inverse and the products with values and keys.  gc: inclusive log-decay inside the chunk, beta: the write strengths.
//
//   mask:  A_ij  = Gk_ij · e^(gc_i − gc_j) · beta_i  (j < i),     qk_ij = Gq_ij · e^(gc_i − gc_j)  (j ≤ i)
//   cols:  Tu_ij = T_ij · beta_j,                               Tw_ij = T_ij · beta_j · e^(gc_j)
//
// and their backward with the row and column sums that go to gc and beta.  As element-wise PyTorch ops these were about 14 launches
// forward and 35 backward per layer over [blocks, 64, 64] fp32 tensors; here each is one pass that reads and writes every
// block once (16 KB per fp32 block; memory-bound).  Whole op, forward / forward + backward, ms, before (with the recurrence kernel as it was
// then) and now: B8 T4096 H6 Dk256 Dv512 1.90 / 6.48 -> 1.42 / 5.01, B3 T2731 1.02 / 2.59 -> 0.66 / 2.06.
// 256 threads per block: thread t does row t / 4, columns 16·(t % 4) .. + 15.  Sums run in a fixed order.  Built without
// --use_fast_math, whose exponential loses bits of strongly decayed factors and flushes those below 2^-126.
#include "sm100.cuh"
#include "api.h"

namespace b200 {

constexpr int GPC = 64, GP_THREADS = 256;

struct GpPos {
  int i, j0;
  size_t off;        // of element (i, j0) of this block
};
__device__ __forceinline__ GpPos gp_pos() {
  const int i = threadIdx.x >> 2, j0 = (threadIdx.x & 3) * 16;
  return {i, j0, (static_cast<size_t>(blockIdx.x) * GPC + i) * GPC + j0};
}
__device__ __forceinline__ void gp_load(const float* p, float (&v)[16]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float4 f = reinterpret_cast<const float4*>(p)[u];
    v[4 * u] = f.x; v[4 * u + 1] = f.y; v[4 * u + 2] = f.z; v[4 * u + 3] = f.w;
  }
}
__device__ __forceinline__ void gp_load(const __nv_bfloat16* p, float (&v)[16]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint4 w = reinterpret_cast<const uint4*>(p)[u];
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { const float2 f = unpack_bf16x2(ww[e]); v[8 * u + 2 * e] = f.x; v[8 * u + 2 * e + 1] = f.y; }
  }
}
__device__ __forceinline__ void gp_store(float* p, const float (&v)[16]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) reinterpret_cast<float4*>(p)[u] = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
}
__device__ __forceinline__ void gp_store(__nv_bfloat16* p, const float (&v)[16]) {
#pragma unroll
  for (int u = 0; u < 2; ++u)
    reinterpret_cast<uint4*>(p)[u] = make_uint4(pack_bf16x2(v[8 * u], v[8 * u + 1]), pack_bf16x2(v[8 * u + 2], v[8 * u + 3]),
                                                pack_bf16x2(v[8 * u + 4], v[8 * u + 5]), pack_bf16x2(v[8 * u + 6], v[8 * u + 7]));
}
// Column sums over the block's 64 rows of what each thread holds for its 16 columns; returned to threads 0..63 (thread = column).
__device__ __forceinline__ float gp_col_sum(float (&v)[16], float (&s)[8][GPC]) {
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    v[e] += __shfl_xor_sync(0xffffffffu, v[e], 4);
    v[e] += __shfl_xor_sync(0xffffffffu, v[e], 8);
    v[e] += __shfl_xor_sync(0xffffffffu, v[e], 16);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();                                   // s may still be read from the sum before
  if (lane < 4) {
#pragma unroll
    for (int e = 0; e < 16; ++e) s[warp][lane * 16 + e] = v[e];
  }
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x < GPC) {
#pragma unroll
    for (int w = 0; w < 8; ++w) t += s[w][threadIdx.x];
  }
  return t;
}
__device__ __forceinline__ float gp_row_sum(float v) {   // over the four threads of a row
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ void gp_stage(const float* gc, const float* beta, float (&s_gc)[GPC], float (&s_b)[GPC]) {
  if (threadIdx.x < GPC) {
    s_gc[threadIdx.x] = gc[static_cast<size_t>(blockIdx.x) * GPC + threadIdx.x];
    s_b[threadIdx.x] = beta[static_cast<size_t>(blockIdx.x) * GPC + threadIdx.x];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(GP_THREADS) gdn_mask_fwd_kernel(const float* __restrict__ Gk, const float* __restrict__ Gq,
                                                                  const float* __restrict__ gc, const float* __restrict__ beta,
                                                                  float* __restrict__ A, __nv_bfloat16* __restrict__ qk) {
  __shared__ float s_gc[GPC], s_b[GPC];
  gp_stage(gc, beta, s_gc, s_b);
  const GpPos p = gp_pos();
  float a[16], q[16];
  gp_load(Gk + p.off, a);
  gp_load(Gq + p.off, q);
  const float gi = s_gc[p.i], bi = s_b[p.i];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int j = p.j0 + e;
    const float dec = j <= p.i ? expf(gi - s_gc[j]) : 0.f;
    a[e] = j < p.i ? a[e] * dec * bi : 0.f;
    q[e] = j <= p.i ? q[e] * dec : 0.f;
  }
  gp_store(A + p.off, a);
  gp_store(qk + p.off, q);
}

__global__ void __launch_bounds__(GP_THREADS) gdn_mask_bwd_kernel(const float* __restrict__ dA, const __nv_bfloat16* __restrict__ dqk,
                                                                  const float* __restrict__ Gk, const float* __restrict__ Gq,
                                                                  const float* __restrict__ gc, const float* __restrict__ beta,
                                                                  __nv_bfloat16* __restrict__ dGk, __nv_bfloat16* __restrict__ dGq,
                                                                  float* __restrict__ dgc, float* __restrict__ dbeta) {
  __shared__ float s_gc[GPC], s_b[GPC], s_row[GPC], s_sum[8][GPC];
  gp_stage(gc, beta, s_gc, s_b);
  const GpPos p = gp_pos();
  float da[16], dq[16], k[16], q[16];
  gp_load(dA + p.off, da);
  gp_load(dqk + p.off, dq);
  gp_load(Gk + p.off, k);
  gp_load(Gq + p.off, q);
  const float gi = s_gc[p.i], bi = s_b[p.i];
  float db = 0.f, row = 0.f;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int j = p.j0 + e;
    const float dec = j <= p.i ? expf(gi - s_gc[j]) : 0.f;
    const float dad = j < p.i ? da[e] * dec : 0.f, dqd = j <= p.i ? dq[e] * dec : 0.f;
    const float t = j < p.i ? dad * k[e] : 0.f;
    db += t;
    da[e] = dad * bi;
    dq[e] = dqd;
    k[e] = t * bi + (j <= p.i ? dqd * q[e] : 0.f);       // dL/d(gc_i − gc_j)
    row += k[e];
  }
  gp_store(dGk + p.off, da);
  gp_store(dGq + p.off, dq);
  db = gp_row_sum(db);
  row = gp_row_sum(row);
  const size_t base = static_cast<size_t>(blockIdx.x) * GPC;
  if ((threadIdx.x & 3) == 0) {
    dbeta[base + p.i] = db;
    s_row[p.i] = row;
  }
  const float col = gp_col_sum(k, s_sum);                // (its barriers also order s_row)
  if (threadIdx.x < GPC) dgc[base + threadIdx.x] = s_row[threadIdx.x] - col;
}

__global__ void __launch_bounds__(GP_THREADS) gdn_cols_fwd_kernel(const float* __restrict__ T, const float* __restrict__ gc,
                                                                  const float* __restrict__ beta, __nv_bfloat16* __restrict__ Tu,
                                                                  __nv_bfloat16* __restrict__ Tw) {
  __shared__ float s_gc[GPC], s_b[GPC];
  gp_stage(gc, beta, s_gc, s_b);
  const GpPos p = gp_pos();
  float t[16], w[16];
  gp_load(T + p.off, t);
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const float b = s_b[p.j0 + e];
    w[e] = t[e] * (b * expf(s_gc[p.j0 + e]));
    t[e] = t[e] * b;
  }
  gp_store(Tu + p.off, t);
  gp_store(Tw + p.off, w);
}

__global__ void __launch_bounds__(GP_THREADS) gdn_cols_bwd_kernel(const __nv_bfloat16* __restrict__ dTu, const __nv_bfloat16* __restrict__ dTw,
                                                                  const float* __restrict__ T, const float* __restrict__ gc,
                                                                  const float* __restrict__ beta, float* __restrict__ dT,
                                                                  float* __restrict__ dgc, float* __restrict__ dbeta) {
  __shared__ float s_gc[GPC], s_b[GPC], s_sum[8][GPC];
  gp_stage(gc, beta, s_gc, s_b);
  const GpPos p = gp_pos();
  float du[16], dw[16], t[16], o[16];
  gp_load(dTu + p.off, du);
  gp_load(dTw + p.off, dw);
  gp_load(T + p.off, t);
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const float b = s_b[p.j0 + e];
    o[e] = du[e] * b + dw[e] * (b * expf(s_gc[p.j0 + e]));
    du[e] *= t[e];
    dw[e] *= t[e];
  }
  gp_store(dT + p.off, o);
  const float su = gp_col_sum(du, s_sum), sw = gp_col_sum(dw, s_sum);
  if (threadIdx.x < GPC) {
    const size_t at = static_cast<size_t>(blockIdx.x) * GPC + threadIdx.x;
    const float e = expf(s_gc[threadIdx.x]);
    dbeta[at] = su + e * sw;
    dgc[at] = s_b[threadIdx.x] * e * sw;
  }
}

}  // namespace b200

// Every matrix argument: [n, 64, 64], rows of 64 elements, 16-byte aligned; gc, beta and their gradients: [n, 64] fp32.
extern "C" int b200_gdn_mask_fwd(const float* Gk, const float* Gq, const float* gc, const float* beta, float* A, void* qk, int n,
                                 cudaStream_t st) {
  if (n <= 0) return 0;
  b200::gdn_mask_fwd_kernel<<<n, b200::GP_THREADS, 0, st>>>(Gk, Gq, gc, beta, A, (__nv_bfloat16*)qk);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
extern "C" int b200_gdn_mask_bwd(const float* dA, const void* dqk, const float* Gk, const float* Gq, const float* gc, const float* beta,
                                 void* dGk, void* dGq, float* dgc, float* dbeta, int n, cudaStream_t st) {
  if (n <= 0) return 0;
  b200::gdn_mask_bwd_kernel<<<n, b200::GP_THREADS, 0, st>>>(dA, (const __nv_bfloat16*)dqk, Gk, Gq, gc, beta, (__nv_bfloat16*)dGk,
                                                            (__nv_bfloat16*)dGq, dgc, dbeta);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
extern "C" int b200_gdn_cols_fwd(const float* T, const float* gc, const float* beta, void* Tu, void* Tw, int n, cudaStream_t st) {
  if (n <= 0) return 0;
  b200::gdn_cols_fwd_kernel<<<n, b200::GP_THREADS, 0, st>>>(T, gc, beta, (__nv_bfloat16*)Tu, (__nv_bfloat16*)Tw);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
extern "C" int b200_gdn_cols_bwd(const void* dTu, const void* dTw, const float* T, const float* gc, const float* beta, float* dT,
                                 float* dgc, float* dbeta, int n, cudaStream_t st) {
  if (n <= 0) return 0;
  b200::gdn_cols_bwd_kernel<<<n, b200::GP_THREADS, 0, st>>>((const __nv_bfloat16*)dTu, (const __nv_bfloat16*)dTw, T, gc, beta, dT, dgc,
                                                            dbeta);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
