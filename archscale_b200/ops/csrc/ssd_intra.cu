// Intra-chunk part of the SSD (Mamba-2) scan, forward and backward, without materialising the per-head 64×64 weight tensors:
//     Y[i, p] = Σ_{j ≤ i, same document} CB[i, j] · exp(cs_i − cs_j) · dt_j · X[j, p]
// per (batch, chunk, head), with CB = C·Bᵀ of the chunk (shared by the heads of a group), cs the inclusive cumulative log-decay
// inside the chunk.  In the reference this is the chunk-scan part of `mamba_chunk_scan_combined` (`lit_gpt/mamba2.py:289-305`);
// as PyTorch ops it is a chain of broadcast / mask / exp / multiply passes over [B, chunks, H, 64, 64] fp32 tensors (268 MB each
// at B8 L4096 H32) plus operand permutes around a batched matmul.
//
// The work is small (2·64·64·P FLOP per problem, ≈ 9 GFLOP per pass at that size), so these are plain fp32 CUDA-core kernels
// with the 64×64 weight matrix and the 64×P operand tile in shared memory:
//   forward   one CTA per (chunk, head, batch): M = CB ∘ E ∘ dt_j (E the masked decay), Y = M·X
//   backward  `hsplit` CTAs per (chunk, group, batch), each looping over its share of the group's heads so that its part of
//             dCB (a sum over heads; the parts are added by the caller) stays in registers:  dM = dY·Xᵀ (masked),  dX = Mᵀ·dY,
//             dCB += dM ∘ E ∘ dt_j,  dcs_i = Σ_j dM∘M − Σ_i' (dM∘M)[i', i],  ddt_j = Σ_i dM ∘ CB ∘ E
// Layouts: x, y, dy, dx [B, Lp, H, P] (x bf16 or fp32 → templated; dy has the type of x; y, dx fp32), dt [B, Lp, H] fp32, cs and dcs [B, nC, H, 64],
// ddt [B, nC, H, 64], CB [B, nC, G, 64, 64] and dCB parts [B, nC, G, hsplit, 64, 64] fp32, bc [B, nC, 64] int32 (document breaks so far inside the chunk) or null.
// Lp = nC·64; P a multiple of 64.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "api.h"

namespace b200 {

constexpr int SI_C = 64;

__device__ __forceinline__ float4 si_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 si_ld4(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// shared: sM[64][65], sX[64][64], s_cs[64], s_dt[64], s_bc[64]
template <typename TX>
__global__ void __launch_bounds__(256) ssd_intra_fwd_kernel(const TX* __restrict__ x, const float* __restrict__ dt,
                                                           const float* __restrict__ cs, const float* __restrict__ CB,
                                                           const int* __restrict__ bc, float* __restrict__ y, int nC, int H, int G,
                                                           int P) {
  __shared__ float sM[SI_C][SI_C + 1];
  __shared__ __align__(16) float sX[SI_C][SI_C];
  __shared__ float s_cs[SI_C], s_dt[SI_C];
  __shared__ int s_bc[SI_C];
  const int n = blockIdx.x, h = blockIdx.y, b = blockIdx.z, g = h / (H / G);
  const int tid = threadIdx.x;
  const size_t Lp = static_cast<size_t>(nC) * SI_C;
  const size_t tok0 = static_cast<size_t>(b) * Lp + static_cast<size_t>(n) * SI_C;
  if (tid < SI_C) {
    s_cs[tid] = cs[((static_cast<size_t>(b) * nC + n) * H + h) * SI_C + tid];
    s_dt[tid] = dt[(tok0 + tid) * H + h];
    s_bc[tid] = bc ? bc[(static_cast<size_t>(b) * nC + n) * SI_C + tid] : 0;
  }
  __syncthreads();
  const float* cb = CB + ((static_cast<size_t>(b) * nC + n) * G + g) * SI_C * SI_C;
  for (int e = tid; e < SI_C * SI_C; e += 256) {
    const int i = e >> 6, j = e & 63;
    float m = 0.f;
    if (j <= i && s_bc[i] == s_bc[j]) m = cb[e] * __expf(s_cs[i] - s_cs[j]) * s_dt[j];
    sM[i][j] = m;
  }
  const int ti = tid >> 4, tp = tid & 15;                  // 4 rows × 4 columns per thread
  for (int p0 = 0; p0 < P; p0 += SI_C) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = ti + 16 * q;
      *reinterpret_cast<float4*>(&sX[j][tp * 4]) = si_ld4(x + ((tok0 + j) * H + h) * P + p0 + tp * 4);
    }
    __syncthreads();
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = 0.f;
    const int jmax = ti * 4 + 3;                           // lower-triangular: nothing beyond the block's last row
    for (int j = 0; j <= jmax; ++j) {
      const float4 xv = *reinterpret_cast<const float4*>(&sX[j][tp * 4]);
      float mv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) mv[a] = sM[ti * 4 + a][j];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        acc[a][0] = fmaf(mv[a], xv.x, acc[a][0]); acc[a][1] = fmaf(mv[a], xv.y, acc[a][1]);
        acc[a][2] = fmaf(mv[a], xv.z, acc[a][2]); acc[a][3] = fmaf(mv[a], xv.w, acc[a][3]);
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
      *reinterpret_cast<float4*>(y + ((tok0 + ti * 4 + a) * H + h) * P + p0 + tp * 4) =
          make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
  }
}

// shared: sM (M), sW (dM, then dM∘M), sX, sDY tiles.  The dM product reads rows of sX and sDY as vectors along p: a row pitch
// of 68 floats and columns j = tp + 16·c per thread put the 16 rows of one load into different banks (with a pitch of 64 and
// j = 4·tp + c all of them met in one bank: the kernel took 1.38 ms at B4 L4096 H62).
constexpr int SI_PX = SI_C + 4;
template <typename TX>
__global__ void __launch_bounds__(256) ssd_intra_bwd_kernel(const TX* __restrict__ x, const float* __restrict__ dt,
                                                           const float* __restrict__ cs, const float* __restrict__ CB,
                                                           const int* __restrict__ bc, const TX* __restrict__ dy,
                                                           float* __restrict__ dx, float* __restrict__ ddt, float* __restrict__ dcs,
                                                           float* __restrict__ dCB, int nC, int H, int G, int P, int hsplit) {
  extern __shared__ __align__(16) float si_dyn[];
  float (*sX)[SI_PX] = reinterpret_cast<float (*)[SI_PX]>(si_dyn);
  float (*sDY)[SI_PX] = sX + SI_C;
  float (*sM)[SI_PX] = sDY + SI_C;                                                       // M = CB∘E∘dt_j
  float (*sW)[SI_C + 1] = reinterpret_cast<float (*)[SI_C + 1]>(&sM[SI_C][0]);           // dM (masked)
  float (*s_col)[2][SI_C] = reinterpret_cast<float (*)[2][SI_C]>(&sW[SI_C][0]);          // column sums of four row classes
  float* s_cs = &s_col[4][0][0];
  float* s_dt = s_cs + SI_C;
  int* s_bc = reinterpret_cast<int*>(s_dt + SI_C);
  // blockIdx.y = group · hsplit + part: the heads of a group are dealt to `hsplit` CTAs, each writes its own partial dCB
  const int n = blockIdx.x, g = blockIdx.y / hsplit, part = blockIdx.y % hsplit, b = blockIdx.z, rep = H / G;
  const int tid = threadIdx.x;
  const int ti = tid >> 4, tp = tid & 15;
  const int ej = tid & 63, er = tid >> 6;                  // entry mapping: column ej, rows er + 4·q
  const size_t Lp = static_cast<size_t>(nC) * SI_C;
  const size_t tok0 = static_cast<size_t>(b) * Lp + static_cast<size_t>(n) * SI_C;
  const float* cb = CB + ((static_cast<size_t>(b) * nC + n) * G + g) * SI_C * SI_C;
  if (tid < SI_C) s_bc[tid] = bc ? bc[(static_cast<size_t>(b) * nC + n) * SI_C + tid] : 0;
  float dcb_acc[16], cbr[16];                              // entries (er + 4·q, ej) of the 64×64 matrix
#pragma unroll
  for (int q = 0; q < 16; ++q) { dcb_acc[q] = 0.f; cbr[q] = cb[(er + 4 * q) * SI_C + ej]; }
  for (int r = part; r < rep; r += hsplit) {
    const int h = g * rep + r;
    __syncthreads();
    if (tid < SI_C) {
      s_cs[tid] = cs[((static_cast<size_t>(b) * nC + n) * H + h) * SI_C + tid];
      s_dt[tid] = dt[(tok0 + tid) * H + h];
    }
    __syncthreads();
    const float csj = s_cs[ej], dtj = s_dt[ej];
    const int bcj = s_bc[ej];
    float ed[16];                                          // masked decay E
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int i = er + 4 * q;
      ed[q] = (ej <= i && s_bc[i] == bcj) ? __expf(s_cs[i] - csj) : 0.f;
      sM[i][ej] = cbr[q] * ed[q] * dtj;
    }
    // dM = Σ_p dY[i, p]·X[j, p] (accumulated over the P blocks), dX = Mᵀ·dY per P block
    float wacc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) wacc[a][c] = 0.f;
    for (int p0 = 0; p0 < P; p0 += SI_C) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = ti + 16 * q;
        const size_t src = ((tok0 + j) * H + h) * P + p0 + tp * 4;
        *reinterpret_cast<float4*>(&sX[j][tp * 4]) = si_ld4(x + src);
        *reinterpret_cast<float4*>(&sDY[j][tp * 4]) = si_ld4(dy + src);
      }
      __syncthreads();
      // this thread's block of dM: rows i = 4·ti + a, columns j = tp + 16·c; column blocks above the diagonal are skipped
      const int cmax = ti >> 2;                            // the same for the two values of ti in a warp
#pragma unroll 4
      for (int p = 0; p < SI_C; p += 4) {
        float4 dv[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) dv[a] = *reinterpret_cast<const float4*>(&sDY[ti * 4 + a][p]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c <= cmax) {
            const float4 xv = *reinterpret_cast<const float4*>(&sX[tp + 16 * c][p]);
#pragma unroll
            for (int a = 0; a < 4; ++a)
              wacc[a][c] += dv[a].x * xv.x + dv[a].y * xv.y + dv[a].z * xv.z + dv[a].w * xv.w;
          }
        }
      }
      // dX[j, p] = Σ_{i ≥ j} M[i, j]·dY[i, p]: rows j = 4·ti + a, columns p = 4·tp + c
      float xacc[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) xacc[a][c] = 0.f;
#pragma unroll 4
      for (int i = ti * 4; i < SI_C; ++i) {
        const float4 dv = *reinterpret_cast<const float4*>(&sDY[i][tp * 4]);
        const float4 m4 = *reinterpret_cast<const float4*>(&sM[i][ti * 4]);
        const float mv[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          xacc[a][0] = fmaf(mv[a], dv.x, xacc[a][0]); xacc[a][1] = fmaf(mv[a], dv.y, xacc[a][1]);
          xacc[a][2] = fmaf(mv[a], dv.z, xacc[a][2]); xacc[a][3] = fmaf(mv[a], dv.w, xacc[a][3]);
        }
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
        *reinterpret_cast<float4*>(dx + ((tok0 + ti * 4 + a) * H + h) * P + p0 + tp * 4) =
            make_float4(xacc[a][0], xacc[a][1], xacc[a][2], xacc[a][3]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) sW[ti * 4 + a][tp + 16 * c] = wacc[a][c];
    __syncthreads();
    // per-entry products; column sums of dM∘CB∘E (→ ddt) and dM∘M in registers, dM∘M back to sW for the row sums
    float col_dt = 0.f, col_w = 0.f;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int i = er + 4 * q;
      const float w = ed[q] != 0.f ? sW[i][ej] : 0.f;      // outside the mask (and where the decay vanishes) dM does not enter
      const float wce = w * cbr[q] * ed[q];
      dcb_acc[q] += w * ed[q] * dtj;
      col_dt += wce;
      col_w += wce * dtj;
      sW[i][ej] = wce * dtj;
    }
    s_col[er][0][ej] = col_w;
    s_col[er][1][ej] = col_dt;
    __syncthreads();
    {
      const int row = tid >> 2, k0 = (tid & 3) * 16;       // four threads per row
      float rs = 0.f;
#pragma unroll
      for (int k = 0; k < 16; ++k) rs += sW[row][k0 + k];
      rs += __shfl_xor_sync(0xffffffffu, rs, 1);
      rs += __shfl_xor_sync(0xffffffffu, rs, 2);
      if ((tid & 3) == 0) {
        const size_t o = ((static_cast<size_t>(b) * nC + n) * H + h) * SI_C + row;
        dcs[o] = rs - ((s_col[0][0][row] + s_col[1][0][row]) + (s_col[2][0][row] + s_col[3][0][row]));
        ddt[o] = (s_col[0][1][row] + s_col[1][1][row]) + (s_col[2][1][row] + s_col[3][1][row]);
      }
    }
  }
  float* out = dCB + (((static_cast<size_t>(b) * nC + n) * G + g) * hsplit + part) * SI_C * SI_C;
#pragma unroll
  for (int q = 0; q < 16; ++q) out[(er + 4 * q) * SI_C + ej] = dcb_acc[q];
}

constexpr int SI_BWD_SMEM = (3 * SI_C * SI_PX + SI_C * (SI_C + 1) + 8 * SI_C + 2 * SI_C) * 4 + SI_C * 4;

}  // namespace b200

// x_dtype: 0 fp32, 1 bf16.  See the top of the file for the layouts.
extern "C" int b200_ssd_intra_fwd(const void* x, int x_dtype, const float* dt, const float* cs, const float* CB, const int* bc,
                                  float* y, int B, int nC, int H, int G, int P, cudaStream_t st) {
  using namespace b200;
  if (B <= 0 || nC <= 0) return 0;
  if (P % SI_C || H % G) return -1;
  const dim3 grid(nC, H, B);
  if (x_dtype == 1)
    ssd_intra_fwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x), dt, cs, CB, bc, y, nC, H, G, P);
  else
    ssd_intra_fwd_kernel<float><<<grid, 256, 0, st>>>(static_cast<const float*>(x), dt, cs, CB, bc, y, nC, H, G, P);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

extern "C" int b200_ssd_intra_bwd(const void* x, int x_dtype, const float* dt, const float* cs, const float* CB, const int* bc,
                                  const void* dy, float* dx, float* ddt, float* dcs, float* dCB, int B, int nC, int H, int G,
                                  int P, int hsplit, cudaStream_t st) {
  using namespace b200;
  if (B <= 0 || nC <= 0) return 0;
  if (P % SI_C || H % G || hsplit < 1 || (H / G) % hsplit) return -1;
  const dim3 grid(nC, G * hsplit, B);
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(ssd_intra_bwd_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, SI_BWD_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(ssd_intra_bwd_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, SI_BWD_SMEM) != cudaSuccess)
      return -2;
    configured = true;
  }
  if (x_dtype == 1)
    ssd_intra_bwd_kernel<__nv_bfloat16><<<grid, 256, SI_BWD_SMEM, st>>>(static_cast<const __nv_bfloat16*>(x), dt, cs, CB, bc, static_cast<const __nv_bfloat16*>(dy), dx,
                                                                       ddt, dcs, dCB, nC, H, G, P, hsplit);
  else
    ssd_intra_bwd_kernel<float><<<grid, 256, SI_BWD_SMEM, st>>>(static_cast<const float*>(x), dt, cs, CB, bc, static_cast<const float*>(dy), dx, ddt, dcs, dCB,
                                                               nC, H, G, P, hsplit);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}
