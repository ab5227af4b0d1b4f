// Few tokens times a weight matrix: out[M, N] = X[M, K] · Wᵀ for M of a few dozen rows (one decoding step that runs the prefix
// again, log-likelihood of a short request), without gradients.
//
// Such a product is bound by reading the weights (5632 × 1024: 11.5 MB, 1.8 µs at the copy rate) and, at this size, by the latency of
// one CTA's chain of loads and by the launches around it.  So the weight rows are the M side of the MMA (128 of them per tile)
// and the tokens its N side (64, rows past the end are zero-filled by the loads), and the K dimension is split over a cluster
// of up to eight CTAs, which adds CTAs where N alone gives few (1024 rows: 8 tiles) and shortens the chain.  The partial
// products of a cluster meet in shared memory: every CTA adds its share of the tokens over the CTAs in rank order (distributed
// shared memory), so a result does not depend on scheduling.  One launch takes up to three weight matrices that share X (the
// query / key / value projections, written as column blocks of one output) or a SwiGLU pair (gate rows first).
// At 41 tokens, µs in a graph (weights not in the L2), this kernel / library: 1024x1024 6.3 / 3.8, 5632x1024 9.2 / 5.3, 1024x2816
// 8.2 / 6.4, 32000x1024 23 / 15: the library's kernels are faster on the device, but such a pass is bound by the host, and
// there one call takes 5 µs instead of 10 and replaces up to three products (or a product and the activation).
//
// 192 threads: warp 0 TMA, warp 1 MMA, warps 2..5 tensor memory → shared memory (thread = weight row); all of them add.
#include "sm100.cuh"
#include "api.h"

namespace b200 {

int make_tmap_2d_bf16(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_elems,
                      uint32_t box_inner, uint32_t box_outer);

constexpr int SKY_BN = 128, SKY_BT = 64, SKY_BK = 64;
constexpr int SKY_STAGES = 4;
constexpr int SKY_A = SKY_BN * SKY_BK * 2, SKY_B = SKY_BT * SKY_BK * 2, SKY_STAGE = SKY_A + SKY_B;
constexpr int SKY_PART = SKY_BT * SKY_BN * 4;          // fp32 partial product [token][weight row]
constexpr int SKY_SMEM = SKY_STAGES * SKY_STAGE + SKY_PART + 1024 + 256;
constexpr int SKY_THREADS = 192;

struct SkinnyParams {
  __nv_bfloat16* out;      // [M, ldo]
  int M, K, ldo;
  int n[3];                // rows of the weight matrices (0: none); swiglu: n[0] = gate rows = up rows
  int tile0[3];            // first tile of each matrix
  int col0[3];             // its first output column
  int swiglu;
  int* status;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t smem_addr, int rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

__global__ void __launch_bounds__(SKY_THREADS, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w0,
                   const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2, const SkinnyParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* part = reinterpret_cast<float*>(smem + SKY_STAGES * SKY_STAGE);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SKY_STAGES * SKY_STAGE + SKY_PART);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + SKY_STAGES;
  uint64_t* done_bar = bars + 2 * SKY_STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 2 * SKY_STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  uint32_t nrank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(nrank));
  const int S = static_cast<int>(nrank), rank = static_cast<int>(cluster_ctarank());
  const int tile = static_cast<int>(blockIdx.x) / S, t0 = static_cast<int>(blockIdx.y) * SKY_BT;
  const int wi = (p.n[2] > 0 && tile >= p.tile0[2]) ? 2 : (p.n[1] > 0 && tile >= p.tile0[1]) ? 1 : 0;
  const int rows = p.swiglu ? SKY_BN / 2 : SKY_BN;      // output columns of this tile
  const int n0 = (tile - p.tile0[wi]) * rows;
  const int num_kb = (p.K + SKY_BK - 1) / SKY_BK, per = (num_kb + S - 1) / S;
  const int kb0 = min(rank * per, num_kb), kb1 = min(kb0 + per, num_kb);

  if (threadIdx.x == 0) {
    for (int s = 0; s < SKY_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_ptr, SKY_BT); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr, 0);

  if (warp == 0) {
    if (lane == 0) {
      const CUtensorMap* tw = wi == 0 ? &tmap_w0 : wi == 1 ? &tmap_w1 : &tmap_w2;
      for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
        const int st = i % SKY_STAGES; const uint32_t ph = (i / SKY_STAGES) & 1;
        if (!mbar_wait(&empty_bar[st], ph ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY)) break;
        uint8_t* sa = smem + st * SKY_STAGE;
        mbar_arrive_expect_tx(&full_bar[st], SKY_STAGE);
        // weight rows in two boxes of 64: for SwiGLU the second one holds the up rows of the same columns
        tma_load_2d(sa, tw, &full_bar[st], kb * SKY_BK, n0);
        tma_load_2d(sa + SKY_A / 2, tw, &full_bar[st], kb * SKY_BK, p.swiglu ? p.n[0] + n0 : n0 + SKY_BN / 2);
        tma_load_2d(sa + SKY_A, &tmap_x, &full_bar[st], kb * SKY_BK, t0);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(SKY_BN, SKY_BT, 0, 0);
    bool ok = true;
    for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
      const int st = i % SKY_STAGES; const uint32_t ph = (i / SKY_STAGES) & 1;
      if (!mbar_wait_warp(&full_bar[st], ph, abort_flag, p.status, STATUS_TIMEOUT_FULL)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sa = smem_u32(smem + st * SKY_STAGE);
#pragma unroll
      for (int k = 0; k < SKY_BK / 16; ++k)
        umma_bf16_warp(tmem_base, make_smem_desc(sa + k * 32, 16, 1024), make_smem_desc(sa + SKY_A + k * 32, 16, 1024), idesc, (i | k) != 0);
      umma_commit_warp(&empty_bar[st]);
    }
    if (ok && kb1 > kb0) umma_commit_warp(done_bar);
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;
    bool ok = true;
    if (kb1 > kb0) ok = mbar_wait_warp(done_bar, 0, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL);
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < SKY_BT / 32; ++c) {
      uint32_t r[32];
      if (ok && kb1 > kb0) {
        tmem_ld_32x32(tmem_base + c * 32 + (static_cast<uint32_t>(q * 32) << 16), r);
        tmem_ld_wait();
      } else {                                           // a rank without a share of K
#pragma unroll
        for (int e = 0; e < 32; ++e) r[e] = 0u;
      }
#pragma unroll
      for (int e = 0; e < 32; ++e) part[(c * 32 + e) * SKY_BN + row] = __uint_as_float(r[e]);
    }
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync_all();                                    // every partial product of the cluster is in shared memory
  {
    const uint32_t pa = smem_u32(part);
    const int tok_per = SKY_BT / S;                      // this CTA adds tokens rank·tok_per ..
    const int vecs = rows / 4;
    const int n_lim = p.n[wi];
    for (int v = threadIdx.x; v < tok_per * vecs; v += SKY_THREADS) {
      const int tk = rank * tok_per + v / vecs, c = (v % vecs) * 4;
      const int tok = t0 + tk, n = n0 + c;
      if (tok >= p.M || n >= n_lim) continue;
      const uint32_t off = pa + (tk * SKY_BN + c) * 4;
      float4 a = ld_cluster_f4(off, 0);
      for (int r = 1; r < S; ++r) {
        const float4 b = ld_cluster_f4(off, r);
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
      }
      uint2 o = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
      if (p.swiglu) {                                    // on the values rounded to bf16, as the unfused pair computes it
        float4 u = ld_cluster_f4(off + SKY_BN / 2 * 4, 0);
        for (int r = 1; r < S; ++r) {
          const float4 b = ld_cluster_f4(off + SKY_BN / 2 * 4, r);
          u.x += b.x; u.y += b.y; u.z += b.z; u.w += b.w;
        }
        const float2 g0 = unpack_bf16x2(o.x), g1 = unpack_bf16x2(o.y);
        const float2 u0 = unpack_bf16x2(pack_bf16x2(u.x, u.y)), u1 = unpack_bf16x2(pack_bf16x2(u.z, u.w));
        o.x = pack_bf16x2(g0.x * (1.f / (1.f + __expf(-g0.x))) * u0.x, g0.y * (1.f / (1.f + __expf(-g0.y))) * u0.y);
        o.y = pack_bf16x2(g1.x * (1.f / (1.f + __expf(-g1.x))) * u1.x, g1.y * (1.f / (1.f + __expf(-g1.y))) * u1.y);
      }
      *reinterpret_cast<uint2*>(p.out + static_cast<size_t>(tok) * p.ldo + p.col0[wi] + n) = o;
    }
  }
  cluster_sync_all();                                    // no CTA leaves while another reads its shared memory
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, SKY_BT);
  }
}

}  // namespace b200

// out[M, Σ n_w] = X[M, K] · [W_0; W_1; …]ᵀ (bf16, fp32 sums), or with swiglu and one W = [gate; up] of 2·n rows: out[M, n] =
// silu(gate)·up.  X, W: rows of K elements, K and every n multiples of 8, 16-byte aligned, row strides ldx, ldw multiples of 8.
extern "C" int b200_gemm_skinny(const void* X, const void* const* W, const int* n_w, int n_mats, int swiglu, void* out, int M, int K,
                                int ldx, const int* ldw, int ldo, int num_sms, int* status, cudaStream_t stream) {
  using namespace b200;
  if (M <= 0) return 0;
  if (K <= 0 || n_mats < 1 || n_mats > 3 || (swiglu && n_mats != 1)) return -1;
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) return -5;
    ctx_bound = true;
  }
  CUtensorMap tx, tw[3];
  int rc = make_tmap_2d_bf16(&tx, X, K, M, ldx, SKY_BK, SKY_BT);
  if (rc) return rc;
  SkinnyParams p{};
  p.out = static_cast<__nv_bfloat16*>(out);
  p.M = M; p.K = K; p.ldo = ldo; p.swiglu = swiglu; p.status = status;
  int tiles = 0, col = 0;
  for (int i = 0; i < 3; ++i) {
    const int j = i < n_mats ? i : 0;
    const int wrows = n_w[j];                            // rows of the matrix
    rc = make_tmap_2d_bf16(&tw[i], W[j], K, wrows, ldw[j], SKY_BK, SKY_BN / 2);
    if (rc) return rc;
    if (i >= n_mats) continue;
    const int n = swiglu ? wrows / 2 : wrows, rows = swiglu ? SKY_BN / 2 : SKY_BN;
    p.n[i] = n; p.tile0[i] = tiles; p.col0[i] = col;
    tiles += (n + rows - 1) / rows;
    col += n;
  }
  const int tt = (M + SKY_BT - 1) / SKY_BT, num_kb = (K + SKY_BK - 1) / SKY_BK;
  int S = 1;
  // clusters of eight only for one block of tokens: two blocks of 1024 rows took 12 µs with them and 7 with clusters of four
  while (S < (tt == 1 ? 8 : 4) && tiles * tt * S * 2 <= num_sms && S * 2 <= num_kb) S *= 2;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SKY_SMEM) != cudaSuccess) return -2;
    configured = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * S, tt);
  cfg.blockDim = dim3(SKY_THREADS);
  cfg.dynamicSmemBytes = SKY_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gemm_skinny_kernel, tx, tw[0], tw[1], tw[2], p) == cudaSuccess ? 0 : -3;
}
