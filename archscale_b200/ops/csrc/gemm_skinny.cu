// Few tokens times a weight matrix: out[M, N] = X[M, K] · Wᵀ for M of a few dozen rows (one decoding step that runs the prefix
// again, log-likelihood of a short request), without gradients.
//
// Such a product is bound by reading the weights (5632 × 1024: 11.5 MB, 1.8 µs at the copy rate) and, at this size, by the latency of
// one CTA's chain of loads and by the launches around it.  So the weight rows are the M side of the MMA (128 of them per tile)
// and the tokens its N side (64, rows past the end are zero-filled by the loads), and the K dimension is split over a cluster
// of up to eight CTAs, which adds CTAs where N alone gives few (1024 rows: 8 tiles) and shortens the chain.  The first loads are
// issued before tensor memory is allocated.  The partial products of a cluster meet in shared memory, in the place of the stages
// (two CTAs fit an SM, so clusters of eight find a place): every CTA adds its share of the tokens over the CTAs in rank order
// (distributed shared memory, the loads of all ranks in flight at once), so a result does not depend on scheduling.  One launch
// takes up to three weight matrices that share X (the query / key / value projections, written as column blocks of one
// output) or a SwiGLU pair (gate rows first).
// At 41 tokens, µs in a graph (weights not in the L2), with one rank's load after the other and one CTA per SM / now / library:
// 1024x1024 6.9 / 5.6 / 4.2, 5632x1024 9.2 / 8.1 / 5.4, 1024x2816 8.2 / 7.0 / 6.4, 2048x2048 14.2 / 7.5 / 5.8, 32000x1024 24.4 / 16.9 /
// 16.2; query, key and value of 1024, 256, 256 x 1024 7.0 / 5.8 / 12.1 (three launches); SwiGLU of 2 x 2816 x 1024 9.3 / 7.9 / 7.4 (with the
// activation's launch), 2 x 5632 x 2048 17.2 / 15.2 / 14.3.  A layer of a 41-token pass takes 26 µs in these four products, the
// library's seven launches 30.
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
constexpr int SKY_PART = SKY_BT * SKY_BN * 4;          // fp32 partial product [token][weight row], over the stages once they are read
constexpr int SKY_SMEM = SKY_STAGES * SKY_STAGE + 1024 + 256;
constexpr int SKY_THREADS = 192;
static_assert(SKY_PART <= SKY_STAGES * SKY_STAGE, "the partial product takes the place of the stages");

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
// Four columns of the partial products of all ranks, added in rank order; the loads are all in flight before the first is used.
template <int S>
__device__ __forceinline__ float4 sum_cluster_f4(uint32_t smem_addr) {
  float4 v[S];
#pragma unroll
  for (int r = 0; r < S; ++r) v[r] = ld_cluster_f4(smem_addr, r);
#pragma unroll
  for (int r = 1; r < S; ++r) { v[0].x += v[r].x; v[0].y += v[r].y; v[0].z += v[r].z; v[0].w += v[r].w; }
  return v[0];
}

template <int S>      // CTAs of a cluster
__global__ void __launch_bounds__(SKY_THREADS, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w0,
                   const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2, const SkinnyParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* part = reinterpret_cast<float*>(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SKY_STAGES * SKY_STAGE);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + SKY_STAGES;
  uint64_t* done_bar = bars + 2 * SKY_STAGES;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 2 * SKY_STAGES + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = S > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = static_cast<int>(blockIdx.x) / S;
  const int wi = (p.n[2] > 0 && tile >= p.tile0[2]) ? 2 : (p.n[1] > 0 && tile >= p.tile0[1]) ? 1 : 0;
  const int rows = p.swiglu ? SKY_BN / 2 : SKY_BN;      // output columns of this tile
  const int n0 = (tile - (wi == 2 ? p.tile0[2] : wi == 1 ? p.tile0[1] : p.tile0[0])) * rows;
  const int num_kb = (p.K + SKY_BK - 1) / SKY_BK, per = (num_kb + S - 1) / S;
  const int kb0 = min(rank * per, num_kb), kb1 = min(kb0 + per, num_kb);      // the last ranks may have no share
  const CUtensorMap* tw = wi == 0 ? &tmap_w0 : wi == 1 ? &tmap_w1 : &tmap_w2;

  auto load = [&](int kb, int st) {
    uint8_t* sa = smem + st * SKY_STAGE;
    mbar_arrive_expect_tx(&full_bar[st], SKY_STAGE);
    // weight rows in two boxes of 64: for SwiGLU the second one holds the up rows of the same columns
    tma_load_2d(sa, tw, &full_bar[st], kb * SKY_BK, n0);
    tma_load_2d(sa + SKY_A / 2, tw, &full_bar[st], kb * SKY_BK, p.swiglu ? p.n[0] + n0 : n0 + SKY_BN / 2);
    tma_load_2d(sa + SKY_A, &tmap_x, &full_bar[st], kb * SKY_BK, 0);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < SKY_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async_smem();
    for (int i = 0; i < SKY_STAGES && kb0 + i < kb1; ++i) load(kb0 + i, i);     // the ring is empty: no wait, and under the set-up
  }
  if (warp == 1) { tmem_alloc(tmem_ptr, SKY_BT); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr, 0);

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0 + SKY_STAGES, i = SKY_STAGES; kb < kb1; ++kb, ++i) {
        const int st = i % SKY_STAGES; const uint32_t ph = (i / SKY_STAGES) & 1;
        if (!mbar_wait(&empty_bar[st], ph ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY)) break;
        load(kb, st);
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
    // every product has been read from the stages when this barrier flips (all loads have landed before that)
    const bool share = kb1 > kb0 && mbar_wait_warp(done_bar, 0, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL);
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < SKY_BT / 32; ++c) {
      if (c * 32 < p.M) {
        uint32_t r[32];
        if (share) {
          tmem_ld_32x32(tmem_base + c * 32 + (static_cast<uint32_t>(q * 32) << 16), r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = 0u;
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) part[(c * 32 + e) * SKY_BN + row] = __uint_as_float(r[e]);
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (S > 1) cluster_sync_all();                         // every partial product of the cluster is in shared memory
  {
    const uint32_t pa = smem_u32(part);
    const int vecs = rows / 4, n_lim = wi == 2 ? p.n[2] : wi == 1 ? p.n[1] : p.n[0];
    const int col0 = (wi == 2 ? p.col0[2] : wi == 1 ? p.col0[1] : p.col0[0]) + n0;
    for (int v = threadIdx.x; v < SKY_BT / S * vecs; v += SKY_THREADS) {
      const int tok = v / vecs * S + rank, c = (v % vecs) * 4, n = n0 + c;      // token r, r + S, … are rank r's to add
      if (tok >= p.M) break;
      if (n >= n_lim) continue;
      const uint32_t off = pa + (tok * SKY_BN + c) * 4;
      const float4 a = sum_cluster_f4<S>(off);
      uint2 o = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
      if (p.swiglu) {                                    // on the values rounded to bf16, as the unfused pair computes it
        const float4 u = sum_cluster_f4<S>(off + SKY_BN / 2 * 4);
        const float2 g0 = unpack_bf16x2(o.x), g1 = unpack_bf16x2(o.y);
        const float2 u0 = unpack_bf16x2(pack_bf16x2(u.x, u.y)), u1 = unpack_bf16x2(pack_bf16x2(u.z, u.w));
        o.x = pack_bf16x2(g0.x * (1.f / (1.f + __expf(-g0.x))) * u0.x, g0.y * (1.f / (1.f + __expf(-g0.y))) * u0.y);
        o.y = pack_bf16x2(g1.x * (1.f / (1.f + __expf(-g1.x))) * u1.x, g1.y * (1.f / (1.f + __expf(-g1.y))) * u1.y);
      }
      *reinterpret_cast<uint2*>(p.out + static_cast<size_t>(tok) * p.ldo + col0 + c) = o;
    }
  }
  if (S > 1) cluster_sync_all();                         // no CTA leaves while another reads its shared memory
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, SKY_BT);
  }
}

template <int S>
static int launch_skinny(const CUtensorMap& tx, const CUtensorMap (&tw)[3], const SkinnyParams& p, int tiles, cudaStream_t stream) {
  auto kern = gemm_skinny_kernel<S>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SKY_SMEM) != cudaSuccess) return -2;
    configured = true;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * S);
  cfg.blockDim = dim3(SKY_THREADS);
  cfg.dynamicSmemBytes = SKY_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, tx, tw[0], tw[1], tw[2], p) == cudaSuccess ? 0 : -3;
}

}  // namespace b200

// out[M, Σ n_w] = X[M, K] · [W_0; W_1; …]ᵀ (bf16, fp32 sums), or with swiglu and one W = [gate; up] of 2·n rows: out[M, n] =
// silu(gate)·up.  X, W: rows of K elements, K and every n multiples of 8, 16-byte aligned, row strides ldx, ldw multiples of 8.
extern "C" int b200_gemm_skinny(const void* X, const void* const* W, const int* n_w, int n_mats, int swiglu, void* out, int M, int K,
                                int ldx, const int* ldw, int ldo, int num_sms, int* status, cudaStream_t stream) {
  using namespace b200;
  if (M <= 0) return 0;
  if (M > SKY_BT || K <= 0 || n_mats < 1 || n_mats > 3 || (swiglu && n_mats != 1)) return -1;
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
  const int num_kb = (K + SKY_BK - 1) / SKY_BK;
  // (More CTAs than SMs, two of them on some: 5632x1024 7.7 against 8.1 µs, SwiGLU 2 x 5632 x 2048 13.9 against 15.2, but 3072x2048 8.3 against
  // 8.1, and another order of the sums.)
  int S = 1;
  while (S < 8 && tiles * S * 2 <= num_sms && S * 2 <= num_kb) S *= 2;
  switch (S) {
    case 8: return launch_skinny<8>(tx, tw, p, tiles, stream);
    case 4: return launch_skinny<4>(tx, tw, p, tiles, stream);
    case 2: return launch_skinny<2>(tx, tw, p, tiles, stream);
    default: return launch_skinny<1>(tx, tw, p, tiles, stream);
  }
}
