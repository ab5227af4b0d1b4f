// MXFP8 block-scaled GEMM on SM pairs (tcgen05.mma.cta_group::2 …block_scale): out[M,N] = alpha · (A ⊙ sfA) · (B ⊙ sfB)ᵀ, the
// operands, scale layout and epilogue of gemm_mxfp8.cu.
//
// Two CTAs share a 256 × NT tile: each stages its 128 rows of A, half of the rows of B, its own A scales and all of the tile's
// B scales (both SMs multiply all NT columns); the leader issues the products and the scale copies for both.  The one-CTA
// kernel moves 40 KB into shared memory per 128 × 192 × 128 step, 105 bytes per cycle beside as many for the operand reads,
// and was held up by that; a pair moves 28 KB per CTA for the same products.  NT is 192 (two accumulators and the scale columns fit
// the 512 columns of tensor memory) or 128 where that needs no more waves of pairs.  A step costs ≈730 cycles at NT 192 and
// ≈670 at 128, of which the products are 390 and 260: the rest is what the instructions of a step take.  (Copying the scales of a step
// before the products of the step before it, into a second set of columns, was slower: 16384x11264x2048 0.334 against 0.313 ms.)
#include "api.h"
#include "sm100.cuh"

namespace b200 {

constexpr int M2_BK = 128, M2_THREADS = 192, M2_GROUP_M = 8;
constexpr int M2_TMEM_SFA = 384, M2_TMEM_SFB = 392;              // columns after the two accumulators

template <int NT>
struct Mx2 {
  static constexpr int A_BYTES = 128 * M2_BK, B_BYTES = NT / 2 * M2_BK;
  static constexpr int SF_CHUNKS = NT > 128 ? 2 : 1;             // 128-row scale chunks a B tile touches
  static constexpr int SFA_OFF = A_BYTES + B_BYTES, SFB_OFF = SFA_OFF + 512;
  static constexpr int LOAD_BYTES = SFB_OFF + SF_CHUNKS * 512;
  static constexpr int STAGE_BYTES = (LOAD_BYTES + 1023) / 1024 * 1024;
  static constexpr int STAGES = 7;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;
};

struct Mx2Params {
  void* out;
  int M, N, K, ldc;
  float alpha;
  int accumulate;
  int* status;
};

// Unswizzled K-major descriptor of a 32-row × 16-byte scale chunk: 8-row groups are 128 bytes apart.
__device__ __forceinline__ uint64_t mx2_sf_desc(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4) | (static_cast<uint64_t>(128 >> 4) << 32) | (static_cast<uint64_t>(1) << 46);
}
// Scale chunk from each CTA's shared memory (same offset) into its own tensor memory.
__device__ __forceinline__ void mx2_cp_sf(uint32_t taddr, uint64_t desc) {
  if (elect_one_sync()) asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
__device__ __forceinline__ void mx2_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t tsfa, uint32_t tsfb,
                                        uint32_t accumulate) {
  if (elect_one_sync())
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n"
        "}\n" ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(tsfa), "r"(tsfb)
        : "memory");
}

template <int NT, int OUT_F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(M2_THREADS, 1)
gemm2_mxfp8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                   const __grid_constant__ CUtensorMap tmap_sfa, const __grid_constant__ CUtensorMap tmap_sfb, const Mx2Params p) {
  using T = Mx2<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + T::STAGES * T::STAGE_BYTES);
  uint64_t* full_bar = bars;                          // [STAGES]  used in the leader CTA
  uint64_t* empty_bar = bars + T::STAGES;             // [STAGES]  each CTA's producer waits on its own
  uint64_t* tmem_full = bars + 2 * T::STAGES;         // [2]       each CTA's epilogue waits on its own
  uint64_t* tmem_empty = bars + 2 * T::STAGES + 2;    // [2]       used in the leader CTA, 8 arrivals (4 warps × 2 CTAs)
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 2 * T::STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x) >> 1, n_pair = static_cast<int>(gridDim.x) >> 1;
  const int num_m = (p.M + 255) / 256, num_n = (p.N + NT - 1) / NT;
  const int num_tiles = num_m * num_n;
  const int KC = p.K / M2_BK;                         // K chunks of 128 elements = 4 scale blocks

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], 8); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a); tma_prefetch_desc(&tmap_b); tma_prefetch_desc(&tmap_sfa); tma_prefetch_desc(&tmap_sfb);
  }
  if (warp == 1) { tmem_alloc_2sm(tmem_ptr, 512); tmem_relinquish_2sm(); }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the peer's barriers are initialised before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr, 0);

  auto tile_coords = [&](int t, int& m0, int& n0) {
    const int per_group = M2_GROUP_M * num_n;
    const int g = t / per_group, first_m = g * M2_GROUP_M;
    const int gsz = min(num_m - first_m, M2_GROUP_M);
    const int r = t - g * per_group;
    m0 = (first_m + (r % gsz)) * 256;
    n0 = (r / gsz) * NT;
  };

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      for (int t = pair; t < num_tiles; t += n_pair) {
        int m0, n0; tile_coords(t, m0, n0);
        const int ma = m0 + rank * 128, nb = n0 + rank * (NT / 2);
        const int ca = (ma >> 7) * KC, cb = (n0 >> 7) * KC;      // first scale chunk of the rows (past the end: zero-filled)
        for (int kb = 0; kb < KC; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY)) goto done;
          uint8_t* sa = smem + stage * T::STAGE_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[stage], 2 * T::LOAD_BYTES);   // both CTAs' loads
          tma_load_2d_2sm(sa, &tmap_a, &full_bar[stage], kb * M2_BK, ma);
          tma_load_2d_2sm(sa + T::A_BYTES, &tmap_b, &full_bar[stage], kb * M2_BK, nb);
          tma_load_2d_2sm(sa + T::SFA_OFF, &tmap_sfa, &full_bar[stage], 0, ca + kb);
#pragma unroll
          for (int c = 0; c < T::SF_CHUNKS; ++c)
            tma_load_2d_2sm(sa + T::SFB_OFF + c * 512, &tmap_sfb, &full_bar[stage], 0, cb + c * KC + kb);
          if (++stage == T::STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {                                   // the whole warp, converged: one lane is elected per instruction
      // e4m3 × e4m3, E8M0 scales, fp32 accumulate, both operands K-major
      constexpr uint32_t idesc0 = (static_cast<uint32_t>(NT >> 3) << 17) | (1u << 23) | (static_cast<uint32_t>(256 >> 4) << 24);
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      for (int t = pair; t < num_tiles; t += n_pair, ++it) {
        const int acc = it & 1; const uint32_t acc_phase = (it >> 1) & 1;
        if (!mbar_wait_warp(&tmem_empty[acc], acc_phase ^ 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_EMPTY)) goto done;
        tc_fence_after();
        int m0, n0; tile_coords(t, m0, n0);
        const uint32_t d_tmem = tmem_base + acc * NT;
        const uint32_t tsfa = tmem_base + M2_TMEM_SFA;
        const uint32_t tsfb = tmem_base + M2_TMEM_SFB + ((n0 >> 5) & 3);   // 0 or 2: rows 64.. of the first chunk
        for (int kb = 0; kb < KC; ++kb) {
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.status, STATUS_TIMEOUT_FULL)) goto done;
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * T::STAGE_BYTES);
          mx2_cp_sf(tmem_base + M2_TMEM_SFA, mx2_sf_desc(sa + T::SFA_OFF));
#pragma unroll
          for (int c = 0; c < T::SF_CHUNKS; ++c)
            mx2_cp_sf(tmem_base + M2_TMEM_SFB + 4 * c, mx2_sf_desc(sa + T::SFB_OFF + 512 * c));
          const uint64_t da = make_smem_desc(sa, 16, 1024), db = make_smem_desc(sa + T::A_BYTES, 16, 1024);
#pragma unroll
          for (uint32_t k = 0; k < M2_BK / 32; ++k)    // K-block k: operands advance 32 bytes, byte k of each scale column is used
            mx2_mma(d_tmem, da + static_cast<uint64_t>(k * 2), db + static_cast<uint64_t>(k * 2), idesc0 | (k << 4) | (k << 29),
                    tsfa | (k << 30), tsfb | (k << 30), (kb != 0 || k != 0) ? 1u : 0u);
          if (elect_one_sync()) umma_commit_2sm(&empty_bar[stage], 3);      // frees the stage in both CTAs
          if (++stage == T::STAGES) { stage = 0; phase ^= 1; }
        }
        if (elect_one_sync()) umma_commit_2sm(&tmem_full[acc], 3);          // both CTAs' epilogues may read their half
      }
    }
  } else {
    const int q = warp & 3;
    const bool wide = p.ldc % (OUT_F32 ? 8 : 16) == 0 && reinterpret_cast<uintptr_t>(p.out) % 32 == 0;   // whole sectors per lane
    int it = 0;
    for (int t = pair; t < num_tiles; t += n_pair, ++it) {
      int m0, n0; tile_coords(t, m0, n0);
      const int acc = it & 1; const uint32_t acc_phase = (it >> 1) & 1;
      if (!mbar_wait(&tmem_full[acc], acc_phase, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) goto done;
      tc_fence_after();
      const int row = m0 + rank * 128 + q * 32 + lane;
      const uint32_t taddr = tmem_base + acc * NT + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < NT / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        tmem_ld_wait();
        const int col = n0 + c * 32;
        if (row < p.M && col < p.N) {
          const size_t at = static_cast<size_t>(row) * p.ldc + col;
          if (OUT_F32) store_row32(reinterpret_cast<float*>(p.out) + at, r, p.alpha, p.accumulate, p.N - col, wide);
          else store_row32(reinterpret_cast<__nv_bfloat16*>(p.out) + at, r, p.alpha, p.N - col, wide);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&tmem_empty[acc]);
    }
  }

done:
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, 512);
  }
}

int make_tmap_2d_u8(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                    uint32_t box_inner, uint32_t box_outer);
int make_tmap_sf_chunks(CUtensorMap* map, const void* ptr, uint64_t chunks);

template <int NT, int OUT_F32>
static int launch_mx2(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tsa, const CUtensorMap& tsb, const Mx2Params& p,
                      int num_sms, cudaStream_t st) {
  auto kern = gemm2_mxfp8_kernel<NT, OUT_F32>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Mx2<NT>::SMEM) != cudaSuccess) return -2;
    configured = true;
  }
  const int tiles = ((p.M + 255) / 256) * ((p.N + NT - 1) / NT), pairs = num_sms / 2;
  kern<<<2 * (tiles < pairs ? tiles : pairs), M2_THREADS, Mx2<NT>::SMEM, st>>>(ta, tb, tsa, tsb, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace b200

// Contract of b200_gemm_mxfp8, which checks the arguments and calls this.  nt: 192 or 128.
extern "C" int b200_gemm2_mxfp8(const void* A, const void* sfa, const void* B, const void* sfb, void* out, int M, int N, int K, int lda,
                                int ldb, int ldc, float alpha, int out_f32, int accumulate, int nt, int num_sms, int* status,
                                cudaStream_t stream) {
  using namespace b200;
  CUtensorMap ta, tb, tsa, tsb;
  int rc = make_tmap_2d_u8(&ta, A, K, M, lda, M2_BK, 128);
  if (rc) return rc;
  rc = make_tmap_2d_u8(&tb, B, K, N, ldb, M2_BK, nt / 2);
  if (rc) return rc;
  const uint64_t kc = K / M2_BK;
  rc = make_tmap_sf_chunks(&tsa, sfa, static_cast<uint64_t>((M + 127) / 128) * kc);
  if (rc) return rc;
  rc = make_tmap_sf_chunks(&tsb, sfb, static_cast<uint64_t>((N + 127) / 128) * kc);
  if (rc) return rc;
  const Mx2Params p{out, M, N, K, ldc, alpha, accumulate, status};
  if (nt == 192)
    return out_f32 ? launch_mx2<192, 1>(ta, tb, tsa, tsb, p, num_sms, stream) : launch_mx2<192, 0>(ta, tb, tsa, tsb, p, num_sms, stream);
  return out_f32 ? launch_mx2<128, 1>(ta, tb, tsa, tsb, p, num_sms, stream) : launch_mx2<128, 0>(ta, tb, tsa, tsb, p, num_sms, stream);
}
