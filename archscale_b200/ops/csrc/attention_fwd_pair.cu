// Attention forward, two query tiles per CTA (the form for grids that fill the GPU; attention_fwd.cu is the other one).
//
// A work item is one KV head and two 128-row query tiles that read the same K / V tiles: the same rows of two neighbouring
// query heads where the KV group has an even number of them (equal masks, equal tile counts), else two neighbouring row
// blocks of one head.  384 threads:
//   warps 0..3   softmax of tile A (thread = query row)      warps 4..7   softmax of tile B
//   warp 8       loads: Q tiles, K / V tiles through one ring of slots; fetches the next work item
//   warp 9       every MMA
// What decides the speed is the order of the MMAs.  One tile pair costs the tensor pipe 4 × 518 cycles and the MUFU
// 2 × 1024; both are only busy if the exponentials of one tile run under the products of the other.  The MMA warp
// alternates per tile:  P·V of A, next S of A | P·V of B, next S of B | …  so that S of B is ready half a period after S of
// A and the two softmax groups stay half a period apart by themselves.  (Both S first and then both P·V, or two issuing
// threads, let the groups fall into step: they then queue for the MUFU together and the tensor pipe idles.)  MMAs of one
// thread execute in order, so S may overwrite the columns that held P without a barrier, and "S of tile t is complete"
// implies "P·V of tile t−1 is complete": the rare rescale of O needs no barrier of its own.
// P·V starts when three quarters of P are written (PV_SPLIT).
// The MMA warp runs converged, in warp-uniform control flow, and elects a lane per instruction: issued from inside a branch
// of one lane an MMA took ≈100 cycles instead of the pipe's 65 (4030 against 3270 cycles a pair).
//
// The kernel is persistent: a running CTA takes over the work of CTAs that have not started yet
// (clusterlaunchcontrol.try_cancel), one item ahead, so the loads and first products of an item run under the last softmax
// and the store of the one before; the fixed cost of a CTA (tensor memory, barriers, first loads) is paid once per SM.
// Items are ordered by KV heads that share the L2 (kv_chunk), inside them longest first.
//
// Masking rule, softmax and lazy rescale as in attention_fwd.cu.
// TMEM columns: S/P of A 0..127 | S/P of B 128..255 | O of A 256..383 | O of B 384..511.  P is packed into the first 64
// columns of its S.
#include "sm100.cuh"
#include "api.h"

namespace b200 {

constexpr int AP_BM = 128, AP_BN = 128;
constexpr int AP_THREADS = 384;
constexpr int PV_SPLIT = 6;               // of the eight 16-key steps of P·V, how many start before the rest of P is written
constexpr float kLog2e_ap = 1.4426950408889634f, kLn2_ap = 0.6931471805599453f;

struct AttnPairParams {
  __nv_bfloat16* out;      // [B, T, H, D]
  float* lse;              // [B, H, T]
  const int* row_start;    // [B*T] first visible key of each row (batch-local) or null
  int B, T, H, G;
  int window_left;         // < 0: unlimited
  int same_rows;           // 1: the two tiles are the same rows of heads 2i, 2i+1; 0: row blocks 2i, 2i+1 of one head
  int n_blk;               // row blocks per head (same_rows) or pairs of them
  int per_kv;              // items per (batch, KV head) and row block
  int kv_chunk;            // (batch, KV head) combinations whose items are interleaved
  float scale_log2;        // softmax scale · log2(e)
  int* status;
};

template <int D>
struct AttnPairSmem {
  static constexpr int TILE = 128 * D * 2;
  static constexpr int SLOTS = D == 128 ? 5 : 8;                       // K / V tiles in flight
  static constexpr int TOTAL = 2 * TILE + SLOTS * TILE + 1024 + 512;
};

struct PairItem {
  int b, g, h[2], q0[2], j_begin, n;
};

__device__ __forceinline__ int pair_lo_of(const AttnPairParams& p, int b, int r) {
  int lo = p.row_start ? p.row_start[static_cast<size_t>(b) * p.T + r] : 0;
  if (p.window_left >= 0) lo = max(lo, r - p.window_left);
  return lo;
}

__device__ __forceinline__ PairItem pair_item(const AttnPairParams& p, int idx) {
  // idx = ((chunk, row block from the last one down), KV head in chunk, item of the KV head)
  const int n_kv = p.B * p.G;
  const int chunk_items = p.kv_chunk * p.n_blk * p.per_kv;
  const int c = idx / chunk_items;
  const int in_chunk = min(p.kv_chunk, n_kv - c * p.kv_chunk);          // the last chunk may be smaller
  int rem = idx - c * chunk_items;
  const int blk = p.n_blk - 1 - rem / (in_chunk * p.per_kv);
  rem %= in_chunk * p.per_kv;
  const int kv = c * p.kv_chunk + rem / p.per_kv, i = rem % p.per_kv;
  PairItem it;
  it.b = kv / p.G;
  it.g = kv % p.G;
  const int h0 = it.g * (p.H / p.G);
  if (p.same_rows) {
    it.h[0] = h0 + 2 * i; it.h[1] = h0 + 2 * i + 1;
    it.q0[0] = it.q0[1] = blk * AP_BM;
  } else {
    it.h[0] = it.h[1] = h0 + i;
    it.q0[0] = 2 * blk * AP_BM; it.q0[1] = it.q0[0] + AP_BM;
  }
  const int j_end = (min(it.q0[1] + AP_BM, p.T) - 1) / AP_BN + 1;
  it.j_begin = min(pair_lo_of(p, it.b, it.q0[0]) / AP_BN, j_end - 1);
  it.n = j_end - it.j_begin;
  return it;
}

// Ask for the work of a CTA that has not started: the answer (16 bytes) arrives in shared memory with the barrier's bytes.
__device__ __forceinline__ void steal_request(void* resp, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(resp)), "r"(smem_u32(bar)) : "memory");
}
// The linear CTA index the answer names, or -1 when there was none left.
__device__ __forceinline__ int steal_result(const void* resp) {
  uint32_t ok, x;
  asm volatile(
      "{\n"
      ".reg .b128 r;\n"
      ".reg .pred p;\n"
      "ld.shared.b128 r, [%2];\n"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "mov.u32 %1, 0;\n"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n"
      "}\n"
      : "=r"(ok), "=r"(x) : "r"(smem_u32(resp)) : "memory");
  return ok ? static_cast<int>(x) : -1;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int D>
__global__ void __launch_bounds__(AP_THREADS, 1)
attn_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, const AttnPairParams p) {
  using SM = AttnPairSmem<D>;
  constexpr int DC = D / 64;                       // 64-element chunks of the head dim (TMA boxes)
  constexpr int CHUNK_BYTES = 128 * 64 * 2;        // one box: 128 rows × 64 elements
  constexpr int NS = SM::SLOTS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sq = smem;                              // Q of A, Q of B
  uint8_t* skv = smem + 2 * SM::TILE;              // slot s at skv + s·TILE; K_0, V_0, K_1, V_1, … in turn
  uint64_t* bars = reinterpret_cast<uint64_t*>(skv + NS * SM::TILE);
  uint64_t* q_full = bars;              // [2]
  uint64_t* q_empty = bars + 2;         // [2]  the item's last S of this tile has completed
  uint64_t* kv_full = bars + 4;         // [NS]
  uint64_t* kv_empty = bars + 12;       // [NS]
  uint64_t* s_full = bars + 20;         // [2]
  uint64_t* p_part = bars + 22;         // [2]  (count 4) the first PV_SPLIT·16 keys of P are in tensor memory
  uint64_t* p_full = bars + 24;         // [2]  (count 4) all of P
  uint64_t* o_done = bars + 26;         // [2]  the item's last P·V of this tile has completed
  uint64_t* nx_full = bars + 28;        // [2]  next work item known
  uint64_t* nx_empty = bars + 30;       // [2]  (count 10) read by the MMA warp, the loader and eight softmax warps
  uint4* nx_resp = reinterpret_cast<uint4*>(bars + 32);                 // [2]
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(nx_resp + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); mbar_init(&s_full[s], 1); mbar_init(&p_part[s], 4);
      mbar_init(&p_full[s], 4); mbar_init(&o_done[s], 1); mbar_init(&nx_full[s], 1); mbar_init(&nx_empty[s], 10);
    }
    for (int s = 0; s < NS; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], 1); }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
  }
  if (warp == 9) { tmem_alloc(tmem_ptr, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr, 0);

  // The item after number `i` of this CTA (the answer to request i), or -1.  One thread per role calls it.
  auto next_item = [&](int i, int& idx) -> bool {
    const int st = i & 1;
    if (!mbar_wait(&nx_full[st], (i >> 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL)) return false;
    idx = steal_result(&nx_resp[st]);
    fence_proxy_async_smem();                          // the read comes before the next answer's (async-proxy) write
    mbar_arrive(&nx_empty[st]);
    return true;
  };
  // the same by a whole warp
  auto next_item_warp = [&](int i, int& idx) -> bool {
    int got = 1, nx = -1;
    if (lane == 0) got = next_item(i, nx) ? 1 : 0;
    got = __shfl_sync(0xffffffffu, got, 0);
    idx = __shfl_sync(0xffffffffu, nx, 0);
    return got != 0;
  };

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 8 && lane == 0) {
      // ---------------------------------------------------------------- loads
      int idx = blockIdx.x;
      uint32_t slot = 0, sph = 0;                      // ring position and its phase
      for (int i = 0; idx >= 0; ++i) {
        const int st = i & 1;
        if (!mbar_wait_relaxed(&nx_empty[st], ((i >> 1) & 1) ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY)) goto done;
        mbar_arrive_expect_tx(&nx_full[st], 16);
        steal_request(&nx_resp[st], &nx_full[st]);
        const PairItem it = pair_item(p, idx);
        auto load_q = [&](int s) -> bool {
          if (!mbar_wait_relaxed(&q_empty[s], (i & 1) ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY)) return false;
          mbar_arrive_expect_tx(&q_full[s], SM::TILE);
#pragma unroll
          for (int c = 0; c < DC; ++c)
            tma_load_2d(sq + s * SM::TILE + c * CHUNK_BYTES, &tmap_q, &q_full[s], it.h[s] * D + c * 64, it.b * p.T + it.q0[s]);
          return true;
        };
        auto load_kv = [&](const CUtensorMap* m, int j) -> bool {
          if (!mbar_wait_relaxed(&kv_empty[slot], sph ^ 1, abort_flag, p.status, STATUS_TIMEOUT_EMPTY)) return false;
          mbar_arrive_expect_tx(&kv_full[slot], SM::TILE);
#pragma unroll
          for (int c = 0; c < DC; ++c)
            tma_load_2d(skv + slot * SM::TILE + c * CHUNK_BYTES, m, &kv_full[slot], it.g * D + c * 64,
                        it.b * p.T + (it.j_begin + j) * AP_BN);
          if (++slot == NS) { slot = 0; sph ^= 1; }
          return true;
        };
        if (!load_kv(&tmap_k, 0)) goto done;
        if (!load_q(0) || !load_q(1)) goto done;
        if (!load_kv(&tmap_v, 0)) goto done;
        for (int j = 1; j < it.n; ++j) {
          if (!load_kv(&tmap_k, j)) goto done;
          if (!load_kv(&tmap_v, j)) goto done;
        }
        if (!next_item(i, idx)) goto done;
      }
    } else if (warp == 9) {
      // ---------------------------------------------------------------- MMA (the whole warp, converged)
      constexpr uint32_t idesc_s = make_idesc_bf16(AP_BM, AP_BN, 0, 0);       // S = Q·Kᵀ  (both K-major)
      constexpr uint32_t idesc_o = make_idesc_bf16(AP_BM, D, 0, 1);           // O += P·V  (V is N-major)
      const uint32_t sqa = smem_u32(sq), skva = smem_u32(skv);
      int idx = blockIdx.x;
      int n = __shfl_sync(0xffffffffu, pair_item(p, idx).n, 0);       // (shuffles make warp-uniform what they return)
      uint32_t slot = 0, sph = 0;                      // ring position of the next tile to be waited for
      uint32_t step = 0;                               // tiles done by this CTA: phase of p_part / p_full
      auto advance = [&]() { if (++slot == NS) { slot = 0; sph ^= 1; } };
      auto issue_s = [&](int s, uint32_t kslot) {
        const uint32_t qa = sqa + s * SM::TILE, ka = skva + kslot * SM::TILE;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k / 4) * CHUNK_BYTES + (k % 4) * 32;
          umma_bf16_warp(tmem_base + s * 128, make_smem_desc(qa + off, 16, 1024), make_smem_desc(ka + off, 16, 1024), idesc_s, k != 0);
        }
        umma_commit_warp(&s_full[s]);
      };
      auto issue_pv = [&](int s, uint32_t vslot, bool first, int k0, int k1) {
        const uint32_t va = skva + vslot * SM::TILE;
#pragma unroll
        for (int k = k0; k < k1; ++k)                  // 16 keys: 8 packed columns of P, 2048 bytes of V
          umma_bf16_ts_warp(tmem_base + 256 + s * 128, tmem_base + s * 128 + k * 8, make_smem_desc(va + k * 2048, CHUNK_BYTES, 1024),
                            idesc_o, !(first && k == 0));
      };
      // first S of both tiles of the first item
      if (!mbar_wait_warp(&kv_full[0], 0, abort_flag, p.status, STATUS_TIMEOUT_FULL)) goto done;
      for (int s = 0; s < 2; ++s) {
        if (!mbar_wait_warp(&q_full[s], 0, abort_flag, p.status, STATUS_TIMEOUT_FULL)) goto done;
        tc_fence_after();
        issue_s(s, 0);
        if (n == 1) umma_commit_warp(&q_empty[s]);
      }
      umma_commit_warp(&kv_empty[0]);
      advance();
      for (int i = 0; idx >= 0; ++i) {
        int idx_next = -1, n_next = 0;
        for (int j = 0; j < n; ++j, ++step) {
          const bool last = j == n - 1;
          if (last) {
            if (!next_item_warp(i, idx_next)) goto done;
            if (idx_next >= 0) n_next = __shfl_sync(0xffffffffu, pair_item(p, idx_next).n, 0);
          }
          const bool more = !last || idx_next >= 0;    // there is another S to issue after this P·V
          const uint32_t vslot = slot, vph = sph;
          advance();
          const uint32_t kslot = slot, kph = sph;
          if (more) advance();
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            if (s == 0 && !mbar_wait_warp(&kv_full[vslot], vph, abort_flag, p.status, STATUS_TIMEOUT_FULL)) goto done;
            if (!mbar_wait_warp(&p_part[s], step & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) goto done;
            tc_fence_after();
            issue_pv(s, vslot, j == 0, 0, PV_SPLIT);
            if (!mbar_wait_warp(&p_full[s], step & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) goto done;
            tc_fence_after();
            issue_pv(s, vslot, false, PV_SPLIT, AP_BN / 16);
            if (last) umma_commit_warp(&o_done[s]);
            if (s == 1) umma_commit_warp(&kv_empty[vslot]);
            if (more) {
              if (s == 0 && !mbar_wait_warp(&kv_full[kslot], kph, abort_flag, p.status, STATUS_TIMEOUT_FULL)) goto done;
              if (last && !mbar_wait_warp(&q_full[s], (i + 1) & 1, abort_flag, p.status, STATUS_TIMEOUT_FULL)) goto done;
              tc_fence_after();
              issue_s(s, kslot);
              if (s == 1) umma_commit_warp(&kv_empty[kslot]);
              if (last ? n_next == 1 : j + 1 == n - 1) umma_commit_warp(&q_empty[s]);
            }
          }
        }
        idx = idx_next; n = n_next;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // ------------------------------------------------------------------ softmax of tile `s`
    const int s = warp >> 2, qtr = warp & 3;
    const uint32_t lane_off = static_cast<uint32_t>(qtr * 32) << 16;
    const uint32_t t_s = tmem_base + s * 128 + lane_off, t_o = tmem_base + 256 + s * 128 + lane_off;
    const float sl2 = p.scale_log2;
    const float2 sl2x2 = make_float2(sl2, sl2);
    uint32_t step = 0;
    int idx = blockIdx.x;
    for (int i = 0; idx >= 0; ++i) {
      const PairItem it = pair_item(p, idx);
      const int q0 = s ? it.q0[1] : it.q0[0], h = s ? it.h[1] : it.h[0];
      const int r = q0 + qtr * 32 + lane;
      const bool row_valid = r < p.T;
      const int lo_r = row_valid ? pair_lo_of(p, it.b, r) : 0;
      const int lo_last = pair_lo_of(p, it.b, min(q0 + AP_BM, p.T) - 1);   // q0 ≥ T (no rows): the last row, never used
      float m_used = -1e30f;
      float2 l2 = make_float2(0.f, 0.f);
      for (int j = 0; j < it.n; ++j, ++step) {
        const int k0 = (it.j_begin + j) * AP_BN;
        if (!mbar_wait(&s_full[s], step & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) goto done;
        tc_fence_after();
        float x[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&x[c * 32]));
        tmem_ld_wait();
        const bool full_tile = (k0 + AP_BN - 1 <= q0) && (k0 >= lo_last);
        if (!full_tile) {
#pragma unroll
          for (int e = 0; e < 128; ++e)
            if (k0 + e > r || k0 + e < lo_r) x[e] = -INFINITY;
        }
        float m4[4];                                   // four independent chains
#pragma unroll
        for (int e = 0; e < 4; ++e) m4[e] = fmaxf(x[2 * e], x[2 * e + 1]);
#pragma unroll
        for (int e = 8; e < 128; e += 2) m4[(e >> 1) & 3] = max3(m4[(e >> 1) & 3], x[e], x[e + 1]);
        const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl2;
        // lazy rescale: only when the running max grew by more than 8 (factor 256); decided per warp.  P·V of the tile
        // before has completed (its completion was committed before S of this tile)
        if (__any_sync(0xffffffffu, mx - m_used > 8.f)) {
          const float m_new = fmaxf(m_used, mx);
          const float alpha = exp2f(m_used - m_new);
          if (j > 0) {
#pragma unroll
            for (int c = 0; c < D / 16; ++c) {
              uint32_t o[16];
              tmem_ld_32x16(t_o + c * 16, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st_32x16(t_o + c * 16, o);
            }
          }
          l2.x *= alpha; l2.y *= alpha;
          m_used = m_new;
        }
        // P = 2^(x·scale − m_used), packed to bf16 over the columns of S; row sum in fp32
        const float2 nm = make_float2(-m_used, -m_used);
        float2 sa = make_float2(0.f, 0.f), sb = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t w[16];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float2 ya = fma_f32x2(make_float2(x[c * 32 + 2 * e], x[c * 32 + 2 * e + 1]), sl2x2, nm);
            const float2 yb = fma_f32x2(make_float2(x[c * 32 + 2 * e + 2], x[c * 32 + 2 * e + 3]), sl2x2, nm);
            const float2 pa = make_float2(exp2f(ya.x), exp2f(ya.y)), pb = make_float2(exp2f(yb.x), exp2f(yb.y));
            sa = add_f32x2(sa, pa); sb = add_f32x2(sb, pb);
            w[e] = pack_bf16x2(pa.x, pa.y); w[e + 1] = pack_bf16x2(pb.x, pb.y);
          }
          tmem_st_32x16(t_s + c * 16, w);
          if (c == PV_SPLIT / 2 - 1) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_part[s]);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[s]);
        l2 = add_f32x2(l2, add_f32x2(sa, sb));
      }
      // ---- O / l and the log-sum-exp
      const float l_sum = l2.x + l2.y;
      const float inv_l = l_sum > 0.f ? 1.f / l_sum : 0.f;
      if (!mbar_wait(&o_done[s], i & 1, abort_flag, p.status, STATUS_TIMEOUT_TMEM_FULL)) goto done;
      tc_fence_after();
      __nv_bfloat16* orow = p.out + ((static_cast<size_t>(it.b) * p.T + r) * p.H + h) * D;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(t_o + c * 32, o);
        tmem_ld_wait();
        if (row_valid) {
#pragma unroll
          for (int e = 0; e < 32; e += 16) {
            uint32_t w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              w[u] = pack_bf16x2(__uint_as_float(o[e + 2 * u]) * inv_l, __uint_as_float(o[e + 2 * u + 1]) * inv_l);
            store_32b(orow + c * 32 + e, w);
          }
        }
      }
      tc_fence_before();                               // O has been read before this warp's next P is announced
      if (row_valid)
        p.lse[(static_cast<size_t>(it.b) * p.H + h) * p.T + r] = l_sum > 0.f ? (m_used + log2f(l_sum)) * kLn2_ap : -INFINITY;
      if (!next_item_warp(i, idx)) goto done;
    }
  }

done:
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

int make_tmap_2d_bf16(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_elems,
                      uint32_t box_inner, uint32_t box_outer);

template <int D>
static int launch_attn_fwd_pair(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnPairParams& p,
                                cudaStream_t st) {
  auto kern = attn_fwd_pair_kernel<D>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnPairSmem<D>::TOTAL) != cudaSuccess) return -2;
    configured = true;
  }
  const unsigned items = static_cast<unsigned>(p.B) * p.G * p.n_blk * p.per_kv;
  kern<<<items, AP_THREADS, AttnPairSmem<D>::TOTAL, st>>>(tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace b200

// Contract of b200_attn_fwd, which checks the arguments and calls this where the grid is large enough.
extern "C" int b200_attn_fwd_pair(const void* q, const void* k, const void* v, void* out, float* lse, const int* row_start,
                                  int B, int T, int H, int G, int D, int window_left, float scale, int* status,
                                  cudaStream_t stream) {
  using namespace b200;
  CUtensorMap tq, tk, tv;
  const uint64_t hd = static_cast<uint64_t>(H) * D, gd = static_cast<uint64_t>(G) * D, bt = static_cast<uint64_t>(B) * T;
  int rc = make_tmap_2d_bf16(&tq, q, hd, bt, hd, 64, 128);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tk, k, gd, bt, gd, 64, 128);
  if (rc) return rc;
  rc = make_tmap_2d_bf16(&tv, v, gd, bt, gd, 64, 128);
  if (rc) return rc;
  const int group = H / G, n_qt = (T + AP_BM - 1) / AP_BM;
  const int same = group % 2 == 0;
  const long long kv_bytes = static_cast<long long>(T) * D * 4;
  const int kv_chunk = static_cast<int>(kv_bytes >= (24ll << 20) ? 1 : (24ll << 20) / kv_bytes);
  AttnPairParams p{static_cast<__nv_bfloat16*>(out), lse, row_start, B, T, H, G, window_left, same, same ? n_qt : (n_qt + 1) / 2,
                   same ? group / 2 : group, kv_chunk, scale * kLog2e_ap, status};
  return D == 128 ? launch_attn_fwd_pair<128>(tq, tk, tv, p, stream) : launch_attn_fwd_pair<64>(tq, tk, tv, p, stream);
}
