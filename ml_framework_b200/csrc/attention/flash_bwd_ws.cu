// Self-attention backward, head_dim 128: 128 x 128 tiles, three warpgroups, P^T kept in tensor memory.
//
// One CTA owns 128 key/value rows of one (batch, kv-head) and walks the 128-row query tiles that can
// see them (all heads of the GQA group). Key-major ("transposed") orientation, so that each thread of the
// compute warpgroup owns one key row and dK / dV accumulate in place across the whole walk:
//   S^T  = K  Q^T        dP^T = V dO^T                 (M128 N128 K128, operands in shared memory)
//   P^T  = exp2(S^T c - lse)        -> packed bf16 into TENSOR MEMORY over S^T (A operand of dV)
//   dS^T = P^T o (dP^T - delta) c   -> packed bf16 into shared memory        (operand of dK and dQ)
//   dV  += P^T  dO       dK  += dS^T Q                 (M128 N128 K128)
//   dQ   = dS   K        (M = query rows)  -> read out by its own warpgroup into swizzled staging tiles
//                                            and added to the fp32 dQ buffer by TMA reduction stores
//                                            (per-thread reductions saturate the L2 atomic path and
//                                            the load/store unit the other warpgroup needs)
// The same 128B-swizzled tiles serve as K-major or MN-major operands through their descriptors, so
// nothing is ever transposed in memory.
//
// 512 threads: warps 0..3 control (warp 0 TMA producer, warp 1 MMA issuer), warps 4..11 compute
// (one key row and half of the tile's queries per thread), warps 12..15 dQ read-out; the control
// warpgroup hands registers to the others (setmaxnreg 56 / 144 / 144 / 168 of 4 x 128).
// TMEM (512 columns): dK | dV | S^T (then P^T) | dP^T (then dQ).
// Bound by the chain dS -> dK, dQ -> dQ read-out -> dP^T -> dS of a tile: without any of the compute
// warpgroups' arithmetic 4 x 2048, 16 heads takes 268 us. A second compute warpgroup and paired fp32
// arithmetic shorten their link: 315 -> 300 us; 2 x 4096, 32 / 8 heads 891 -> 862 us.
// Around the chain: a CTA's first S^T waits for K and Q only, dK and dV leave through the copy engine, only the blocks that
// the mask cuts for a warp are masked, and the launch overlaps the end of the one before. With the statistics' pass
// (attn_delta_kernel), all launches of a backward: 4 x 2048, 16 heads 302 -> 274 us; 2 x 4096, 32 / 8 heads 855 -> 840 us;
// 3 x 777, 8 heads 56 -> 42 us; 8 x 512, 16 heads 107 -> 86 us (dQ ahead of dK: 275, 868, 43, 85 us).
// Issue order on the tensor pipe: dV(i), S^T(i+1), dK(i), dQ(i), dP^T(i+1): the next tile's
// exponentials run while this tile's gradients are multiplied. The issuing thread polls its barriers:
// it is on the chain, and a suspended wait wakes late (2 x 4096, 32 / 8 heads: 854 -> 811 us; 4 x 2048,
// 16 heads: 306 -> 303 us; in the forward kernel, whose chain is in the softmax, polling costs 3 %).
//
// The reference has no attention backward (its attention layers are forward-only,
// src/MLFramework/Inference/PagedAttention/Layers/PagedAttentionLayer.cs:102-144); training the
// GPT and Llama configurations requires it.
#include <float.h>

#include "../common/host.h"
#include "../common/ptx.cuh"
#include "../mlf_api.h"

namespace mlf {

int cached_tmap_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t bi, uint32_t bo, bool swizzle = true);

constexpr int G_T = 128;                       // tile edge (keys and queries)
constexpr int G_D = 128;
constexpr int G_THREADS = 512;
constexpr int G_TILE = G_T * G_D * 2;          // 32 KB: two 64-column blocks of 16 KB
constexpr int G_HALF = G_TILE / 2;
constexpr int G_STATS = 2 * G_T * 4;           // lse (log2 domain) | delta, fp32, per stage
constexpr int G_DQ_STG = 32 * 32 * 4;          // dQ staging tile of one warp: 32 rows x 32 fp32 columns, 128B-swizzled
constexpr int G_SMEM = 7 * G_TILE + 2 * G_STATS + 256;   // K, V, Q x 2, dO, dS, 8 staging tiles (= 1 tile)
constexpr int G_TMEM_COLS = 512;

struct FlashBwdWsParams {
  float* dq_accum;          // fp32 [tokens, Hq*128], zeroed by the launcher
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  const float* lse2;        // [B, Hq, stat_pitch] logsumexp * log2(e)
  const float* delta;       // [B, Hq, stat_pitch] rowsum(dO o O)
  int stat_pitch;           // whole tiles; entries from S on are 0, so that a masked score gives P = 0 and dS = 0
  long long lddk, lddv;
  int B, S, Hq, Hkv, causal;
  float scale, scale_log2;
  int* err;
};

__device__ __forceinline__ void bulk_g2s(uint32_t smem_dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}

__global__ void __launch_bounds__(G_THREADS, 1)
flash_bwd_ws_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                    const __grid_constant__ CUtensorMap tmDV, const FlashBwdWsParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sK = sbase;
  const uint32_t sV = sK + G_TILE;
  auto sQ = [&](int s) { return sV + G_TILE + (uint32_t)s * G_TILE; };
  const uint32_t sdO = sV + 3u * G_TILE;                  // single buffer: reloaded once dV of the previous tile has read it
  const uint32_t sdS = sV + 4u * G_TILE;
  const uint32_t sStg = sV + 5u * G_TILE;                  // two dQ staging tiles of 4 KB for each of four warps
  const uint32_t sStats = sStg + G_TILE;                    // stage s at + s * G_STATS
  const uint32_t bars = sStats + 2 * G_STATS;
  // barriers: k_full, q_full[2], q_empty[2], s_full, dp_full, p_full, ds_full, dq_full, dq_empty, do_full, do_empty, v_full
  const uint32_t k_full = bars, v_full = bars + 8u * 13;
  auto q_full = [&](int s) { return bars + 8u * (1 + s); };
  auto q_empty = [&](int s) { return bars + 8u * (3 + s); };
  const uint32_t s_full = bars + 8u * 5, dp_full = bars + 8u * 6, p_full = bars + 8u * 7, ds_full = bars + 8u * 8,
                 dq_full = bars + 8u * 9, dq_empty = bars + 8u * 10, do_full = bars + 8u * 11, do_empty = bars + 8u * 12;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + (bars - sbase) + 8 * 14);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_kt = (p.S + G_T - 1) / G_T;
  // 1-D grid ordered by work: under a causal mask the first key tiles see the most query tiles
  const int per_kt = p.Hkv * p.B;
  const int kt = (int)blockIdx.x / per_kt;
  const int hkv = ((int)blockIdx.x % per_kt) % p.Hkv;
  const int b = ((int)blockIdx.x % per_kt) / p.Hkv;
  const int group = p.Hq / p.Hkv;
  const int k0 = kt * G_T;
  const long long row_base = (long long)b * p.S;
  const int qt0 = p.causal ? kt : 0;
  const int per_head = n_kt - qt0;           // query tiles per head (n_qt == n_kt: same tile edge)
  const int n_it = per_head * group;

  if ((sbase & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.err, 0, ERR_BAD_INDEX);
    return;
  }
  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(q_full(s), 1);
      mbar_init(q_empty(s), 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 256);
    mbar_init(ds_full, 256);
    mbar_init(dq_full, 1);
    mbar_init(dq_empty, 128);
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_ptr_smem), G_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_trigger();
  pdl_wait();
  const uint32_t t_dK = tmem_base, t_dV = tmem_base + 128, t_S = tmem_base + 256, t_dP = tmem_base + 384;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0) {
      // ===================== TMA producer =====================
      if (elect_one()) {
        const int krow = (int)(row_base + k0);
        mbar_expect_tx(k_full, G_TILE);
        tma_load_2d(sK, &tmK, hkv * G_D, krow, k_full);
        tma_load_2d(sK + G_HALF, &tmK, hkv * G_D + 64, krow, k_full);
        for (int it = 0; it < n_it; ++it) {
          const int s = it & 1;
          if (!mbar_wait(q_empty(s), ((it >> 1) & 1) ^ 1u, abort_flag, p.err, ERR_WAIT_ATTN)) break;
          const int h = hkv * group + it / per_head;
          const int q0 = (qt0 + it % per_head) * G_T;
          const int qrow = (int)(row_base + q0);
          const long long sidx = ((long long)b * p.Hq + h) * p.stat_pitch + q0;
          mbar_expect_tx(q_full(s), G_TILE + G_STATS);
          tma_load_2d(sQ(s), &tmQ, h * G_D, qrow, q_full(s));
          tma_load_2d(sQ(s) + G_HALF, &tmQ, h * G_D + 64, qrow, q_full(s));
          bulk_g2s(sStats + s * G_STATS, p.lse2 + sidx, G_T * 4, q_full(s));
          bulk_g2s(sStats + s * G_STATS + G_T * 4, p.delta + sidx, G_T * 4, q_full(s));
          if (it == 0) {                         // V behind the operands of the first S^T
            mbar_expect_tx(v_full, G_TILE);
            tma_load_2d(sV, &tmV, hkv * G_D, krow, v_full);
            tma_load_2d(sV + G_HALF, &tmV, hkv * G_D + 64, krow, v_full);
          }
          if (!mbar_wait(do_empty, (it & 1) ^ 1u, abort_flag, p.err, ERR_WAIT_ATTN)) break;
          mbar_expect_tx(do_full, G_TILE);
          tma_load_2d(sdO, &tmdO, h * G_D, qrow, do_full);
          tma_load_2d(sdO + G_HALF, &tmdO, h * G_D + 64, qrow, do_full);
        }
      }
    } else if (warp == 1) {
      // ===================== MMA issuer =====================
      if (elect_one()) {
        const uint32_t idesc_kk = make_idesc_bf16(128, 128, 0, 0);   // S^T, dP^T: both operands K-major
        const uint32_t idesc_kn = make_idesc_bf16(128, 128, 0, 1);   // dV, dK: B (dO / Q) MN-major
        const uint32_t idesc_nn = make_idesc_bf16(128, 128, 1, 1);   // dQ: A (dS) and B (K) MN-major
        auto issue_kk = [&](uint32_t d_tmem, uint32_t a, uint32_t bm) {
#pragma unroll
          for (int k = 0; k < G_D / 16; ++k) {
            const uint32_t off = (k >> 2) * G_HALF + (k & 3) * 32;
            umma_bf16_ss(d_tmem, make_smem_desc_sw128(a + off, 16, 1024), make_smem_desc_sw128(bm + off, 16, 1024), idesc_kk, k != 0);
          }
        };
        bool ok = mbar_wait_poll(k_full, 0, abort_flag, p.err, ERR_WAIT_ATTN);
        if (ok && n_it > 0) ok = mbar_wait_poll(q_full(0), 0, abort_flag, p.err, ERR_WAIT_ATTN);
        if (ok && n_it > 0) {
          tc_fence_after_sync();
          issue_kk(t_S, sK, sQ(0));
          umma_commit(s_full);
          ok = mbar_wait_poll(v_full, 0, abort_flag, p.err, ERR_WAIT_ATTN) && mbar_wait_poll(do_full, 0, abort_flag, p.err, ERR_WAIT_ATTN);
          if (ok) {
            tc_fence_after_sync();
            issue_kk(t_dP, sV, sdO);
            umma_commit(dp_full);
          }
        }
        for (int it = 0; it < n_it && ok; ++it) {
          const int s = it & 1;
          if (!mbar_wait_poll(p_full, it & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
          tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < G_T / 16; ++k)     // dV += P^T dO   (A from tensor memory)
            umma_bf16_ts(t_dV, t_S + 8u * (k & 3) + 64u * (k >> 2), make_smem_desc_sw128(sdO + k * 2048, G_HALF, 1024), idesc_kn, (it | k) != 0);
          umma_commit(do_empty);                   // dO of this tile has been read (dP^T earlier, dV now)
          const bool more = it + 1 < n_it;
          if (more) {                              // S^T of the next tile goes in behind dV
            if (!mbar_wait_poll(q_full(s ^ 1), ((it + 1) >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
            tc_fence_after_sync();
            issue_kk(t_S, sK, sQ(s ^ 1));
            umma_commit(s_full);
          }
          if (!mbar_wait_poll(ds_full, it & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
          tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < G_T / 16; ++k)     // dK += dS^T Q
            umma_bf16_ss(t_dK, make_smem_desc_sw128(sdS + (k >> 2) * G_HALF + (k & 3) * 32, 16, 1024),
                         make_smem_desc_sw128(sQ(s) + k * 2048, G_HALF, 1024), idesc_kn, (it | k) != 0);
          if (it > 0) {                            // dQ lands where the previous dQ was: wait for its read-out
            if (!mbar_wait_poll(dq_empty, (it - 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
            tc_fence_after_sync();
          }
#pragma unroll
          for (int k = 0; k < G_T / 16; ++k)     // dQ = dS K
            umma_bf16_ss(t_dP, make_smem_desc_sw128(sdS + k * 2048, G_HALF, 1024),
                         make_smem_desc_sw128(sK + k * 2048, G_HALF, 1024), idesc_nn, k != 0);
          umma_commit(dq_full);
          umma_commit(q_empty(s));
          if (more) {                              // dP^T of the next tile needs the dQ columns back
            if (!mbar_wait_poll(dq_empty, it & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
            if (!mbar_wait_poll(do_full, (it + 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
            tc_fence_after_sync();
            issue_kk(t_dP, sV, sdO);
            umma_commit(dp_full);
          }
        }
      }
    }
  } else if (warp < 12) {
    // ===================== compute warpgroups: one key row and 64 of the tile's queries per thread =====================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    const int qd = warp & 3;
    const int g = (warp - 4) >> 2;             // which 64 query columns
    const int r = qd * 32 + lane;
    const int kv_i = k0 + r, kv_w = k0 + qd * 32;     // this thread's key, its warp's first
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    const uint32_t t_Sg = t_S + 64u * g, t_dPg = t_dP + 64u * g;      // P^T of these columns replaces their own S^T
    const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2), scale2 = pack_f32x2(p.scale, p.scale);
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int s = it & 1;
      const int q0 = (qt0 + it % per_head) * G_T;
      const bool need_mask = (p.causal && q0 < k0 + G_T - 1) || (q0 + G_T > p.S) || (k0 + G_T > p.S);
      // the statistics arrive with Q / dO on q_full
      if (!mbar_wait_warp(q_full(s), (it >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
      if (!mbar_wait_warp(s_full, it & 1, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
      tc_fence_after_sync();
      uint32_t pk[32];
      const uint32_t st_addr = sStats + s * G_STATS + g * 256;     // shared-window address of these columns' statistics
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        // 32 columns at a time: S^T from tensor memory and the row statistics from shared memory are all requested up
        // front so that their latencies overlap
        uint32_t sv[32];
        tmem_ld_32x32b_x32(t_Sg + 32 * hh + lane_off, sv);
        uint64_t ls[16];                       // -logsumexp of two queries each
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4)
          asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(ls[2 * c4]), "=l"(ls[2 * c4 + 1]) : "r"(st_addr + (32 * hh + 4 * c4) * 4));
        tmem_wait_ld();
        const int qb = q0 + 64 * g + 32 * hh;
        if (need_mask && (qb + 32 > p.S || kv_w + 32 > p.S || (p.causal && qb < kv_w + 31))) {
          // blocks of a diagonal or ragged tile that the mask cuts for this warp: masked scores become -inf, exp2 gives 0
          const int lo = kv_i >= p.S ? 32 : p.causal ? kv_i - qb : 0, hi = p.S - qb;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < lo || i >= hi) sv[i] = __float_as_uint(-INFINITY);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float e0, e1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), c2, neg_f32x2(ls[i])), e0, e1);
          pk[16 * hh + i] = pack_bf16x2(exp2f(e0), exp2f(e1));
        }
      }
      tmem_st_32x32b_x32(t_Sg + lane_off, pk);
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(p_full);
      // dS^T from the rounded P^T (the same values dV is multiplied with)
      if (!mbar_wait_warp(dp_full, it & 1, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t drow = sdS + g * G_HALF + r * 128;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t dp[32];
        tmem_ld_32x32b_x32(t_dPg + 32 * hh + lane_off, dp);
        uint64_t dl[16];
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4)
          asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(dl[2 * c4]), "=l"(dl[2 * c4 + 1])
                       : "r"(st_addr + (G_T + 32 * hh + 4 * c4) * 4));
        tmem_wait_ld();
        uint32_t dsk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint32_t pa = pk[16 * hh + i];
          const uint64_t pp = pack_f32x2(__uint_as_float(pa << 16), __uint_as_float(pa & 0xffff0000u));
          const uint64_t d = add_f32x2(pack_f32x2(__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1])), neg_f32x2(dl[i]));
          float d0, d1;
          unpack_f32x2(mul_f32x2(mul_f32x2(pp, d), scale2), d0, d1);
          dsk[i] = pack_bf16x2(d0, d1);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t off = ((uint32_t)((4 * hh + c) ^ (r & 7))) << 4;
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(drow + off), "r"(dsk[4 * c]), "r"(dsk[4 * c + 1]),
                       "r"(dsk[4 * c + 2]), "r"(dsk[4 * c + 3]) : "memory");
        }
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(ds_full);
    }
    // with the last Q buffer given back every product has been added up, and nothing reads the Q buffers any more
    if (ok && n_it > 0) ok = mbar_wait_warp(q_empty((n_it - 1) & 1), ((n_it - 1) >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN);
    if (ok && n_it > 0) {
      tc_fence_after_sync();
      if (kv_w + 32 <= p.S) {
        // The warp's 32 rows of dK and of dV, 64 columns each, leave through the Q buffers and the copy engine: row stores
        // of 16 bytes a thread were most of the 6000 clocks that a CTA's end took.
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          uint32_t a[64];
          tmem_ld_32x32b_x32((o ? t_dV : t_dK) + 64 * g + lane_off, *reinterpret_cast<uint32_t(*)[32]>(&a[0]));
          tmem_ld_32x32b_x32((o ? t_dV : t_dK) + 64 * g + 32 + lane_off, *reinterpret_cast<uint32_t(*)[32]>(&a[32]));
          tmem_wait_ld();
          const uint32_t stg = sQ(o) + g * G_HALF + (uint32_t)qd * 4096u;
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            const uint32_t addr = stg + lane * 128 + (((uint32_t)v ^ (uint32_t)(lane & 7)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                         "r"(pack_bf16x2(__uint_as_float(a[8 * v + 0]), __uint_as_float(a[8 * v + 1]))),
                         "r"(pack_bf16x2(__uint_as_float(a[8 * v + 2]), __uint_as_float(a[8 * v + 3]))),
                         "r"(pack_bf16x2(__uint_as_float(a[8 * v + 4]), __uint_as_float(a[8 * v + 5]))),
                         "r"(pack_bf16x2(__uint_as_float(a[8 * v + 6]), __uint_as_float(a[8 * v + 7])))
                         : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(o ? &tmDV : &tmDK, stg, hkv * G_D + 64 * g, (int)(row_base + kv_w));
            tma_store_commit();
          }
        }
        if (lane == 0) tma_store_wait_all<0>();
      } else {
        const bool row_ok = kv_i < p.S;
        __nv_bfloat16* dk_row = p.dk + (row_base + kv_i) * p.lddk + (long long)hkv * G_D;
        __nv_bfloat16* dv_row = p.dv + (row_base + kv_i) * p.lddv + (long long)hkv * G_D;
#pragma unroll
        for (int c = 2 * g; c < 2 * g + 2; ++c) {
          uint32_t a[32], e[32];
          tmem_ld_32x32b_x32(t_dK + 32 * c + lane_off, a);
          tmem_ld_32x32b_x32(t_dV + 32 * c + lane_off, e);
          tmem_wait_ld();
          if (row_ok) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 w, x;
              w.x = pack_bf16x2(__uint_as_float(a[8 * v + 0]), __uint_as_float(a[8 * v + 1]));
              w.y = pack_bf16x2(__uint_as_float(a[8 * v + 2]), __uint_as_float(a[8 * v + 3]));
              w.z = pack_bf16x2(__uint_as_float(a[8 * v + 4]), __uint_as_float(a[8 * v + 5]));
              w.w = pack_bf16x2(__uint_as_float(a[8 * v + 6]), __uint_as_float(a[8 * v + 7]));
              x.x = pack_bf16x2(__uint_as_float(e[8 * v + 0]), __uint_as_float(e[8 * v + 1]));
              x.y = pack_bf16x2(__uint_as_float(e[8 * v + 2]), __uint_as_float(e[8 * v + 3]));
              x.z = pack_bf16x2(__uint_as_float(e[8 * v + 4]), __uint_as_float(e[8 * v + 5]));
              x.w = pack_bf16x2(__uint_as_float(e[8 * v + 6]), __uint_as_float(e[8 * v + 7]));
              reinterpret_cast<uint4*>(dk_row + 32 * c)[v] = w;
              reinterpret_cast<uint4*>(dv_row + 32 * c)[v] = x;
            }
          }
        }
      }
    }
    tc_fence_before_sync();
  } else {
    // ===================== dQ read-out warpgroup: one query row per thread =====================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int qd = warp & 3;
    const int r = qd * 32 + lane;
    const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
    // Each warp stages its own 32 rows and hands them to the copy engine by itself, two units in flight: with one tile
    // for the four warps every unit waited for the slowest warp and for the previous unit to leave shared memory,
    // which kept the next tile's dQ waiting (4 x 2048, 16 heads: 339 -> 311 us; 2 x 4096, 32 / 8 heads: 1003 -> 897 us).
    const uint32_t my_stg = sStg + (uint32_t)qd * 2u * G_DQ_STG;
    for (int it = 0; it < n_it; ++it) {
      const int h = hkv * group + it / per_head;
      const int q0 = (qt0 + it % per_head) * G_T;
      if (!mbar_wait_warp(dq_full, it & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
      tc_fence_after_sync();
      uint32_t dq[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_dP + 32 * c + lane_off, *reinterpret_cast<uint32_t(*)[32]>(&dq[32 * c]));
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(dq_empty);
      // Rows past the end of this sequence would land in the next sequence's rows: they add zeros.
      const bool row_ok = q0 + r < p.S;
#pragma unroll
      for (int u = 0; u < 4; ++u) {            // four 32-column units of 128 bytes per row
        const uint32_t buf = my_stg + (u & 1u) * G_DQ_STG;
        const uint32_t rowaddr = buf + lane * 128;
        if (lane == 0) tma_store_wait_read<1>();   // the unit before the previous one has been read out of this buffer
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t addr = rowaddr + (((uint32_t)c ^ (uint32_t)(lane & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(row_ok ? dq[32 * u + 4 * c] : 0u),
                       "r"(row_ok ? dq[32 * u + 4 * c + 1] : 0u), "r"(row_ok ? dq[32 * u + 4 * c + 2] : 0u),
                       "r"(row_ok ? dq[32 * u + 4 * c + 3] : 0u) : "memory");
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                       ::"l"(reinterpret_cast<uint64_t>(&tmDQ)), "r"(buf), "r"(h * G_D + 32 * u), "r"((int)(row_base + q0) + qd * 32)
                       : "memory");
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
    tc_fence_before_sync();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, G_TMEM_COLS);
  }
}

// Launches the main kernel only; the caller has zeroed dq_accum and filled lse2 / delta.
int launch_flash_bwd_ws(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                        float* dq_accum, void* dk, void* dv, const float* lse2, const float* delta, int stat_pitch, long long lddk, long long lddv,
                        int B, int S, int Hq, int Hkv, float scale, int causal, cudaStream_t st) {
  FlashBwdWsParams p;
  p.dq_accum = dq_accum;
  p.dk = static_cast<__nv_bfloat16*>(dk);
  p.dv = static_cast<__nv_bfloat16*>(dv);
  p.lse2 = lse2;
  p.delta = delta;
  p.stat_pitch = stat_pitch;
  p.lddk = lddk; p.lddv = lddv;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.err = device_status_word();
  MLF_REQUIRE(p.err != nullptr, "no device status word");
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    MLF_CHECK_CUDA(cudaFuncSetAttribute(flash_bwd_ws_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G_SMEM));
    attr_set[dev & 63] = true;
  }
  // fp32 dQ accumulator as a 2-D tensor [tokens, Hq * 128]: tiles of 32 columns x 32 rows, 128B swizzle
  CUtensorMap tdq;
  {
    const int rc = make_tmap_2d(&tdq, dq_accum, 4, (uint64_t)Hq * G_D, (uint64_t)B * S, (uint64_t)Hq * G_D, 32, 32, true);
    if (rc) return rc;
  }
  CUtensorMap tdk, tdv;
  int rc;
  if ((rc = cached_tmap_bf16(&tdk, dk, (uint64_t)Hkv * G_D, (uint64_t)B * S, (uint64_t)lddk, 64, 32))) return rc;
  if ((rc = cached_tmap_bf16(&tdv, dv, (uint64_t)Hkv * G_D, (uint64_t)B * S, (uint64_t)lddv, 64, 32))) return rc;
  dim3 grid(((S + G_T - 1) / G_T) * Hkv * B);
  MLF_CHECK_CUDA(launch_pdl(flash_bwd_ws_kernel, grid, dim3(G_THREADS), G_SMEM, st, tq, tk, tv, tdo, tdq, tdk, tdv, p));
  count_launch();
  return 0;
}

}  // namespace mlf
