// bf16 GEMM with CTA-pair tensor-core instructions (tcgen05.mma.cta_group::2).
//
// Two CTAs on neighbouring SMs (a cluster of 2) compute one 256 x 256 output tile: each CTA
// stages its own 128 rows of A and its own half (128 columns) of B, and one tcgen05.mma issued by
// the leader CTA drives both tensor cores, each reading the peer's half of B from the peer's
// shared memory. Per SM and per k-block that is 16 KB of A + 16 KB of B for 128 x 256 x 64 of
// math, instead of 16 KB + 32 KB in the single-CTA kernel: the L2 -> shared-memory traffic, which
// bounds the single-CTA kernel near 63 % tensor-pipe utilisation, drops by a third. No load is
// shared between CTAs through the copy engine: every CTA fetches exactly the bytes it owns.
//
// Synchronisation (all barriers live at the same shared-memory offsets in both CTAs):
//   full[s]   in the leader, count 1: the leader's producer arrives with the byte count of both
//             CTAs' loads; every load of the pair completes on that barrier (2-SM form of the TMA
//             load). A peer load may land before the leader's arrive of the same phase, never in
//             an earlier phase: the peer refills a stage only after the MMAs that read it are done.
//   empty[s]  in each CTA: the leader commits twice after the k-block's MMAs, once to its own and
//             once to the peer's barrier (address translated with mapa).
//   tfull[a]  in each CTA (same double commit), tempty[a] in the leader, count 8 or 16: the
//             epilogue warps of each CTA arrive (the peer's through a cluster-scope arrive).
// When the last round of tiles would occupy at most half of the pairs, its tiles run as two items of 128 columns each.
// Every wait is bounded; a cluster barrier at the end keeps either CTA from exiting while the
// other may still touch its shared memory.
#include <cooperative_groups.h>

#include "gemm_common.cuh"

namespace mlf {

int cached_tmap_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t bi, uint32_t bo, bool swizzle = true);

constexpr int T2_BN = 256;                       // tile columns (both CTAs)
constexpr int T2_BNH = 128;                      // columns of B staged per CTA
constexpr int T2_STAGE_A = BM * BK * 2;          // 16 KB
constexpr int T2_STAGE_B = T2_BNH * BK * 2;      // 16 KB
constexpr int T2_STAGE = T2_STAGE_A + T2_STAGE_B;
constexpr int T2_STAGES = 6;
constexpr int T2_EPI_WARPS = 8;
constexpr int T2_THREADS = 64 + 32 * T2_EPI_WARPS;
constexpr int T2_STG_BYTES = 32 * 64 * 2;      // staging tile of one epilogue warp: 32 rows x 64 bf16 columns, 128B-swizzled
constexpr int T2_SMEM = T2_STAGES * T2_STAGE + 1024 /*barriers*/ + T2_EPI_WARPS * T2_STG_BYTES + 1024 /*align*/;
constexpr int T2_TMEM_COLS = 512;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_cluster(uint32_t cluster_addr, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(cluster_addr), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-SM TMA tile load: data lands in this CTA's shared memory, completion bytes are counted on the
// barrier at `bar_cluster_addr`, which may belong to the peer CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* tm, int x, int y, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_ss_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at a cluster address once all MMAs issued so far by this thread are done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// Output tensor maps of the row owners when the epilogue routes rows to peers (GEMM -> reduce-scatter).
struct alignas(64) PeerMaps {
  CUtensorMap m[8];
};

// TMA reduction store: global[tile] += shared[tile], element type taken from the tensor map (bf16).
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* tm, uint32_t smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_src), "r"(x), "r"(y)
               : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(T2_THREADS, 1)
gemm_tcgen05_2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const __grid_constant__ CUtensorMap tmOut, const __grid_constant__ CUtensorMap tmPre,
                         const __grid_constant__ CUtensorMap tmAux, const __grid_constant__ PeerMaps peer_maps,
                         const GemmKernelParams p, const int tma_epilogue, const int tma_aux, const int k_splits,
                         const int reduce_out, const int epi_halves, const int n_whole) {
  // Copy CTAs come in whole clusters (their count is even) and never touch the cluster barrier.
  if ((int)blockIdx.x < p.n_copy_ctas) {
    gather_copy_role(p);
    return;
  }
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + T2_STAGES * T2_STAGE;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (T2_STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * T2_STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * T2_STAGES + 2 + a); };
  auto aux_bar = [&](int w) { return bar_base + 8u * (2 * T2_STAGES + 4 + w); };   // aux_in tile of epilogue warp w landed
  const uint32_t stg_base = bar_base + 1024u;                        // staging tiles of the epilogue warps
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem_al + T2_STAGES * T2_STAGE + 8 * (2 * T2_STAGES + 4 + T2_EPI_WARPS));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();     // 0 = leader
  const uint32_t peer = rank ^ 1u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T2_STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 8 * epi_halves);
    }
    for (int w = 0; w < T2_EPI_WARPS; ++w) mbar_init(aux_bar(w), 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_ptr_smem), T2_TMEM_COLS);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                          // both CTAs' barriers are initialised before any remote arrive
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_trigger();                               // tensor memory is allocated: the next kernel may become resident

  const int pair = ((int)blockIdx.x - p.n_copy_ctas) >> 1;
  const int n_pairs = ((int)gridDim.x - p.n_copy_ctas) >> 1;
  // Work items: (tile, k-split). Splits of one tile are consecutive items, their partial products meet in
  // global memory through TMA reduction stores (the host cleared or kept `out` accordingly).
  // Tiles from n_whole on (k_splits is 1 then) are two items each, of 128 columns.
  const int whole_items = n_whole * k_splits;
  const int num_items = whole_items + 2 * (p.tiles_m * p.tiles_n - n_whole);
  auto item_at = [&](int t, int& tm, int& col0, int& cols) {
    int tile = t / k_splits, tn;
    cols = T2_BN;
    col0 = 0;
    if (t >= whole_items) {
      tile = n_whole + ((t - whole_items) >> 1);
      cols = T2_BN / 2;
      col0 = ((t - whole_items) & 1) * cols;
    }
    tile_coords(tile, p.tiles_m, p.tiles_n, p.rot_m, p.rot_n, tm, tn);
    col0 += tn * T2_BN;
  };
  const int num_kb_all = (p.K + BK - 1) / BK;
  const int kb_per = (num_kb_all + k_splits - 1) / k_splits;

  if (warp == 0) {
    // ===================== TMA producer (both CTAs) =====================
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      // A weight that nobody writes starts streaming while the kernels ahead are still running: the first pass over
      // the ring gets its B halves here, its A halves after the wait.
      int pre = 0;
      // `cols / 2` columns of B per CTA, 64 of them (8 KB) per load
      auto load_b = [&](uint32_t sb, int k0, int n0, int cols, uint32_t bar) {
        for (int j = 0; j < cols / 128; ++j) {
          const int n = n0 + 64 * j;
          tma_load_2d_pair(sb + j * (BK * 128), &tmB, p.b_mn ? n : k0, p.b_mn ? k0 : n, bar);
        }
      };
      if (p.b_static && pair < num_items) {
        int tm, col0, cols;
        item_at(pair, tm, col0, cols);
        const int kb0 = (pair % k_splits) * kb_per, kb1 = min(num_kb_all, kb0 + kb_per);
        const int n0 = col0 + (int)rank * (cols / 2);
        for (; pre < T2_STAGES && kb0 + pre < kb1; ++pre) {
          const uint32_t sb = smem_base + pre * T2_STAGE + T2_STAGE_A;
          const uint32_t lead_full = mapa_u32(full_bar(pre), 0);
          if (rank == 0) mbar_expect_tx(full_bar(pre), 2 * T2_STAGE_A + cols * (BK * 2));
          load_b(sb, (kb0 + pre) * BK, n0, cols, lead_full);
        }
      }
      pdl_wait();
      for (int t = pair; t < num_items; t += n_pairs) {
        int tm, col0, cols;
        item_at(t, tm, col0, cols);
        const int kb0 = (t % k_splits) * kb_per, kb1 = min(num_kb_all, kb0 + kb_per);
        if (kb0 >= kb1) continue;
        const int m0 = tm * 256 + (int)rank * BM;
        const int n0 = col0 + (int)rank * (cols / 2);
        bool ok = true;
        if (p.gather_operand != 0) {
          // this CTA's 128 rows of the gathered operand must have landed
          const int r0 = p.gather_operand == 1 ? m0 : n0;
          const int r1 = min(p.total_rows, r0 + 128) - 1;
          for (int c = r0 / p.flag_rows; c <= r1 / p.flag_rows && ok; ++c)
            ok = wait_flag_ge_gpu(&p.counters[c], (uint32_t)p.copy_group, abort_flag, p.err, ERR_WAIT_CHUNK_FLAG);
          if (!ok) break;
          fence_proxy_async_all();
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          const bool b_loaded = pre > 0;
          if (b_loaded) --pre;
          else if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, p.err, ERR_WAIT_SMEM_EMPTY)) { ok = false; break; }
          const uint32_t sa = smem_base + s * T2_STAGE;
          const uint32_t sb = sa + T2_STAGE_A;
          const uint32_t lead_full = mapa_u32(full_bar(s), 0);
          if (rank == 0 && !b_loaded) mbar_expect_tx(full_bar(s), 2 * T2_STAGE_A + cols * (BK * 2));
          const int k0 = kb * BK;
          if (!p.a_mn) {
            tma_load_2d_pair(sa, &tmA, k0, m0, lead_full);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * (BK * 128), &tmA, m0 + 64 * j, k0, lead_full);
          }
          if (!b_loaded) load_b(sb, k0, n0, cols, lead_full);
          if (++s == T2_STAGES) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader CTA only) =====================
    if (rank == 0 && elect_one()) {
      const uint32_t idesc_whole = make_idesc_bf16(256, T2_BN, p.a_mn, p.b_mn);
      const uint32_t idesc_half = make_idesc_bf16(256, T2_BN / 2, p.a_mn, p.b_mn);
      const uint32_t a_lbo = p.a_mn ? BK * 128 : 16, a_kstep = p.a_mn ? UMMA_K * 128 : UMMA_K * 2;
      const uint32_t b_lbo = p.b_mn ? BK * 128 : 16, b_kstep = p.b_mn ? UMMA_K * 128 : UMMA_K * 2;
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      bool ok = true;
      // The first A tile is requested behind the producer's wait for the kernels ahead: waiting for it from before that
      // would count their remaining run time against this kernel's wait budget.
      pdl_wait();
      for (int t = pair; t < num_items && ok; t += n_pairs) {
        const uint32_t idesc = t < whole_items ? idesc_whole : idesc_half;
        const int kb0 = (t % k_splits) * kb_per, kb1 = min(num_kb_all, kb0 + kb_per);
        if (kb0 >= kb1) continue;
        const int acc = it & 1;
        const uint32_t acc_ph = (it >> 1) & 1;
        if (!mbar_wait(tempty_bar(acc), acc_ph ^ 1u, abort_flag, p.err, ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * T2_BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(full_bar(s), ph, abort_flag, p.err, ERR_WAIT_SMEM_FULL)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_base + s * T2_STAGE;
          const uint32_t sb = sa + T2_STAGE_A;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t ad = make_smem_desc_sw128(sa + k * a_kstep, a_lbo, 1024);
            const uint64_t bd = make_smem_desc_sw128(sb + k * b_kstep, b_lbo, 1024);
            umma_bf16_ss_pair(d_tmem, ad, bd, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit_pair(mapa_u32(empty_bar(s), 0));
          umma_commit_pair(mapa_u32(empty_bar(s), 1));
          if (++s == T2_STAGES) { s = 0; ph ^= 1u; }
        }
        if (ok) {
          umma_commit_pair(mapa_u32(tfull_bar(acc), 0));
          umma_commit_pair(mapa_u32(tfull_bar(acc), 1));
        }
        ++it;
      }
    }
  } else if (warp < 2 + 4 * epi_halves) {
    // ===================== epilogue (warps 2..5 or 2..9 of both CTAs) =====================
    // One warp per 32-lane quarter of the accumulator, or two with half of the columns each (epi_halves). A warp stages
    // its own 32 rows x 64 columns and hands them to the copy engine by itself, so that no warp waits for another one.
    pdl_wait();                                // `out` and aux_in may be in use by earlier kernels until here
    const int q = warp & 3;
    const int ew = warp - 2;
    const int half = ew >> 2;                  // which half of the tile's columns (0 when there is one warp per quarter)
    const bool two_bufs = epi_halves == 1;     // the staging tiles of the absent warps are the second ones; never with an aux tile
    const bool out_fp32 = (p.flags & MLF_EPI_OUT_FP32) != 0;
    const bool swiglu = (p.flags & MLF_EPI_SWIGLU) != 0;
    const bool dswiglu = (p.flags & MLF_EPI_DSWIGLU) != 0;
    // Column units of this warp: 64 accumulator columns, or 32 where (gate, up) pairs make 64 output columns of them.
    const int unit_cols = dswiglu ? 32 : 64;
    const uint32_t stg0 = stg_base + (uint32_t)ew * T2_STG_BYTES;
    uint32_t emits = 0;                        // staging tiles handed out by this warp
    uint32_t aux_units = 0;                    // aux tiles consumed by this warp
    // aux_in (residual, dGELU or dSwiGLU input) comes in through the warp's one staging tile: the next unit's is requested
    // when the store of this unit has read the tile, the first one of a tile while its products are still running
    int ax_t = pair, ax_u = -1;                // unit whose aux tile was requested last
    auto request_aux = [&]() {                 // lane 0; the staging tile it goes to is free
      while (true) {
        ++ax_u;
        if (ax_t >= num_items) return;
        int tm, col0, cols;
        item_at(ax_t, tm, col0, cols);         // k_splits is 1 whenever there is an aux_in
        const int my_cols = cols / epi_halves;
        if (ax_u * unit_cols >= my_cols) { ax_u = -1; ax_t += n_pairs; continue; }
        const int nb = col0 + half * my_cols + ax_u * unit_cols;
        if (nb >= p.N) continue;
        mbar_expect_tx(aux_bar(ew), T2_STG_BYTES);
        tma_load_2d(stg0, &tmAux, dswiglu ? 2 * nb : nb, tm * 256 + (int)rank * BM + q * 32, aux_bar(ew));
        return;
      }
    };
    if (tma_aux && lane == 0) request_aux();
    int it = 0;
    for (int t = pair; t < num_items; t += n_pairs) {
      if ((t % k_splits) * kb_per >= min(num_kb_all, (t % k_splits) * kb_per + kb_per)) continue;
      const int acc = it & 1;
      const uint32_t acc_ph = (it >> 1) & 1;
      int tm, col0, cols;
      item_at(t, tm, col0, cols);
      const int my_cols = cols / epi_halves;
      const int n_units = my_cols / unit_cols;
      const int m0 = tm * 256 + (int)rank * BM;
      const int m = m0 + q * 32 + lane;
      const int nh = col0 + half * my_cols;                             // first column of this warp
      const uint32_t t_acc = tmem_base + acc * T2_BN + half * my_cols + ((uint32_t)(q * 32) << 16);
      if (!mbar_wait_warp(tfull_bar(acc), acc_ph, abort_flag, p.err, ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after_sync();
      const bool row_ok = m < p.M;
      if (tma_epilogue) {
        // a staged row: 64 columns (128 bytes) at x of tmap, or 32 columns (64 bytes, not swizzled) when narrow
        auto emit = [&](const float* v, const CUtensorMap* tmap, int x, bool narrow) {
          const uint32_t buf = stg0 + (two_bufs ? (emits & 1u) * 4u * T2_STG_BYTES : 0u);
          if (!tma_aux) {                      // with an aux tile the buffer is free: its store was waited for before the request
            if (lane == 0) {
              if (two_bufs) tma_store_wait_read<1>();
              else tma_store_wait_read<0>();
            }
            __syncwarp();
          }
          if (!narrow) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const uint32_t addr = buf + lane * 128 + (((uint32_t)c ^ (uint32_t)(lane & 7)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(pack_bf16x2(v[8 * c], v[8 * c + 1])),
                           "r"(pack_bf16x2(v[8 * c + 2], v[8 * c + 3])), "r"(pack_bf16x2(v[8 * c + 4], v[8 * c + 5])),
                           "r"(pack_bf16x2(v[8 * c + 6], v[8 * c + 7])) : "memory");
            }
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(buf + lane * 64 + c * 16), "r"(pack_bf16x2(v[8 * c], v[8 * c + 1])),
                           "r"(pack_bf16x2(v[8 * c + 2], v[8 * c + 3])), "r"(pack_bf16x2(v[8 * c + 4], v[8 * c + 5])),
                           "r"(pack_bf16x2(v[8 * c + 6], v[8 * c + 7])) : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int y = m0 + q * 32;
            if (p.scatter_out) {                 // the whole 128-row block belongs to one owner (possibly a peer)
              const int owner = min(m0 / p.rows_per_owner, p.world - 1);
              tma_store_2d(&peer_maps.m[owner], buf, x, p.rank * p.rows_per_owner + (y - owner * p.rows_per_owner));
            } else if (reduce_out) {
              tma_reduce_add_2d(tmap, buf, x, y);
            } else {
              tma_store_2d(tmap, buf, x, y);
            }
            tma_store_commit();
          }
          ++emits;
        };
        // this warp's aux row of the current unit, 64 bf16 in the staging tile
        auto aux_row = [&](float (&a)[64]) -> bool {
          if (!mbar_wait_warp(aux_bar(ew), aux_units & 1u, abort_flag, p.err, ERR_WAIT_TMEM_FULL)) return false;
          ++aux_units;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint4 w;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                         : "r"(stg0 + lane * 128 + (((uint32_t)c ^ (uint32_t)(lane & 7)) << 4)));
            const float2 f0 = unpack_bf16x2(w.x), f1 = unpack_bf16x2(w.y), f2 = unpack_bf16x2(w.z), f3 = unpack_bf16x2(w.w);
            a[8 * c + 0] = f0.x; a[8 * c + 1] = f0.y; a[8 * c + 2] = f1.x; a[8 * c + 3] = f1.y;
            a[8 * c + 4] = f2.x; a[8 * c + 5] = f2.y; a[8 * c + 6] = f3.x; a[8 * c + 7] = f3.y;
          }
          return true;
        };
        bool ok = true;
#pragma unroll 1
        for (int u = 0; u < n_units && ok; ++u) {
          const int nb = nh + u * unit_cols;
          if (nb >= p.N) break;
          if (dswiglu) {
            // v = dL/dh of 32 hidden columns; aux holds their (gate, up) pairs, out gets (dgate, dup)
            uint32_t t32[32];
            tmem_ld_32x32b_x32(t_acc + u * 32, t32);
            float gu[64];
            ok = aux_row(gu);
            if (!ok) break;
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float gate = gu[2 * j], up = gu[2 * j + 1], dh = __uint_as_float(t32[j]) * p.alpha;
              const float sg = 1.f / (1.f + __expf(-gate));
              gu[2 * j] = dh * up * sg * (1.f + gate * (1.f - sg));
              gu[2 * j + 1] = dh * gate * sg;
            }
            emit(gu, &tmOut, 2 * nb, false);
          } else {
            float v[64];
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
              uint32_t t32[32];
              tmem_ld_32x32b_x32(t_acc + u * 64 + h2 * 32, t32);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 32; ++j) v[32 * h2 + j] = __uint_as_float(t32[j]) * p.alpha;
            }
            const int nvalid = min(64, p.N - nb);
            if (p.flags & MLF_EPI_BIAS) {
              if (nvalid == 64 && ((reinterpret_cast<uintptr_t>(p.bias + nb) & 15) == 0)) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                  const uint4 w = reinterpret_cast<const uint4*>(p.bias + nb)[c];
                  const float2 f0 = unpack_bf16x2(w.x), f1 = unpack_bf16x2(w.y), f2 = unpack_bf16x2(w.z), f3 = unpack_bf16x2(w.w);
                  v[8 * c + 0] += f0.x; v[8 * c + 1] += f0.y; v[8 * c + 2] += f1.x; v[8 * c + 3] += f1.y;
                  v[8 * c + 4] += f2.x; v[8 * c + 5] += f2.y; v[8 * c + 6] += f3.x; v[8 * c + 7] += f3.y;
                }
              } else {
#pragma unroll
                for (int j = 0; j < 64; ++j)
                  if (j < nvalid) v[j] += __bfloat162float(p.bias[nb + j]);
              }
            }
            if (p.flags & MLF_EPI_STORE_PRE) emit(v, &tmPre, nb, false);
            if (swiglu) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = silu(v[2 * j]) * v[2 * j + 1];
              emit(v, &tmOut, nb / 2, true);
              continue;
            }
            if (p.flags & MLF_EPI_GELU) {
#pragma unroll
              for (int j = 0; j < 64; ++j) v[j] = gelu_tanh(v[j]);
            }
            if (p.flags & (MLF_EPI_RESIDUAL | MLF_EPI_DGELU_MUL)) {
              const bool resid = (p.flags & MLF_EPI_RESIDUAL) != 0;
              if (tma_aux) {
                float a[64];
                ok = aux_row(a);
                if (!ok) break;
#pragma unroll
                for (int j = 0; j < 64; ++j) v[j] = resid ? v[j] + a[j] : v[j] * dgelu_tanh(a[j]);
              } else if (row_ok) {
                const __nv_bfloat16* ar = p.aux_in + (long long)m * p.ld_aux_in + nb;
#pragma unroll
                for (int j = 0; j < 64; ++j) {
                  const float a1 = j < nvalid ? __bfloat162float(ar[j]) : 0.f;
                  v[j] = resid ? v[j] + a1 : v[j] * dgelu_tanh(a1);
                }
              }
            }
            emit(v, &tmOut, nb, false);
          }
          if (tma_aux && lane == 0) {          // the next unit's aux tile, once the store that read its buffer is through
            tma_store_wait_read<0>();
            request_aux();
          }
        }
        if (!ok) break;
      } else {
        char* out_row = nullptr;
        if (row_ok) {
          const int esz = out_fp32 ? 4 : 2;
          if (p.scatter_out) {               // rows routed to their owner's partial buffer (possibly on a peer)
            const int owner = min(m / p.rows_per_owner, p.world - 1);
            const long long lr = (long long)p.rank * p.rows_per_owner + (m - owner * p.rows_per_owner);
            out_row = static_cast<char*>(p.out_peer[owner]) + lr * p.ldo * esz;
          } else {
            out_row = static_cast<char*>(p.out) + (long long)m * p.ldo * esz;
          }
        }
#pragma unroll 1
        for (int c = 0; c < my_cols / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_acc + c * 32, r);
          tmem_wait_ld();
          const int nb = nh + c * 32;
          if (!row_ok || nb >= p.N) continue;
          gemm_epilogue_chunk(p, m, nb, r, out_row, out_fp32, swiglu, dswiglu);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(tempty_bar(acc), 0));
      ++it;
    }
    if (tma_epilogue && lane == 0) tma_store_wait_all<0>();   // shared memory stays valid until the copies have read it
  }

  // ===================== teardown =====================
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();                          // neither CTA leaves while the other may still signal it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, T2_TMEM_COLS);
  }
}

}  // namespace mlf

using namespace mlf;

// Clears the output that the splits of K add into (rows 16-byte aligned, pitch in elements). A kernel with launch overlap on
// both sides in place of a memset, behind which neither the one nor the product's ramp overlaps (a step with
// 17 of them, 2.9 ms: 25 us).
namespace mlf {
__global__ void __launch_bounds__(256) clear_rows_kernel(__nv_bfloat16* out, int M, int N, long long ld) {
  const int nv = (N + 7) / 8;
  pdl_trigger();
  pdl_wait();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)M * nv; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % nv) * 8;
    __nv_bfloat16* dst = out + i / nv * ld + c;
    if (c + 8 <= N) *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
    else for (int j = c; j < N; ++j) *dst++ = __float2bfloat16(0.f);
  }
}
}  // namespace mlf

// A last round with work for at most half of the pairs: its tiles are cut into two items of 128 columns each, which
// costs 0.8 - 0.9 of a whole round (at N = 128 an MMA reads A from shared memory for half the math), with the same sums:
// 8192 x 2048 x 2048 49.4 -> 46.8 us, 8192 x 2048 x 8192 189.5 -> 185.3, 8192 x 2048 x 50304 1189 -> 1124,
// 4096 x 4096 x 4096 with a residual 102.1 -> 98.3. Above half a round two of the items would meet on one pair again.
namespace mlf {
bool halves_last_round(int num_tiles, int pairs) {
  const int rest = num_tiles % pairs;
  return rest > 0 && 2 * rest <= pairs;
}
}  // namespace mlf

// Parts of K for `num_tiles` tiles on `pairs` CTA pairs when the tiles alone cannot fill the GPU (weight gradients of
// narrow layers: few tiles, long K). Splits add their partial products into `out` with TMA reduction stores.
// Candidates are the counts that save a tenth of the rounds each, coarse ones first. One is taken when it saves a fifth
// of the time that the product takes in one piece (its last round halved where that applies): a split clears the output,
// adds every tile once more in L2 and rounds the partial sums to bf16. Cost in rounds, then us and the error against 64
// bits in units of 1e-3, in one piece and split:
//   75 tiles 1.20 of 1.80 (1280 x 3840 x 8192 in six)  74.8 / 1.66 and 65.1 / 3.62     taken
//   96 tiles 1.33 of 1.80 (2048 x 3072 x 8192 in three) 78.0 / 1.66 and 73.5 / 2.85    taken
//  100 tiles 1.50 of 1.80 (2560 x 2560 in two, K = 8192) 80.8 / 1.66 and 77.8 / 2.45, (K = 4096) 42.8 and 44.7   not
//  108 tiles 1.50 of 1.80 (2304 x 3072 in two, K = 8192) 85.1 and 81.4, (K = 4096) 43.2 and 45.4                 not
//  112 tiles 1.67 of 2.00 (2048 x 3584 in three, K = 8192) 88.1 and 87.0, (K = 4096) 48.4 and 50.1               not
//   56 tiles 0.80 of 1.00 (2048 x 1792 in five, K = 8192) 49.4 and 48.1, (K = 4096) 28.8 and 33.0                not
//  128 tiles 1.75 of 2.00 (2048 x 4096 x 14336 in four) 161 and 170                                              not
// A finer count never stands in for a coarse one that does not pay: 100 tiles in five (1.40) take 79.5 us at K = 8192 and
// 49.4 at 4096, with twice the error of one piece.
MLF_API int mlf_gemm_k_splits(int num_tiles, int K, int pairs) {
  const int kb_all = (K + BK - 1) / BK;
  double best = (double)((num_tiles + pairs - 1) / pairs);
  const double whole = best - (halves_last_round(num_tiles, pairs) ? 0.2 : 0.0);
  int k_splits = 1;
  for (int ks = 2; ks <= 8 && kb_all / ks >= 8; ++ks) {
    const double cost = (double)((num_tiles * ks + pairs - 1) / pairs) / ks;
    if (cost >= best * 0.9) continue;
    best = cost;
    if (cost < whole * 0.8) k_splits = ks;
  }
  return k_splits;
}

// GEMM on CTA pairs, with the same in-kernel communication options as the single-CTA kernel (copy
// CTAs that gather an operand or prefetch extra segments; an epilogue that routes rows to their
// owners). Same arguments as mlf_gemm_bf16; returns -4 without launching when the problem is not a
// fit (the caller then uses the single-CTA kernel). split_few_rows: a plain product of up to 256 rows may split K, which
// the caller decides by its small_m rule; the partial products meet in bf16.
MLF_API int mlf_gemm_bf16_2cta(const MlfGemmArgs* a, int split_few_rows, uint64_t stream) {
  MLF_REQUIRE(a != nullptr, "null args");
  const MlfGemmComm* cm = a->comm;
  // one row of tiles that is mostly padding only as a plain product (optionally accumulated), where K is split over the pairs
  if (a->N < 256 || (a->M < 256 && cm != nullptr) ||
      (a->M <= 128 && (a->flags & ~(MLF_EPI_ACCUM | MLF_EPI_B_STATIC)) != 0)) return -4;
  const bool gatherA = cm && cm->gather_operand == 1;
  const bool gatherB = cm && cm->gather_operand == 2;
  if (cm && cm->gather_operand && (cm->flag_rows <= 0 || cm->flag_rows % 128 != 0)) return -4;
  if (cm && cm->scatter_out && cm->rows_per_owner % 128 != 0) return -4;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  GemmKernelParams p;
  memset(&p, 0, sizeof(p));
  p.M = a->M; p.N = a->N; p.K = a->K;
  p.a_mn = a->a_mn ? 1 : 0; p.b_mn = a->b_mn ? 1 : 0;
  p.flags = a->flags; p.alpha = a->alpha;
  p.b_static = (a->flags & MLF_EPI_B_STATIC) != 0 && cm == nullptr ? 1 : 0;
  p.out = a->out;
  p.bias = static_cast<const __nv_bfloat16*>(a->bias);
  p.aux_in = static_cast<const __nv_bfloat16*>(a->aux_in);
  p.aux_out = static_cast<__nv_bfloat16*>(a->aux_out);
  p.ldo = a->ldo; p.ld_aux_in = a->ld_aux_in; p.ld_aux_out = a->ld_aux_out;
  p.tiles_m = (a->M + 255) / 256;
  p.tiles_n = (a->N + T2_BN - 1) / T2_BN;
  p.err = device_status_word();
  MLF_REQUIRE(p.err != nullptr, "no device status word");
  if ((a->flags & MLF_EPI_BIAS)) MLF_REQUIRE(a->bias, "MLF_EPI_BIAS without bias");
  if ((a->flags & (MLF_EPI_RESIDUAL | MLF_EPI_DGELU_MUL | MLF_EPI_DSWIGLU))) MLF_REQUIRE(a->aux_in, "epilogue needs aux_in");
  if ((a->flags & MLF_EPI_STORE_PRE)) MLF_REQUIRE(a->aux_out, "MLF_EPI_STORE_PRE without aux_out");
  const int sms_all = a->max_ctas > 0 ? a->max_ctas : sm_count();
  const void* a_base = a->a;
  const void* b_base = a->b;
  int n_copy = 0;
  if (cm && (cm->gather_operand || cm->n_extra > 0)) {
    MLF_REQUIRE(cm->n_copy_ctas >= 1 && cm->n_copy_ctas + 2 < sms_all, "n_copy_ctas out of range");
    n_copy = (cm->n_copy_ctas + 1) & ~1;          // whole clusters
    p.n_copy_ctas = n_copy;
    p.copy_group = 1;
    p.extra_segs = cm->extra_segs;
    p.n_extra = cm->n_extra;
  }
  if (cm && cm->gather_operand) {
    MLF_REQUIRE(cm->world >= 1 && cm->world <= 8, "world %d out of range", cm->world);
    MLF_REQUIRE(cm->rows_per_rank % cm->flag_rows == 0, "rows_per_rank must be a multiple of flag_rows");
    MLF_REQUIRE(cm->row_bytes % 16 == 0, "row_bytes must be a multiple of 16");
    MLF_REQUIRE(!(gatherA && a->a_mn) && !(gatherB && a->b_mn), "gathered operand must be K-major");
    p.gather_operand = cm->gather_operand;
    p.world = cm->world; p.rank = cm->rank;
    p.rows_per_rank = cm->rows_per_rank; p.flag_rows = cm->flag_rows; p.row_bytes = cm->row_bytes;
    p.copy_group = copy_group_size(n_copy, (long long)cm->flag_rows * cm->row_bytes);
    p.total_rows = gatherA ? a->M : a->N;
    for (int r = 0; r < 8; ++r) p.src[r] = cm->src[r];
    p.gathered = cm->gathered;
    p.flags_ready = cm->flags; p.counters = cm->counters;
    // start with the tiles whose rows are already local
    if (gatherA) { a_base = cm->gathered; p.rot_m = (cm->rank * cm->rows_per_rank) / 256; }
    else { b_base = cm->gathered; p.rot_n = (cm->rank * cm->rows_per_rank) / T2_BN; }
    if (p.rot_m >= p.tiles_m) p.rot_m = 0;
    if (p.rot_n >= p.tiles_n) p.rot_n = 0;
  }
  if (cm && cm->scatter_out) {
    MLF_REQUIRE(cm->world >= 1 && cm->world <= 8, "world %d out of range", cm->world);
    p.scatter_out = 1; p.rows_per_owner = cm->rows_per_owner;
    p.world = cm->world; p.rank = cm->rank;
    for (int r = 0; r < 8; ++r) p.out_peer[r] = cm->out_peer[r];
    p.rot_m = (((cm->rank + 1) % cm->world) * cm->rows_per_owner) / 256;   // remote traffic starts first
    if (p.rot_m >= p.tiles_m) p.rot_m = 0;
  }
  CUtensorMap tmA, tmB;
  int rc;
  if (!a->a_mn) rc = cached_tmap_bf16(&tmA, a_base, a->K, a->M, a->lda, BK, BM);
  else rc = cached_tmap_bf16(&tmA, a_base, a->M, a->K, a->lda, 64, BK);
  if (rc) return rc;
  if (!a->b_mn) rc = cached_tmap_bf16(&tmB, b_base, a->K, a->N, a->ldb, BK, 64);
  else rc = cached_tmap_bf16(&tmB, b_base, a->N, a->K, a->ldb, 64, BK);
  if (rc) return rc;
  // Outputs go through TMA stores when they are bf16 rows with aligned pitches.
  CUtensorMap tmOut = tmA, tmPre = tmA, tmAux = tmA;
  PeerMaps peer_maps;                        // only read by the kernel when rows are routed
  memset(&peer_maps, 0, sizeof(peer_maps));
  int tma_epi = 0, tma_aux = 0;
  const bool scatter = cm && cm->scatter_out;
  const bool plain = (a->flags & ~(MLF_EPI_ACCUM | MLF_EPI_B_STATIC)) == 0 && cm == nullptr;      // nothing but (optionally) out += product
  const bool sw = (a->flags & MLF_EPI_SWIGLU) != 0, dsw = (a->flags & MLF_EPI_DSWIGLU) != 0;
  const bool aux_aligned = a->ld_aux_in % 8 == 0 && (reinterpret_cast<uintptr_t>(a->aux_in) & 15) == 0;
  // (gate, up) forms: no other operation beside theirs, whole pairs, and the aux tile through the copy engine
  const bool gated_ok = !(sw || dsw) || (!scatter && !(sw && dsw) && a->N % 2 == 0 &&
                                         !(a->flags & (MLF_EPI_GELU | MLF_EPI_RESIDUAL | MLF_EPI_DGELU_MUL)) &&
                                         (!dsw || (aux_aligned && !(a->flags & (MLF_EPI_STORE_PRE | MLF_EPI_BIAS)))));
  if (!(a->flags & MLF_EPI_OUT_FP32) && gated_ok && (!(a->flags & MLF_EPI_ACCUM) || plain) && a->ldo % 8 == 0 &&
      (scatter || (reinterpret_cast<uintptr_t>(a->out) & 15) == 0) &&
      (!(a->flags & MLF_EPI_STORE_PRE) || (a->ld_aux_out % 8 == 0 && (reinterpret_cast<uintptr_t>(a->aux_out) & 15) == 0))) {
    if (scatter) {
      for (int r = 0; r < cm->world; ++r) {
        MLF_REQUIRE((reinterpret_cast<uintptr_t>(cm->out_peer[r]) & 15) == 0, "partial buffers must be 16-byte aligned");
        rc = cached_tmap_bf16(&peer_maps.m[r], cm->out_peer[r], a->N, (uint64_t)cm->world * cm->rows_per_owner, a->ldo, 64, 32);
        if (rc) return rc;
      }
    } else if (sw) {
      rc = cached_tmap_bf16(&tmOut, a->out, a->N / 2, a->M, a->ldo, 32, 32, false);
      if (rc) return rc;
    } else {
      rc = cached_tmap_bf16(&tmOut, a->out, dsw ? 2 * (uint64_t)a->N : a->N, a->M, a->ldo, 64, 32);
      if (rc) return rc;
    }
    if (a->flags & MLF_EPI_STORE_PRE) {
      rc = cached_tmap_bf16(&tmPre, a->aux_out, a->N, a->M, a->ld_aux_out, 64, 32);
      if (rc) return rc;
    }
    tma_epi = 1;
    if ((a->flags & (MLF_EPI_RESIDUAL | MLF_EPI_DGELU_MUL | MLF_EPI_DSWIGLU)) && !(a->flags & MLF_EPI_STORE_PRE) && aux_aligned) {
      rc = cached_tmap_bf16(&tmAux, a->aux_in, dsw ? 2 * (uint64_t)a->N : a->N, a->M, a->ld_aux_in, 64, 32);
      if (rc) return rc;
      tma_aux = 1;
    }
  }
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    MLF_CHECK_CUDA(cudaFuncSetAttribute(gemm_tcgen05_2cta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T2_SMEM));
    attr_set[dev & 63] = true;
  }
  const int sms = sms_all - n_copy;
  const int num_tiles = p.tiles_m * p.tiles_n;
  static int max_clusters[64] = {0};
  if (!max_clusters[dev & 63]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    cfg.blockDim = dim3(T2_THREADS);
    cfg.dynamicSmemBytes = T2_SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_tcgen05_2cta_kernel, &cfg) != cudaSuccess || n <= 0) n = sm_count() / 2;
    max_clusters[dev & 63] = n;
  }
  int avail = sms / 2;                       // CTA pairs that run at a time
  if (avail > max_clusters[dev & 63]) avail = max_clusters[dev & 63];
  if (avail < 1) avail = 1;
  const bool halve = cm == nullptr && halves_last_round(num_tiles, avail);
  // Below 512 rows a product keeps its single fp32 sum, a decode step's rows aside.
  const int k_splits = plain && tma_epi && ((split_few_rows && a->M <= 256) || a->M >= 512) ? mlf_gemm_k_splits(num_tiles, a->K, avail) : 1;
  const int n_whole = halve && k_splits == 1 ? num_tiles - num_tiles % avail : num_tiles;
  const int num_items = n_whole * k_splits + 2 * (num_tiles - n_whole);
  // Two epilogue warps per quarter where the work of one does not fit behind the next tile's products: gated and
  // derivative epilogues (8192 x 14336 x 4096 with dSwiGLU 960 -> 691 us, 4096 x 28672 x 4096 with SwiGLU 686 -> 612 us,
  // 8192 x 8192 x 2048 with dGELU 225 -> 211 us), a residual (its tile has to arrive first), and any short K (2331 x 4096
  // x 1024 with GELU 33.5 -> 28.1 us). Elsewhere the second warp only takes power from the products: 8192 x 8192 x 2048
  // plain 182 us with one, 186 us with two.
  // Every product with an aux tile is one of these: its loads use the one staging tile that a warp has then.
  const bool heavy = (a->flags & (MLF_EPI_DGELU_MUL | MLF_EPI_SWIGLU | MLF_EPI_DSWIGLU | MLF_EPI_RESIDUAL)) != 0;
  const int epi_halves = heavy || a->K <= 1024 * k_splits ? 2 : 1;
  const int reduce_out = (k_splits > 1 || (a->flags & MLF_EPI_ACCUM)) ? 1 : 0;
  if (k_splits > 1 && !(a->flags & MLF_EPI_ACCUM)) {
    const long long work = (long long)a->M * ((a->N + 7) / 8);
    MLF_CHECK_CUDA(launch_pdl(clear_rows_kernel, dim3((unsigned)min((work + 255) / 256, 8LL * sm_count())), dim3(256), 0, st,
                              static_cast<__nv_bfloat16*>(a->out), a->M, a->N, (long long)a->ldo));
    count_launch();
  }
  const int pairs = avail < num_items ? avail : num_items;
  if (cm == nullptr) {
    MLF_CHECK_CUDA(launch_pdl(gemm_tcgen05_2cta_kernel, dim3(2 * pairs), dim3(T2_THREADS), T2_SMEM, st, tmA, tmB, tmOut, tmPre, tmAux,
                              peer_maps, p, tma_epi, tma_aux, k_splits, reduce_out, epi_halves, n_whole));
  } else {                                       // copy CTAs and routed rows touch peers' memory: after everything ahead
    gemm_tcgen05_2cta_kernel<<<n_copy + 2 * pairs, T2_THREADS, T2_SMEM, st>>>(tmA, tmB, tmOut, tmPre, tmAux, peer_maps, p, tma_epi, tma_aux,
                                                                                k_splits, reduce_out, epi_halves, n_whole);
    MLF_CHECK_CUDA(cudaGetLastError());
  }
  count_launch();
  return 0;
}
