// Self-attention forward, head_dim 128: two 128-row query tiles per item, ping-ponged; a CTA goes from item to item.
//
// An item is 256 query rows of one (batch, head) as two tiles of 128. 384 threads in three warpgroups;
// the control warpgroup hands most of its registers to the softmax warpgroups (setmaxnreg 56 / 224 / 224 of 3 x 168). With fewer
// the softmax's instructions come in a slower order or spill, on the chain below: 128 queries of 4096 keys, one query tile
// alone, 53.4 us, 56.6 with 72 / 216; 4 x 2048, 16 heads 74.2, 75.0, and 4 % more with 88 / 208. So the MMA issuer gets by with few: no
// state of a tile is addressed by a variable (it would be in local memory), one descriptor per operand, stepped by constants:
//   warp 0        TMA producer: an item's Q tiles, its K and V tiles of 128 keys through 2-stage rings
//   warp 1        MMA issuer (one thread). Per key tile j and query tile t:
//                   S_t = Q_t K_j^T   (M128 N128 K128, operands in shared memory)  -> TMEM S_t
//                   O_t += P_t V_j    (M128 N128 K128, P read from TENSOR MEMORY, V from shared memory)
//                 issued in the order PV_0(j), S_0(j+1), PV_1(j), S_1(j+1) so that the tensor pipe
//                 works on one tile while the other tile's softmax runs (an issuing thread per tile lets the tiles fall
//                 into step: 2 x 4096, 32 / 8 heads 4 % slower)
//   warps 4..7    softmax of tile 0: one query row per thread; reads S_0 from TMEM into registers,
//                 running max / sum in the log2 domain, writes P_0 as packed bf16 back over S_0
//   warps 8..11   softmax of tile 1
// TMEM (512 columns): S_0 | S_1 | O_0 | O_1, 128 fp32 columns each; P_t occupies the first 64
// columns of S_t. The MMAs of one thread execute in issue order, so S_t(j+1) overwrites P_t(j)
// only after PV_t(j) has read it. O is rescaled lazily: only when a row's maximum has grown by
// more than 2^8 since the value P and O are expressed against (then O_t is read, scaled and
// written back by its softmax warps, after PV_t(j-1) has completed).
// The chain S -> P -> PV -> next S of a tile bounds the kernel (about 3300 clocks for 2048 of tensor work): P is published
// in halves so that PV starts on the first 64 keys while the exponentials of the others run, and the arithmetic around the
// exponentials is done two elements at a time. (Every eighth pair of exponentials as a polynomial on the FMA pipe, as exact as
// the special-function unit's, took 4 % off long sequences and changed every bit of the output; every fourth cost 1 %.)
// A CTA takes over items instead of ending with its first: set-up, the first loads and the write-out took a third of the
// clocks of an item of eight key tiles and two thirds of one of two. The next item's Q, K and V arrive and its first S is
// issued behind the last products of this one, while the softmax warps write its rows out, each through its own staging
// tile and the copy engine (32 rows of 16 bytes per store instruction took 2500 clocks). Only the 32-column blocks of a
// diagonal tile that a warp does not see whole are masked (2000 clocks a tile before).
// The grid has a CTA per item, the longest first; a CTA that nears its end has the launch control cancel one that has not
// started and does that one's item. Rounds of fixed shares (a CTA per SM) left the shares of CTAs that found no place beside
// another stream's kernel until the others had ended. us back to back, a CTA that ends with its item / fixed shares / now: 4 x 2048,
// 16 heads 98 / 85 / 78, with 1 SM held by another kernel 100 / 142 / 81, with 8 102 / 143 / 83; 8 x 512, 32 / 8 heads
// 54 / 41 / 38, 55 / 60 / 39, 57 / 61 / 40; 2 x 4096, 32 / 8 heads 284 / 264 / 245, 292 / 471 / 255, 307 / 474 / 263.
// Per SM and key tile: 4 x 128x128x128 of tensor work against 2 x 16384 exponentials.
//
// Math reference: StandardPagedAttentionKernel.ComputePagedAttention
// (src/MLFramework/Inference/PagedAttention/Kernels/StandardPagedAttentionKernel.cs:21-84;
// causal rule :219-255).
#include <float.h>

#include "../common/host.h"
#include "../common/ptx.cuh"
#include "../mlf_api.h"

namespace mlf {

int cached_tmap_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                     uint32_t bi, uint32_t bo, bool swizzle = true);

constexpr int W_BQ = 128;                       // rows per query tile
constexpr int W_BKV = 128;
constexpr int W_D = 128;
constexpr int W_THREADS = 384;   // warps 0..3 control (TMA, MMA, two idle), 4..7 softmax of tile 0, 8..11 softmax of tile 1
constexpr int W_TILE_BYTES = 128 * 128 * 2;     // 32 KB: two 64-column blocks of 16 KB
constexpr int W_STAGES = 2;
constexpr int W_STG_BYTES = 32 * 128;           // output staging tile of a softmax warp: 32 rows x 64 bf16 columns, 128B-swizzled
constexpr int W_SMEM = 2 * W_TILE_BYTES + 2 * W_STAGES * W_TILE_BYTES + 8 * W_STG_BYTES + 256;
constexpr int W_TMEM_COLS = 512;

struct FlashWsParams {
  __nv_bfloat16* out;
  float* lse;
  long long ldo;
  int B, S, Hq, Hkv;           // S: query rows per sequence
  int Skv, qoff;               // key/value rows per sequence; query row i sits at position i + qoff (= Skv - S)
  int causal;
  float scale_log2;
  int* err;
  // paged keys / values: the K and V tensor maps then cover the KV cache as token rows
  // [num_blocks * 2 * 16, Hkv * 128] (K rows of block b start at row b * 32, V rows at b * 32 + 16) with a box of
  // 16 rows, and every 128-key tile is fetched page by page through this sequence's row of the block table
  const int* block_table;      // [B, max_blocks] physical block ids, or null for contiguous K / V
  int max_blocks, num_blocks;
};

constexpr int W_PAGE = 16;                      // tokens per KV-cache block on the paged path
constexpr int W_PAGE_BYTES = W_PAGE * 128;      // one page of one 64-column half: 16 rows of 128 bytes

// One unit of work: 256 query rows of one (batch, head).
struct FlashWsItem {
  int q0, h, hkv, b;
  int n_t[2];                  // key tiles that each query tile needs (0: the tile lies past the sequence)
  int n_kv;
};

// Item i. Items are numbered by work, the longest query pairs first; false for i < 0.
__device__ __forceinline__ bool flash_ws_item(const FlashWsParams& p, int i, FlashWsItem& it) {
  if (i < 0) return false;
  const int n_pairs = (p.S + 2 * W_BQ - 1) / (2 * W_BQ);
  const int hb = p.Hq * p.B;
  const int pair = p.causal ? n_pairs - 1 - i / hb : i / hb;
  it.h = (i % hb) % p.Hq;
  it.b = (i % hb) / p.Hq;
  it.hkv = it.h / (p.Hq / p.Hkv);
  it.q0 = pair * 2 * W_BQ;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int qs = it.q0 + t * W_BQ;
    int n = (p.Skv + W_BKV - 1) / W_BKV;
    if (p.causal) n = min(n, (qs + p.qoff + W_BQ + W_BKV - 1) / W_BKV);
    it.n_t[t] = qs < p.S ? n : 0;
  }
  it.n_kv = max(it.n_t[0], it.n_t[1]);
  return true;
}

__global__ void __launch_bounds__(W_THREADS, 1)
flash_fwd_ws_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FlashWsParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase;                                  // 2 tiles
  const uint32_t sK = sQ + 2 * W_TILE_BYTES;                  // W_STAGES tiles
  const uint32_t sV = sK + W_STAGES * W_TILE_BYTES;           // W_STAGES tiles
  const uint32_t sStg = sV + W_STAGES * W_TILE_BYTES;         // one staging tile per softmax warp
  const uint32_t bars = sStg + 8 * W_STG_BYTES;
  // barriers: q_full[2] k_full[2] v_full[2] k_empty[2] v_empty[2] s_full[2] p_full[2] pv_done[2] p_half[2] q_empty[2]
  auto q_full = [&](int t) { return bars + 8u * t; };
  auto k_full = [&](int s) { return bars + 8u * (2 + s); };
  auto v_full = [&](int s) { return bars + 8u * (4 + s); };
  auto k_empty = [&](int s) { return bars + 8u * (6 + s); };
  auto v_empty = [&](int s) { return bars + 8u * (8 + s); };
  auto s_full = [&](int t) { return bars + 8u * (10 + t); };
  auto p_full = [&](int t) { return bars + 8u * (12 + t); };
  auto pv_done = [&](int t) { return bars + 8u * (14 + t); };
  auto p_half = [&](int t) { return bars + 8u * (16 + t); };
  auto q_empty = [&](int t) { return bars + 8u * (18 + t); };
  // the next item: answers of the launch control, two of them in turn
  auto next_full = [&](int s) { return bars + 8u * (20 + s); };
  auto next_empty = [&](int s) { return bars + 8u * (22 + s); };
  auto answer = [&](int s) { return bars + 8u * 26 + 16u * s; };
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + (bars - sbase) + 8 * 24);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if ((sbase & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.err, 0, ERR_BAD_INDEX);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_full(i), 1);
      mbar_init(k_full(i), 1);
      mbar_init(v_full(i), 1);
      mbar_init(k_empty(i), 1);
      mbar_init(v_empty(i), 1);
      mbar_init(s_full(i), 1);
      mbar_init(p_full(i), 128);
      mbar_init(p_half(i), 128);
      mbar_init(pv_done(i), 1);
      mbar_init(q_empty(i), 1);
      mbar_init(next_full(i), 1);
      mbar_init(next_empty(i), 9);              // the MMA issuer and eight softmax warps have read the answer
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_ptr_smem), W_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  pdl_trigger();
  pdl_wait();
  auto tS = [&](int t) { return tmem_base + 128u * t; };
  auto tO = [&](int t) { return tmem_base + 256u + 128u * t; };
  FlashWsItem w;

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  if (warp == 0) {
    // ===================== TMA producer =====================
    if (elect_one()) {
      int kt = 0;                               // key tiles fetched so far: ring position and phase
      int n_q[2] = {0, 0};                      // query tiles fetched so far
      bool ok = true;
      const int seq_pages = (p.Skv + W_PAGE - 1) / W_PAGE;
      int item = blockIdx.x;
      for (int k = 0; ok && flash_ws_item(p, item, w); ++k) {
        const long long row_base = (long long)w.b * p.S;
        const long long kv_row_base = (long long)w.b * p.Skv;
        const int* bt = p.block_table ? p.block_table + (long long)w.b * p.max_blocks : nullptr;
        for (int j = 0; j < w.n_kv && ok; ++j, ++kt) {
          const int s = kt & 1;
          const uint32_t ph = (kt >> 1) & 1;
          const int krow = (int)(kv_row_base + j * W_BKV);
          int blk[W_BKV / W_PAGE];
          if (bt) {
            // the eight table entries of this tile first (independent loads); pages past the end of the sequence
            // repeat its first page: their keys are masked, they only have to be readable
#pragma unroll
            for (int g = 0; g < W_BKV / W_PAGE; ++g) {
              const int pg = j * (W_BKV / W_PAGE) + g;
              blk[g] = bt[pg < seq_pages && pg < p.max_blocks ? pg : 0];
            }
#pragma unroll
            for (int g = 0; g < W_BKV / W_PAGE; ++g)
              if (blk[g] < 0 || blk[g] >= p.num_blocks) { atomicCAS(p.err, 0, ERR_BAD_INDEX); blk[g] = 0; }
          }
          if (!mbar_wait(k_empty(s), ph ^ 1u, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
          mbar_expect_tx(k_full(s), W_TILE_BYTES);
          if (bt) {
#pragma unroll
            for (int g = 0; g < W_BKV / W_PAGE; ++g) {
              const uint32_t dst = sK + s * W_TILE_BYTES + g * W_PAGE_BYTES;
              tma_load_2d(dst, &tmK, w.hkv * W_D, blk[g] * 2 * W_PAGE, k_full(s));
              tma_load_2d(dst + W_TILE_BYTES / 2, &tmK, w.hkv * W_D + 64, blk[g] * 2 * W_PAGE, k_full(s));
            }
          } else {
            tma_load_2d(sK + s * W_TILE_BYTES, &tmK, w.hkv * W_D, krow, k_full(s));
            tma_load_2d(sK + s * W_TILE_BYTES + W_TILE_BYTES / 2, &tmK, w.hkv * W_D + 64, krow, k_full(s));
          }
          if (j == 0) {
            // this item's queries, each as soon as the previous item's last S of that tile has read its buffer
            for (int t = 0; t < 2; ++t) {
              if (w.n_t[t] == 0) continue;
              if (!mbar_wait(q_empty(t), (n_q[t] & 1) ^ 1u, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
              ++n_q[t];
              mbar_expect_tx(q_full(t), W_TILE_BYTES);
              const int qrow = (int)(row_base + w.q0 + t * W_BQ);
              tma_load_2d(sQ + t * W_TILE_BYTES, &tmQ, w.h * W_D, qrow, q_full(t));
              tma_load_2d(sQ + t * W_TILE_BYTES + W_TILE_BYTES / 2, &tmQ, w.h * W_D + 64, qrow, q_full(t));
            }
            if (!ok) break;
          }
          if (j == max(0, w.n_kv - 2)) {
            // the next item, asked for as late as its answer (a microsecond) allows: an item that a CTA has taken waits for it
            if (!mbar_wait(next_empty(k & 1), ((k >> 1) & 1) ^ 1u, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
            mbar_expect_tx(next_full(k & 1), 16);
            clc_try_cancel(answer(k & 1), next_full(k & 1));
          }
          if (!mbar_wait(v_empty(s), ph ^ 1u, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
          mbar_expect_tx(v_full(s), W_TILE_BYTES);
          if (bt) {
#pragma unroll
            for (int g = 0; g < W_BKV / W_PAGE; ++g) {
              const uint32_t dst = sV + s * W_TILE_BYTES + g * W_PAGE_BYTES;
              tma_load_2d(dst, &tmV, w.hkv * W_D, (blk[g] * 2 + 1) * W_PAGE, v_full(s));
              tma_load_2d(dst + W_TILE_BYTES / 2, &tmV, w.hkv * W_D + 64, (blk[g] * 2 + 1) * W_PAGE, v_full(s));
            }
          } else {
            tma_load_2d(sV + s * W_TILE_BYTES, &tmV, w.hkv * W_D, krow, v_full(s));
            tma_load_2d(sV + s * W_TILE_BYTES + W_TILE_BYTES / 2, &tmV, w.hkv * W_D + 64, krow, v_full(s));
          }
        }
        if (!ok || !mbar_wait(next_full(k & 1), (k >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) break;
        item = clc_answer(answer(k & 1));
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    if (elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(128, W_BKV, 0, 0);
      const uint32_t idesc_pv = make_idesc_bf16(128, W_D, 0, 1);
      auto issue_s = [&](int t, int stage) {
        uint64_t q = make_smem_desc_sw128(sQ + t * W_TILE_BYTES, 16, 1024), kd = make_smem_desc_sw128(sK + stage * W_TILE_BYTES, 16, 1024);
        asm volatile("" : "+l"(q), "+l"(kd));      // sixteen descriptors kept in registers ahead of time would spill
#pragma unroll
        for (int kk = 0; kk < W_D / 16; ++kk) {
          const uint32_t off = ((kk >> 2) * (W_TILE_BYTES / 2) + (kk & 3) * 32) >> 4;     // a descriptor counts 16 bytes
          umma_bf16_ss(tS(t), q + off, kd + off, idesc_s, kk != 0);
        }
        umma_commit(s_full(t));
      };
      auto issue_pv = [&](int t, int stage, int half, bool first) {   // 64 keys: P's half, as soon as the softmax has published it
        uint64_t v = make_smem_desc_sw128(sV + stage * W_TILE_BYTES, W_TILE_BYTES / 2, 1024);
        asm volatile("" : "+l"(v));
#pragma unroll
        for (int i = 0; i < W_BKV / 32; ++i) {
          const int kk = half * (W_BKV / 32) + i;
          umma_bf16_ts(tO(t), tS(t) + 8u * kk, v + (kk * 2048 >> 4), idesc_pv, !first || kk != 0);
        }
      };
      int kt = 0;                               // ring position of this item's first key tile
      uint32_t p_phase[2] = {0, 0};             // per query tile: parity of its key tiles multiplied so far
      uint32_t q_phase[2] = {0, 0};
      bool ok = true;
      bool have = flash_ws_item(p, blockIdx.x, w);
      // S_t(0) of an item, its K and Q waited for; the last S of a tile gives its Q buffer back
      auto first_s = [&](const FlashWsItem& x, int ring, int t) -> bool {
        if (x.n_t[t] == 0) return true;
        if (!mbar_wait(k_full(ring & 1), (ring >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) return false;
        if (!mbar_wait(q_full(t), q_phase[t], abort_flag, p.err, ERR_WAIT_ATTN)) return false;
        q_phase[t] ^= 1;
        tc_fence_after_sync();
        issue_s(t, ring & 1);
        if (x.n_t[t] == 1) umma_commit(q_empty(t));
        return true;
      };
      if (have) {
        ok = first_s(w, 0, 0) && first_s(w, 0, 1);
        if (ok) umma_commit(k_empty(0));          // K_0 consumed by both tiles' S
      }
      for (int k = 0; ok && have; ++k) {
        FlashWsItem nx;
        bool more = false;
        for (int j = 0; j < w.n_kv && ok; ++j) {
          const int r = kt + j, s = r & 1;
          const uint32_t ph = (r >> 1) & 1;
          const bool last = j + 1 == w.n_kv;
          bool k_next_ready = false;
          // called with each tile's number, so that no state of a tile is addressed by a variable
          auto tile = [&](const int t) -> bool {
            if (j < w.n_t[t]) {
              if (!mbar_wait(v_full(s), ph, abort_flag, p.err, ERR_WAIT_ATTN)) return false;
              if (!mbar_wait(p_half(t), p_phase[t], abort_flag, p.err, ERR_WAIT_ATTN)) return false;
              tc_fence_after_sync();
              issue_pv(t, s, 0, j == 0);
              if (!mbar_wait(p_full(t), p_phase[t], abort_flag, p.err, ERR_WAIT_ATTN)) return false;
              tc_fence_after_sync();
              issue_pv(t, s, 1, j == 0);
              umma_commit(pv_done(t));
              p_phase[t] ^= 1;
            }
            if (j + 1 < w.n_t[t]) {
              if (!k_next_ready) {
                if (!mbar_wait(k_full((r + 1) & 1), ((r + 1) >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) return false;
                k_next_ready = true;
                tc_fence_after_sync();
              }
              issue_s(t, (r + 1) & 1);
              if (j + 2 == w.n_t[t]) umma_commit(q_empty(t));
            } else if (last) {
              // the next item's first S goes in behind this item's last products: its softmax warps find it ready when
              // they have written their rows
              if (t == 0) {
                if (!mbar_wait(next_full(k & 1), (k >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) return false;
                more = flash_ws_item(p, clc_answer(answer(k & 1)), nx);
                mbar_arrive(next_empty(k & 1));
              }
              if (more && !first_s(nx, r + 1, t)) return false;
            }
            return true;
          };
          ok = tile(0) && tile(1);
          if (!ok) break;
          umma_commit(v_empty(s));                               // V_j consumed by both tiles' PV
          if (!last || more) umma_commit(k_empty((r + 1) & 1));  // K_{j+1}, or the next item's K_0, consumed by both tiles' S
        }
        kt += w.n_kv;
        w = nx;
        have = more;
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // ===================== softmax warpgroups =====================
    const int t = (warp - 4) >> 2;            // query tile of this warpgroup
    const int q = warp & 3;                   // TMEM lane quarter this warp may access
    const int r = q * 32 + lane;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    int n = 0;                                // key tiles seen so far (phase of every barrier of this tile)
    bool ok = true;
    int item = blockIdx.x;
    auto next_item = [&](int k) {
      if (!mbar_wait_warp(next_full(k & 1), (k >> 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) return false;
      item = clc_answer(answer(k & 1));
      __syncwarp();
      if (lane == 0) mbar_arrive(next_empty(k & 1));
      return true;
    };
    for (int k = 0; ok && flash_ws_item(p, item, w); ok = ok && next_item(k), ++k) {
    const int qi = w.q0 + t * W_BQ + r;
    const int n_mine = w.n_t[t];
    float m_used = 0.f, l = 0.f;
    for (int j = 0; j < n_mine; ++j, ++n) {
      if (!mbar_wait_warp(s_full(t), n & 1, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
      tc_fence_after_sync();
      const int k0 = j * W_BKV;
      uint32_t sv[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(tS(t) + 32 * c + lane_off, *reinterpret_cast<uint32_t(*)[32]>(&sv[32 * c]));
      tmem_wait_ld();
      // last visible column of this row, and of the warp's first row: blocks of 32 columns that the whole warp sees are
      // left alone, so that a diagonal tile costs as little as it can
      const int lim = (p.causal ? min(p.Skv - 1, qi + p.qoff) : p.Skv - 1) - k0;
      const int lim_warp = (p.causal ? min(p.Skv - 1, w.q0 + t * W_BQ + q * 32 + p.qoff) : p.Skv - 1) - k0;
      if (lim_warp < W_BKV - 1) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (32 * c + 31 > lim_warp) {
#pragma unroll
            for (int i = 32 * c; i < 32 * c + 32; ++i)
              if (i > lim) sv[i] = __float_as_uint(-INFINITY);
          }
        }
      }
      // The tile's maximum first (three-input maxima), so that P can be published in halves: the tensor pipe multiplies
      // keys 0..63 while the exponentials of keys 64..127 run. P and O are expressed against m_used, which only moves when
      // some row's maximum has grown by more than 2^8; exponents stay below 2^8.
      float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
      for (int i = 0; i < 128; i += 8) {
        m0 = fmax3(m0, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
        m1 = fmax3(m1, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
        m2 = fmax3(m2, __uint_as_float(sv[i + 4]), __uint_as_float(sv[i + 5]));
        m3 = fmax3(m3, __uint_as_float(sv[i + 6]), __uint_as_float(sv[i + 7]));
      }
      const float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * p.scale_log2;     // scale > 0: max commutes with the scaling
      if (j == 0) m_used = mx == -INFINITY ? 0.f : mx;
      const bool grow = j > 0 && mx > m_used + 8.f;
      if (__any_sync(0xffffffffu, grow)) {
        if (!mbar_wait_warp(pv_done(t), (n - 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
        tc_fence_after_sync();
        const float f = grow ? exp2f(m_used - mx) : 1.f;
#pragma unroll
        for (int c = 0; c < W_D / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(tO(t) + c * 32 + lane_off, o);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          tmem_st_32x32b_x32(tO(t) + c * 32 + lane_off, o);
        }
        l *= f;
        if (grow) m_used = mx;
      }
      // two elements per fused multiply-add and addition: the pipes beside the exponentials' one issue half as often
      const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2), nm2 = pack_f32x2(-m_used, -m_used);
      uint64_t rs = 0ull;                      // sums of the even and of the odd keys (four sums are no faster)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint64_t e = fma_f32x2(pack_f32x2(__uint_as_float(sv[64 * hh + 2 * i]), __uint_as_float(sv[64 * hh + 2 * i + 1])), c2, nm2);
          float e0, e1;
          unpack_f32x2(e, e0, e1);
          e0 = exp2f(e0);
          e1 = exp2f(e1);
          rs = add_f32x2(rs, pack_f32x2(e0, e1));
          pk[i] = pack_bf16x2(e0, e1);
        }
        tmem_st_32x32b_x32(tS(t) + 32 * hh + lane_off, pk);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(hh == 0 ? p_half(t) : p_full(t));
      }
      float rs0, rs1;
      unpack_f32x2(rs, rs0, rs1);
      l += rs0 + rs1;
    }
    if (!ok || n_mine == 0) continue;
    if (!mbar_wait_warp(pv_done(t), (n - 1) & 1, abort_flag, p.err, ERR_WAIT_ATTN)) { ok = false; break; }
    // O_t is free for the next item's first product once this warpgroup publishes that item's first P, which every
    // thread does after its reads here
    tc_fence_after_sync();
    const float inv = l > 0.f ? 1.f / l : 0.f;
    const bool row_ok = qi < p.S;
    const long long row = (long long)w.b * p.S + qi;
    if (w.q0 + t * W_BQ + q * 32 + 32 <= p.S) {
      // the warp's 32 rows go through its own swizzled staging tile, 64 columns at a time
      const uint32_t stg = sStg + (uint32_t)(warp - 4) * W_STG_BYTES;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t o[64];
        tmem_ld_32x32b_x32(tO(t) + hh * 64 + lane_off, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));
        tmem_ld_32x32b_x32(tO(t) + hh * 64 + 32 + lane_off, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
        tmem_wait_ld();
        if (lane == 0) tma_store_wait_read<0>();   // the store before has left the staging tile
        __syncwarp();
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const uint32_t addr = stg + lane * 128 + (((uint32_t)v ^ (uint32_t)(lane & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                       "r"(pack_bf16x2(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv)),
                       "r"(pack_bf16x2(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv)),
                       "r"(pack_bf16x2(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv)),
                       "r"(pack_bf16x2(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv))
                       : "memory");
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmO, stg, w.h * W_D + hh * 64, (int)((long long)w.b * p.S + w.q0 + t * W_BQ + q * 32));
          tma_store_commit();
        }
      }
    } else {
      // the sequence's last rows: the ones behind them belong to the next sequence
      __nv_bfloat16* orow = p.out + row * p.ldo + (long long)w.h * W_D;
#pragma unroll
      for (int c = 0; c < W_D / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(tO(t) + c * 32 + lane_off, o);
        tmem_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 x;
            x.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv);
            x.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv);
            x.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv);
            x.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv);
            reinterpret_cast<uint4*>(orow + 32 * c)[v] = x;
          }
        }
      }
    }
    if (row_ok && p.lse) p.lse[((long long)w.b * p.Hq + w.h) * p.S + qi] = (m_used + log2f(l)) * 0.6931471805599453f;
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
    tmem_dealloc(tmem_base, W_TMEM_COLS);
  }
}

static int launch_flash_ws(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FlashWsParams& p, cudaStream_t st) {
  CUtensorMap to;
  if (int rc = cached_tmap_bf16(&to, p.out, (uint64_t)p.Hq * W_D, (uint64_t)p.B * p.S, (uint64_t)p.ldo, 64, 32)) return rc;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    MLF_CHECK_CUDA(cudaFuncSetAttribute(flash_fwd_ws_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, W_SMEM));
    attr_set[dev & 63] = true;
  }
  // a CTA per item, of which one per SM starts (shared memory and tensor memory hold no second one) and takes over the others
  const long long items = (long long)((p.S + 2 * W_BQ - 1) / (2 * W_BQ)) * p.Hq * p.B;
  MLF_REQUIRE(items < (1LL << 31), "flash_fwd: too many rows");
  MLF_CHECK_CUDA(launch_pdl(flash_fwd_ws_kernel, dim3((unsigned)items), dim3(W_THREADS), W_SMEM, st, tq, tk, tv, to, p));
  count_launch();
  return 0;
}

}  // namespace mlf

using namespace mlf;

// Queries [B * Sq rows] against keys / values [B * Skv rows], Skv >= Sq: query row i of a sequence sits at
// position i + (Skv - Sq), i.e. the queries are the LAST Sq positions (a prompt chunk attending to its cached
// prefix plus itself). Skv == Sq is plain self-attention.
MLF_API int mlf_flash_fwd_prefix(const void* q, const void* k, const void* v, void* out, float* lse, int B, int Sq, int Skv, int Hq,
                                 int Hkv, long long ldq, long long ldk, long long ldv, long long ldo, float scale, int causal,
                                 uint64_t stream) {
  const int S = Sq;
  MLF_REQUIRE(B > 0 && S > 0 && Skv >= Sq && Hq > 0 && Hkv > 0 && Hq % Hkv == 0, "flash_fwd: bad shape");
  MLF_REQUIRE(scale > 0.f, "flash_fwd: softmax scale must be positive");
  MLF_REQUIRE(ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0, "flash_fwd: out must be 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap tq, tk, tv;
  int rc;
  const uint64_t rows = (uint64_t)B * S, kv_rows = (uint64_t)B * Skv;
  if ((rc = cached_tmap_bf16(&tq, q, (uint64_t)Hq * W_D, rows, ldq, 64, W_BQ))) return rc;
  if ((rc = cached_tmap_bf16(&tk, k, (uint64_t)Hkv * W_D, kv_rows, ldk, 64, W_BKV))) return rc;
  if ((rc = cached_tmap_bf16(&tv, v, (uint64_t)Hkv * W_D, kv_rows, ldv, 64, W_BKV))) return rc;
  FlashWsParams p;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.ldo = ldo;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.Skv = Skv; p.qoff = Skv - Sq;
  p.causal = causal;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.err = device_status_word();
  p.block_table = nullptr;
  p.max_blocks = p.num_blocks = 0;
  MLF_REQUIRE(p.err != nullptr, "no device status word");
  return launch_flash_ws(tq, tk, tv, p, st);
}

// Prefill attention whose keys and values are read straight out of the paged KV cache: queries [B * Sq rows] are the
// LAST Sq positions of sequences of Skv cached tokens each (the chunk's own K / V are already in the cache), and
// every 128-key tile is fetched page by page through the sequence's row of the block table by the kernel's TMA
// producer - no gather of the cached prefix into a contiguous buffer. cache: [num_blocks, 2, 16, Hkv, 128] bf16;
// block_table: int32 [B, max_blocks]. The reference walks the block table per token
// (src/MLFramework/Inference/PagedAttention/Layers/PagedAttentionLayer.cs:332-389, Phases/PrefillOrchestrator.cs:62-78).
MLF_API int mlf_flash_fwd_paged(const void* q, const void* cache, const int* block_table, void* out, float* lse, int B, int Sq, int Skv,
                                int Hq, int Hkv, long long ldq, long long ldo, int num_blocks, int block_size, int max_blocks, float scale,
                                int causal, uint64_t stream) {
  MLF_REQUIRE(B > 0 && Sq > 0 && Skv >= Sq && Hq > 0 && Hkv > 0 && Hq % Hkv == 0, "flash_fwd_paged: bad shape");
  MLF_REQUIRE(block_size == W_PAGE, "flash_fwd_paged: the block size must be %d tokens", W_PAGE);
  MLF_REQUIRE(block_table != nullptr && num_blocks > 0 && (long long)max_blocks * W_PAGE >= Skv,
              "flash_fwd_paged: %d table entries cannot describe %d tokens", max_blocks, Skv);
  MLF_REQUIRE(scale > 0.f, "flash_fwd_paged: softmax scale must be positive");
  MLF_REQUIRE(ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0, "flash_fwd_paged: out must be 16-byte aligned");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap tq, tkv;
  int rc;
  if ((rc = cached_tmap_bf16(&tq, q, (uint64_t)Hq * W_D, (uint64_t)B * Sq, ldq, 64, W_BQ))) return rc;
  if ((rc = cached_tmap_bf16(&tkv, cache, (uint64_t)Hkv * W_D, (uint64_t)num_blocks * 2 * W_PAGE, (uint64_t)Hkv * W_D, 64, W_PAGE))) return rc;
  FlashWsParams p;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.ldo = ldo;
  p.B = B; p.S = Sq; p.Hq = Hq; p.Hkv = Hkv;
  p.Skv = Skv; p.qoff = Skv - Sq;
  p.causal = causal;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.err = device_status_word();
  p.block_table = block_table;
  p.max_blocks = max_blocks;
  p.num_blocks = num_blocks;
  MLF_REQUIRE(p.err != nullptr, "no device status word");
  return launch_flash_ws(tq, tkv, tkv, p, st);
}

// Same arguments as mlf_flash_fwd.
MLF_API int mlf_flash_fwd_ws(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int Hq,
                             int Hkv, long long ldq, long long ldk, long long ldv, long long ldo, float scale, int causal,
                             uint64_t stream) {
  return mlf_flash_fwd_prefix(q, k, v, out, lse, B, S, S, Hq, Hkv, ldq, ldk, ldv, ldo, scale, causal, stream);
}
