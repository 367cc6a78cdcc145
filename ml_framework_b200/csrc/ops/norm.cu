// LayerNorm and RMSNorm, forward and backward, bf16 activations with fp32 statistics.
//
// Forward: one warp owns one row at a time and keeps it in registers as packed bf16 (NV 16-byte
// vectors per lane), so x is read from HBM exactly once per pass; from D = 2048 on a CTA owns whole rows, unless rows are
// many and D is no 2048 or 4096. Backward: every thread owns fixed columns of the rows that pass by and keeps its share of the
// gamma / beta gradients in registers, one partial per CTA; a second tiny kernel sums the partials.
//
// The reference has no norm kernels (its AMP rules only name layernorm as an fp32 op,
// src/MLFramework/Amp/DefaultAmpRules.cs:48-110); these are required by the GPT and Llama
// model families.
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "../mlf_api.h"

namespace mlf {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  return u;
}

// CTAs past the first `norm_ctas` of a forward launch clear a buffer for a later kernel (the output that the next
// product adds its partial tiles into): a clearing launch of its own would stand in the chain of kernels.
__device__ __forceinline__ void zero_role(uint4* z, long long n, int norm_ctas) {
  const long long stride = (long long)(gridDim.x - norm_ctas) * blockDim.x;
  for (long long i = (long long)(blockIdx.x - norm_ctas) * blockDim.x + threadIdx.x; i < n; i += stride) z[i] = make_uint4(0u, 0u, 0u, 0u);
}

constexpr int NORM_CTAS = 2;                 // CTAs of norm_fwd_cta_kernel that an SM holds

// D = NV * 256. rms != 0 selects RMSNorm (no mean subtraction, no beta). gamma and beta are loaded GV vectors at a time
// ahead of the stores that use them: behind a store, which may alias as far as the compiler knows, every vector waited for its own load
// (8192 rows of 8192: 67 us, 55 us with GV = 4; with GV = NV the registers cost warps: 8192 x 1024 7.8 us, 6.8 us with 2).
template <int NV>
__global__ void __launch_bounds__(256, NV <= 3 ? 4 : NV <= 6 ? 3 : NV <= 12 ? 2 : 1)   // NV = 12 unasked: 130 registers, half the warps
norm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gamma, const __nv_bfloat16* beta, __nv_bfloat16* y,
                float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, float eps, int rms, int norm_ctas,
                uint4* zero, long long n_zero) {
  constexpr int D = NV * 256;
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= norm_ctas) {
    zero_role(zero, n_zero, norm_ctas);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int warps_per_cta = blockDim.x >> 5;
  for (int row = blockIdx.x * warps_per_cta + (threadIdx.x >> 5); row < rows; row += norm_ctas * warps_per_cta) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (long long)row * D);
    const uint4* gr = reinterpret_cast<const uint4*>(gamma);
    const uint4* br = reinterpret_cast<const uint4*>(beta);
    constexpr int GV = NV <= 3 ? NV : NV <= 12 ? 2 : 4;
    uint4 xv[NV], gv[GV], bv[GV];
#pragma unroll
    for (int i = 0; i < NV; ++i) xv[i] = xr[i * 32 + lane];
    auto load_affine = [&](int i0) {
#pragma unroll
      for (int i = 0; i < GV; ++i) gv[i] = gr[(i0 + i) * 32 + lane];
      if (beta) {
#pragma unroll
        for (int i = 0; i < GV; ++i) bv[i] = br[(i0 + i) * 32 + lane];
      }
    };
    load_affine(0);
    float s = 0.f;
    if (!rms) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        float f[8];
        unpack8(xv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += f[j];
      }
      s = warp_sum(s) * (1.f / D);
    }
    const float mean = rms ? 0.f : s;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float f[8];
      unpack8(xv[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = f[j] - mean;
        ss += d * d;
      }
    }
    const float rstd = rsqrtf(warp_sum(ss) * (1.f / D) + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
    uint4* yr = reinterpret_cast<uint4*>(y + (long long)row * D);
#pragma unroll
    for (int i0 = 0; i0 < NV; i0 += GV) {
      if (i0 > 0) load_affine(i0);
#pragma unroll
      for (int i = 0; i < GV; ++i) {
        float f[8], g[8], b[8];
        unpack8(xv[i0 + i], f);
        unpack8(gv[i], g);
        if (beta) unpack8(bv[i], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = (f[j] - mean) * rstd * g[j] + (beta ? b[j] : 0.f);
        yr[(i0 + i) * 32 + lane] = pack8(f);
      }
    }
  }
}

// Forward for D = NVT * 2048 with whole-CTA rows: 256 threads own 8 * NVT fixed columns each (gamma / beta in
// registers, packed), R rows are loaded together and the next R while these are summed and written, and the row sums meet
// across the eight warps through shared memory. Few rows (a decode step: 64 x 4096) then still occupy one CTA per row
// group instead of one warp per row. Bound by memory; two CTAs per SM hold both sets of rows without spills, and the grid
// has no more of them (four per SM, of which three were resident, ran a nearly empty second round): RMS norm of 4096 x 4096
// 18.4 -> 14.3 us, 8192 x 4096 37 -> 29 us, layer norm of 8192 x 2048 23.4 -> 18.4 us (three CTAs: 18.4, 35, 24.6).
template <int NVT, int R>
__global__ void __launch_bounds__(256, NORM_CTAS)
norm_fwd_cta_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gamma,
                    const __nv_bfloat16* beta, __nv_bfloat16* y,
                    float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, float eps, int rms, int norm_ctas,
                    uint4* zero, long long n_zero) {
  constexpr int D = NVT * 2048;
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= norm_ctas) {
    zero_role(zero, n_zero, norm_ctas);
    return;
  }
  __shared__ float red[2][2][8][R];          // [iteration parity][sum | centred squares][warp][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint4 xv[R][NVT], gv[NVT], bv[NVT];
  auto load_rows = [&](int row0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const long long base = (long long)(row0 + r < rows ? row0 + r : row0) * (D / 8);
#pragma unroll
      for (int v = 0; v < NVT; ++v) xv[r][v] = reinterpret_cast<const uint4*>(x)[base + v * 256 + tid];
    }
  };
  load_rows(blockIdx.x * R);
#pragma unroll
  for (int v = 0; v < NVT; ++v) {
    gv[v] = reinterpret_cast<const uint4*>(gamma)[v * 256 + tid];
    bv[v] = beta ? reinterpret_cast<const uint4*>(beta)[v * 256 + tid] : make_uint4(0u, 0u, 0u, 0u);
  }
  const float inv_d = 1.f / D;
  int par = 0;
  for (int row0 = blockIdx.x * R; row0 < rows; row0 += norm_ctas * R, par ^= 1) {
    uint4 cur[R][NVT];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int v = 0; v < NVT; ++v) cur[r][v] = xv[r][v];
    if (row0 + norm_ctas * R < rows) load_rows(row0 + norm_ctas * R);
    float mean[R];
    if (!rms) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float sm = 0.f;
#pragma unroll
        for (int v = 0; v < NVT; ++v) {
          float f[8];
          unpack8(cur[r][v], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) sm += f[j];
        }
        sm = warp_sum(sm);
        if (lane == 0) red[par][0][warp][r] = sm;
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red[par][0][w][r];
        mean[r] = t * inv_d;
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) mean[r] = 0.f;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float ss = 0.f;
#pragma unroll
      for (int v = 0; v < NVT; ++v) {
        float f[8];
        unpack8(cur[r][v], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float d = f[j] - mean[r];
          ss = fmaf(d, d, ss);
        }
      }
      ss = warp_sum(ss);
      if (lane == 0) red[par][1][warp][r] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (row0 + r >= rows) break;
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) t += red[par][1][w][r];
      const float rstd = rsqrtf(t * inv_d + eps);
      if (tid == 0) {
        if (mean_out) mean_out[row0 + r] = mean[r];
        if (rstd_out) rstd_out[row0 + r] = rstd;
      }
#pragma unroll
      for (int v = 0; v < NVT; ++v) {
        float f[8], g[8], bt[8];
        unpack8(cur[r][v], f);
        unpack8(gv[v], g);
        unpack8(bv[v], bt);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = fmaf((f[j] - mean[r]) * rstd, g[j], bt[j]);
        reinterpret_cast<uint4*>(y)[(long long)(row0 + r) * (D / 8) + v * 256 + tid] = pack8(f);
      }
    }
  }
}

// Forward of not too many rows for the wide D that are no multiple of 2048 (3072, 5120, 6144) and for 8192: one thread per
// 16-byte vector of a row, D / 8 threads per CTA, R rows loaded together. One warp per row keeps D / 256 vectors per lane
// and walks them three times, which no other warp of the SM covers when there are few rows: 24 x 5120 took 8.5 us (RMS)
// that way, 2.2 us here. With many rows the other warps do, and the two CTAs per SM that fit here meet twice per row:
// 8192 x 5120 34 us that way, 55 us here; norm_row_line() says up to where this kernel is used.
template <int R>
__global__ void __launch_bounds__(1024)
norm_fwd_row_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gamma, const __nv_bfloat16* beta,
                    __nv_bfloat16* y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int D, float eps, int rms,
                    int norm_ctas, uint4* zero, long long n_zero) {
  pdl_trigger();
  pdl_wait();
  if ((int)blockIdx.x >= norm_ctas) {
    zero_role(zero, n_zero, norm_ctas);
    return;
  }
  __shared__ float red[2][2][32][R];         // [iteration parity][sum | centred squares][warp][row]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, n_warps = blockDim.x >> 5;
  float g[8], bt[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  unpack8(reinterpret_cast<const uint4*>(gamma)[tid], g);
  if (beta) unpack8(reinterpret_cast<const uint4*>(beta)[tid], bt);
  const float inv_d = 1.f / D;
  int par = 0;
  for (int row0 = blockIdx.x * R; row0 < rows; row0 += norm_ctas * R, par ^= 1) {
    float f[R][8], mean[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      unpack8(reinterpret_cast<const uint4*>(x)[(long long)(row0 + r < rows ? row0 + r : row0) * (D / 8) + tid], f[r]);
#pragma unroll
    for (int r = 0; r < R; ++r) mean[r] = 0.f;
    if (!rms) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float sm = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) sm += f[r][j];
        sm = warp_sum(sm);
        if (lane == 0) red[par][0][warp][r] = sm;
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r) mean[r] = warp_sum(lane < n_warps ? red[par][0][lane][r] : 0.f) * inv_d;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = f[r][j] - mean[r];
        ss = fmaf(d, d, ss);
      }
      ss = warp_sum(ss);
      if (lane == 0) red[par][1][warp][r] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (row0 + r >= rows) break;
      const float rstd = rsqrtf(warp_sum(lane < n_warps ? red[par][1][lane][r] : 0.f) * inv_d + eps);
      if (tid == 0) {
        if (mean_out) mean_out[row0 + r] = mean[r];
        if (rstd_out) rstd_out[row0 + r] = rstd;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) f[r][j] = fmaf((f[r][j] - mean[r]) * rstd, g[j], bt[j]);
      reinterpret_cast<uint4*>(y)[(long long)(row0 + r) * (D / 8) + tid] = pack8(f[r]);
    }
  }
}

// f = (f - mean) * rstd. x * rstd - mean * rstd would be one operation an element but rounds mean * rstd: rows of 1000 +- 4 come
// out up to 7.6e-6 off, 1.2e-7 here. Two elements an instruction, so that it costs the same (us, warm, that form / this one / this
// one element by element: 8192 x 1536 24.1 / 23.9 / 24.8, 8192 x 2048 29.2 / 29.3 / 30.5, 8192 x 3072 41.7 / 41.5 / 42.9,
// and with a thread per vector 8192 x 6144 155 / 159 / 166, 8192 x 8192 190 / 192 / 202).
template <bool RMS>
__device__ __forceinline__ void normalise8(float (&f)[8], float mean, float rstd) {
  const uint64_t m2 = pack_f32x2(-mean, -mean), r2 = pack_f32x2(rstd, rstd);
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const uint64_t x = pack_f32x2(f[j], f[j + 1]);
    unpack_f32x2(mul_f32x2(RMS ? x : add_f32x2(x, m2), r2), f[j], f[j + 1]);
  }
}

// Backward. D = 256, 512, 1024, 2048 and 4096: 2048 columns' worth of rows side by side (GROUPS rows of D = 2048 / GROUPS, or a
// row of D = NVT * 2048), a CTA of 256 threads; other widths: a row to a CTA of as many threads as it has vectors, or half as many
// above 4096. Every thread has a fixed set of 8 * NVT columns, so that gamma and the gamma / beta gradient partials sit in registers.
// R rows of x, dy and the skip gradient are summed and written while the next R are in flight. The two row sums meet across the
// warps of a row through a double-buffered shared array: one barrier per R rows.
// us, before (one warp per row; for 2048 and 4096 no rows in flight ahead) -> now: 8192 x 4096 RMS 69 -> 56 (floor 41), 2331 x 1024
// 21.5 -> 15.4, 2331 x 3072 73 -> 21.5; one launch behind the other 8192 x 5120 layer / RMS norm 497 / 344 -> 121 / 62, 8192 x 8192
// 1136 / 992 -> 154 / 78 (a thread per vector, whose 64 registers spill: 190 / 83).
template <int NVT, int R, int GROUPS, bool RMS, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1)
norm_bwd_cta_kernel(const __nv_bfloat16* x, const __nv_bfloat16* dy,
                    const __nv_bfloat16* gamma, const float* mean_in,
                    const float* rstd_in, __nv_bfloat16* dx,
                    float* partials /* [grid, 2, D] */, int rows,
                    const __nv_bfloat16* dx_add /* optional: added to dx */) {
  static_assert(NVT == 1 || GROUPS == 1, "a row is either shared by the CTA or a group's own");
  // threads and warps of a row: THREADS != 256 stands for any number of up to THREADS threads, all of them on one row
  const int TPR = THREADS == 256 ? 256 / GROUPS : (int)blockDim.x, WPR = TPR / 32, D = NVT * 8 * TPR;
  __shared__ float red[2][THREADS / 32][2 * R];
  __shared__ float fold[GROUPS > 1 ? 2 * 2048 / GROUPS : 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int grp = tid / TPR, col = tid % TPR, warp0 = grp * WPR;
  pdl_trigger();
  pdl_wait();
  uint4 gv[NVT];
  float dg[NVT][8], db[RMS ? 1 : NVT][8];
#pragma unroll
  for (int v = 0; v < NVT; ++v) {
    gv[v] = reinterpret_cast<const uint4*>(gamma)[v * TPR + col];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dg[v][j] = 0.f;
      if (!RMS) db[RMS ? 0 : v][j] = 0.f;
    }
  }
  const float inv_d = 1.f / (float)D;
  uint4 nx[R][NVT], nd[R][NVT], ne[R][NVT];
  float nmean[R], nrstd[R];
  const int step = gridDim.x * GROUPS * R;
  auto load = [&](int row0) {                  // rows past the end: the last row, with a gradient of zero
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool ok = row0 + r < rows;
      const int row = ok ? row0 + r : rows - 1;
      const long long base = (long long)row * (D / 8);
#pragma unroll
      for (int v = 0; v < NVT; ++v) {
        nx[r][v] = reinterpret_cast<const uint4*>(x)[base + v * TPR + col];
        nd[r][v] = ok ? reinterpret_cast<const uint4*>(dy)[base + v * TPR + col] : make_uint4(0, 0, 0, 0);
        ne[r][v] = dx_add ? reinterpret_cast<const uint4*>(dx_add)[base + v * TPR + col] : make_uint4(0, 0, 0, 0);
      }
      nmean[r] = RMS ? 0.f : mean_in[row];
      nrstd[r] = rstd_in[row];
    }
  };
  int row0 = (blockIdx.x * GROUPS + grp) * R, buf = 0;
  load(row0);
  // every group makes the CTA's number of rounds: they meet at its barrier
  for (int first = blockIdx.x * GROUPS * R; first < rows; first += step, row0 += step, buf ^= 1) {
    uint4 xv[R][NVT], dv[R][NVT], ev[R][NVT];
    float mean[R], rstd[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int v = 0; v < NVT; ++v) {
        xv[r][v] = nx[r][v];
        dv[r][v] = nd[r][v];
        ev[r][v] = ne[r][v];
      }
      mean[r] = nmean[r];
      rstd[r] = nrstd[r];
    }
    if (first + step < rows) load(row0 + step);
    float c[2 * R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float c1 = 0.f, c2 = 0.f;
#pragma unroll
      for (int v = 0; v < NVT; ++v) {
        float f[8], d[8], g[8];
        unpack8(xv[r][v], f);
        normalise8<RMS>(f, mean[r], rstd[r]);
        unpack8(dv[r][v], d);
        unpack8(gv[v], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float dxh = d[j] * g[j];
          c1 += dxh;
          c2 = fmaf(dxh, f[j], c2);
          dg[v][j] = fmaf(d[j], f[j], dg[v][j]);
          if (!RMS) db[RMS ? 0 : v][j] += d[j];
        }
      }
      c[2 * r] = RMS ? 0.f : warp_sum(c1);
      c[2 * r + 1] = warp_sum(c2);
    }
    if (lane < 2 * R) {
      float mine = c[0];
#pragma unroll
      for (int k = 1; k < 2 * R; ++k) mine = lane == k ? c[k] : mine;
      red[buf][warp][lane] = mine;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2 * R; ++k) {
      float t = 0.f;
      if (THREADS == 256) {
#pragma unroll
        for (int w = 0; w < 8 / GROUPS; ++w) t += red[buf][warp0 + w][k];
      } else {
        t = warp_sum(lane < WPR ? red[buf][lane][k] : 0.f);
      }
      c[k] = t * inv_d;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (row0 + r >= rows) break;
      const float c1 = RMS ? 0.f : c[2 * r], c2 = c[2 * r + 1];
#pragma unroll
      for (int v = 0; v < NVT; ++v) {
        float f[8], d[8], e[8], g[8], o[8];
        unpack8(xv[r][v], f);
        normalise8<RMS>(f, mean[r], rstd[r]);
        unpack8(dv[r][v], d);
        unpack8(ev[r][v], e);
        unpack8(gv[v], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j] = fmaf(rstd[r], fmaf(d[j], g[j], -c1) - f[j] * c2, e[j]);
        }
        reinterpret_cast<uint4*>(dx)[(long long)(row0 + r) * (D / 8) + v * TPR + col] = pack8(o);
      }
    }
  }
  // the groups' partial sums of a column, one group after the other
  if (GROUPS > 1) {
#pragma unroll 1
    for (int k = 1; k < GROUPS; ++k) {
      __syncthreads();
      if (grp == k) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          fold[j * TPR + col] = dg[0][j];
          if (!RMS) fold[D + j * TPR + col] = db[0][j];
        }
      }
      __syncthreads();
      if (grp == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dg[0][j] += fold[j * TPR + col];
          if (!RMS) db[0][j] += fold[D + j * TPR + col];
        }
      }
    }
    if (grp != 0) return;
  }
  float* po = partials + (long long)blockIdx.x * 2 * D;
#pragma unroll
  for (int v = 0; v < NVT; ++v) {
    float4* pg = reinterpret_cast<float4*>(po + (v * TPR + col) * 8);
    pg[0] = make_float4(dg[v][0], dg[v][1], dg[v][2], dg[v][3]);
    pg[1] = make_float4(dg[v][4], dg[v][5], dg[v][6], dg[v][7]);
    if (!RMS) {
      float4* pb = reinterpret_cast<float4*>(po + D + (v * TPR + col) * 8);
      pb[0] = make_float4(db[RMS ? 0 : v][0], db[RMS ? 0 : v][1], db[RMS ? 0 : v][2], db[RMS ? 0 : v][3]);
      pb[1] = make_float4(db[RMS ? 0 : v][4], db[RMS ? 0 : v][5], db[RMS ? 0 : v][6], db[RMS ? 0 : v][7]);
    }
  }
}

// dgamma[c] = sum_g partials[g][0][c]; dbeta likewise. 32 columns x 32 partial-lanes per CTA (a few hundred
// partial rows: the kernel is pure load latency, so the rows are spread over 32 warps).
constexpr int NF_WARPS = 32;
__global__ void __launch_bounds__(NF_WARPS * 32)
norm_bwd_finalize_kernel(const float* partials, int nparts, int D, void* dgamma, void* dbeta,
                         int out_fp32, int accumulate_gamma, int accumulate_beta) {
  __shared__ float sg[NF_WARPS][33], sb[NF_WARPS][33];
  pdl_trigger();
  pdl_wait();
  const int cl = threadIdx.x & 31, pl = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cl;
  float g = 0.f, b = 0.f;
  if (c < D) {
#pragma unroll 4
    for (int p = pl; p < nparts; p += NF_WARPS) {
      g += partials[(long long)p * 2 * D + c];
      if (dbeta) b += partials[(long long)p * 2 * D + D + c];
    }
  }
  sg[pl][cl] = g;
  sb[pl][cl] = b;
  __syncthreads();
  if (pl != 0 || c >= D) return;
#pragma unroll
  for (int k = 1; k < NF_WARPS; ++k) { g += sg[k][cl]; b += sb[k][cl]; }
  if (out_fp32) {
    float* dgp = static_cast<float*>(dgamma);
    dgp[c] = g + (accumulate_gamma ? dgp[c] : 0.f);
    if (dbeta) {
      float* dbp = static_cast<float*>(dbeta);
      dbp[c] = b + (accumulate_beta ? dbp[c] : 0.f);
    }
  } else {
    __nv_bfloat16* dgp = static_cast<__nv_bfloat16*>(dgamma);
    dgp[c] = __float2bfloat16(g + (accumulate_gamma ? __bfloat162float(dgp[c]) : 0.f));
    if (dbeta) {
      __nv_bfloat16* dbp = static_cast<__nv_bfloat16*>(dbeta);
      dbp[c] = __float2bfloat16(b + (accumulate_beta ? __bfloat162float(dbp[c]) : 0.f));
    }
  }
}

// Rows from which one warp per row is as fast as one thread per vector, in us there / here (RMS norm; layer norm, which meets
// once more here and walks once more there, crosses at the same rows): 1024 x 3072 4.8 / 4.6, 1536 x 3072 5.6 / 6.4,
// 600 x 5120 6.2 / 5.6, 1024 x 5120 6.2 / 8.4, 600 x 6144 7.3 / 6.6, 1024 x 6144 7.3 / 9.0, 1536 x 8192 16.1 / 14.3,
// 2048 x 8192 17.8 / 17.2, 2304 x 8192 19.1 / 19.5, 8192 x 8192 55 / 71.
static int norm_row_line(int D) { return D == 8192 ? 2304 : D == 3072 ? 1184 : 800; }

template <int NV>
static int launch_fwd(const void* x, const void* g, const void* b, void* y, float* mean, float* rstd, int rows,
                      float eps, int rms, uint4* zero, long long n_zero, int zero_ctas, cudaStream_t st) {
  const int grid = min((rows + 7) / 8, sm_count() * 8);
  MLF_CHECK_CUDA(launch_pdl(norm_fwd_kernel<NV>, dim3(grid + zero_ctas), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(x),
                            static_cast<const __nv_bfloat16*>(g), static_cast<const __nv_bfloat16*>(b), static_cast<__nv_bfloat16*>(y), mean,
                            rstd, rows, eps, rms, grid, zero, n_zero));
  count_launch();
  return 0;
}

}  // namespace mlf

using namespace mlf;

// y = norm(x) * gamma (+ beta). D must be a multiple of 256 from {256..1024, 1536, 2048, 3072,
// 4096, 5120, 6144, 8192}. mean/rstd (fp32 [rows]) may be null for inference. `zero` (optional, 16-byte aligned,
// zero_bytes a multiple of 16) is cleared by additional CTAs of the same launch.
MLF_API int mlf_norm_fwd_zero(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                              int rows, int D, float eps, int rms, void* zero, long long zero_bytes, uint64_t stream) {
  MLF_REQUIRE(D % 256 == 0, "norm: D=%d must be a multiple of 256", D);
  MLF_REQUIRE(zero_bytes >= 0 && zero_bytes % 16 == 0 && (reinterpret_cast<uintptr_t>(zero) & 15) == 0, "norm: the buffer to clear must be 16-byte aligned");
  uint4* zp = static_cast<uint4*>(zero);
  const long long nz = zero != nullptr ? zero_bytes / 16 : 0;
  // 32 KB per CTA: eight 16-byte stores per thread
  const int zc = (int)(nz == 0 ? 0 : (nz + 2047) / 2048 < sm_count() ? (nz + 2047) / 2048 : sm_count());
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (D == 2048 || D == 4096) {
    const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
    const __nv_bfloat16* gp = static_cast<const __nv_bfloat16*>(gamma);
    const __nv_bfloat16* bp = static_cast<const __nv_bfloat16*>(beta);
    __nv_bfloat16* yp = static_cast<__nv_bfloat16*>(y);
    const int cap = NORM_CTAS * sm_count();
    if (D == 2048) {
      const int r = rows >= 4 * cap ? 4 : (rows >= 2 * cap ? 2 : 1);      // few rows: one row per CTA, more CTAs
      const int grid = min((rows + r - 1) / r, cap);
      const auto kernel = r == 4 ? norm_fwd_cta_kernel<1, 4> : r == 2 ? norm_fwd_cta_kernel<1, 2> : norm_fwd_cta_kernel<1, 1>;
      MLF_CHECK_CUDA(launch_pdl(kernel, dim3(grid + zc), dim3(256), 0, st, xp, gp, bp, yp, mean, rstd, rows, eps, rms, grid, zp, nz));
    } else {
      const int r = rows >= 2 * cap ? 2 : 1;
      const int grid = min((rows + r - 1) / r, cap);
      const auto kernel = r == 2 ? norm_fwd_cta_kernel<2, 2> : norm_fwd_cta_kernel<2, 1>;
      MLF_CHECK_CUDA(launch_pdl(kernel, dim3(grid + zc), dim3(256), 0, st, xp, gp, bp, yp, mean, rstd, rows, eps, rms, grid, zp, nz));
    }
    count_launch();
    return 0;
  }
  if ((D == 3072 || D == 5120 || D == 6144 || D == 8192) && rows < norm_row_line(D)) {
    // two rows per CTA once every SM has two CTAs with work
    const int cap = 2 * sm_count();
    const int r = rows >= 2 * cap ? 2 : 1;
    const int grid = min((rows + r - 1) / r, cap);
    const auto kernel = r == 2 ? norm_fwd_row_kernel<2> : norm_fwd_row_kernel<1>;
    MLF_CHECK_CUDA(launch_pdl(kernel, dim3(grid + zc), dim3(D / 8), 0, st, static_cast<const __nv_bfloat16*>(x),
                              static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta),
                              static_cast<__nv_bfloat16*>(y), mean, rstd, rows, D, eps, rms, grid, zp, nz));
    count_launch();
    return 0;
  }
#define CALL(NV) launch_fwd<NV>(x, gamma, beta, y, mean, rstd, rows, eps, rms, zp, nz, zc, st)
  switch (D / 256) {
    case 1: return CALL(1); case 2: return CALL(2); case 3: return CALL(3); case 4: return CALL(4); case 6: return CALL(6);
    case 12: return CALL(12); case 20: return CALL(20); case 24: return CALL(24); case 32: return CALL(32);
    default: break;
  }
#undef CALL
  set_error("norm: unsupported D=%d", D);
  return -2;
}

MLF_API int mlf_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                         int rows, int D, float eps, int rms, uint64_t stream) {
  return mlf_norm_fwd_zero(x, gamma, beta, y, mean, rstd, rows, D, eps, rms, nullptr, 0, stream);
}

// Rows that a CTA of the backward takes at a time, and how many CTAs there are: as many as an SM holds.
static int norm_bwd_rows(int D) { return D == 4096 || D > 4096 ? 1 : D == 256 || D == 512 || D == 1024 ? 2 * (2048 / D) : 2; }
static int norm_bwd_grid(int rows, int D) {
  const int r = norm_bwd_rows(D), per_sm = D == 768 ? 5 : D == 1536 ? 2 : D == 3072 || D > 4096 ? 1 : 2;
  return min((rows + r - 1) / r, per_sm * sm_count());
}

// Number of fp32 elements the caller must provide as `partials` scratch for mlf_norm_bwd.
MLF_API long long mlf_norm_bwd_scratch_elems(int rows, int D) {
  return (long long)norm_bwd_grid(rows, D) * 2 * D;
}

// dx_add (optional, bf16 [rows, D]) is added to dx: the gradient arriving over a skip connection that
// branched off the normalised tensor's input, so that the sum needs no pass of its own. dgamma and dbeta are of one type (fp32 if
// grads_fp32, else bf16); each is written or added to by a switch of its own.
MLF_API int mlf_norm_bwd_add(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd,
                             void* dx, void* dgamma, void* dbeta, float* partials, int rows, int D, int rms,
                             int grads_fp32, int accumulate_gamma, int accumulate_beta, const void* dx_add, uint64_t stream) {
  MLF_REQUIRE(D % 256 == 0, "norm: D=%d must be a multiple of 256", D);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = norm_bwd_grid(rows, D);
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* dyp = static_cast<const __nv_bfloat16*>(dy);
  const __nv_bfloat16* gp = static_cast<const __nv_bfloat16*>(gamma);
  __nv_bfloat16* dxp = static_cast<__nv_bfloat16*>(dx);
  const __nv_bfloat16* addp = static_cast<const __nv_bfloat16*>(dx_add);
#define LAUNCH(NVT, R, GROUPS, THREADS, BLOCK)                                                                             \
  {                                                                                                                        \
    const auto kernel = rms ? norm_bwd_cta_kernel<NVT, R, GROUPS, true, THREADS> : norm_bwd_cta_kernel<NVT, R, GROUPS, false, THREADS>; \
    MLF_CHECK_CUDA(launch_pdl(kernel, dim3(grid), dim3(BLOCK), 0, st, xp, dyp, gp, mean, rstd, dxp, partials, rows, addp));   \
  } break;
  switch (D) {
    case 256: LAUNCH(1, 2, 8, 256, 256)
    case 512: LAUNCH(1, 2, 4, 256, 256)
    case 1024: LAUNCH(1, 2, 2, 256, 256)
    case 2048: LAUNCH(1, 2, 1, 256, 256)
    case 4096: LAUNCH(2, 1, 1, 256, 256)
    case 768: case 1536: case 3072: LAUNCH(1, 2, 1, 384, D / 8)
    case 5120: case 6144: case 8192: LAUNCH(2, 1, 1, 512, D / 16)
    default: MLF_REQUIRE(false, "norm: unsupported D=%d", D);
  }
#undef LAUNCH
  count_launch();
  MLF_CHECK_CUDA(launch_pdl(norm_bwd_finalize_kernel, dim3((D + 31) / 32), dim3(NF_WARPS * 32), 0, st, (const float*)partials, grid, D, dgamma,
                            rms ? (void*)nullptr : dbeta, grads_fp32, accumulate_gamma, accumulate_beta));
  count_launch();
  return 0;
}

MLF_API int mlf_norm_bwd(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd,
                         void* dx, void* dgamma, void* dbeta, float* partials, int rows, int D, int rms,
                         int grads_fp32, int accumulate, uint64_t stream) {
  return mlf_norm_bwd_add(x, dy, gamma, mean, rstd, dx, dgamma, dbeta, partials, rows, D, rms, grads_fp32, accumulate, accumulate, nullptr,
                          stream);
}
