// Rotary embedding (rotate-half): the angle and the rotation of a pair (d, d + head_dim / 2), for every kernel that rotates
// heads. The roundings are spelled out, so that what one kernel rotates equals bit for bit what another one does.
#pragma once

namespace mlf {

// (cosine, sine) of a pair at position `pos`: pos * theta^-x, where x = 2 d / head_dim.
__device__ __forceinline__ float2 rope_cos_sin(float pos, float log_theta, float x) {
  const float inv_freq = __expf(__fmul_rn(-log_theta, x));
  float2 cs;
  sincosf(__fmul_rn(pos, inv_freq), &cs.y, &cs.x);
  return cs;
}
// x of pair d: the exact quotient, a product where the head dimension is a power of two (the same value, without the
// division that made 2048 tokens of 32 + 2 x 8 heads 16.5 us instead of 12.0).
template <int HEAD_DIM>
__device__ __forceinline__ float rope_exponent(int d) {
  static_assert((HEAD_DIM & (HEAD_DIM - 1)) == 0, "a power of two");
  return __fmul_rn((float)d, 2.f / HEAD_DIM);
}
__device__ __forceinline__ float rope_exponent(int d, int head_dim) { return __fdiv_rn(2.f * d, (float)head_dim); }

__device__ __forceinline__ void rope_rotate(float& a, float& b, float2 cs) {
  const float x = a, y = b;
  a = __fmaf_rn(x, cs.x, -__fmul_rn(y, cs.y));
  b = __fmaf_rn(x, cs.y, __fmul_rn(y, cs.x));
}

}  // namespace mlf
