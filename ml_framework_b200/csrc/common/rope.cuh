// Rotary embedding (rotate-half): the angle and the rotation of a pair (d, d + head_dim / 2), for every kernel that rotates
// heads. The roundings are spelled out, so that what one kernel rotates equals bit for bit what another one does.
#pragma once

namespace mlf {

// (cosine, sine) of pair d of a head at position `pos`: pos * theta^(-2 d / head_dim).
__device__ __forceinline__ float2 rope_cos_sin(float pos, float log_theta, int d, int head_dim) {
  const float inv_freq = __expf(__fmul_rn(-log_theta, __fdiv_rn(2.f * d, (float)head_dim)));
  float2 cs;
  sincosf(__fmul_rn(pos, inv_freq), &cs.y, &cs.x);
  return cs;
}

__device__ __forceinline__ void rope_rotate(float& a, float& b, float2 cs) {
  const float x = a, y = b;
  a = __fmaf_rn(x, cs.x, -__fmul_rn(y, cs.y));
  b = __fmaf_rn(x, cs.y, __fmul_rn(y, cs.x));
}

}  // namespace mlf
