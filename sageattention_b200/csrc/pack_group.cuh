// One group of the K-packing mode (15 tokens -> group mean + 15 residuals), shared by the packing kernel (pack.cu) and the
// K quantisation + delta_s kernel, which packs on the way in (delta_s.cu).  See pack.cu for what a group becomes.
#pragma once

#include "common.cuh"

namespace sage3 {

constexpr int kGroup = 15;

// magnitude of an E2M1 code: 0, 0.5, 1, 1.5, 2, 3, 4, 6 (sign in bit 3)
__device__ __forceinline__ float e2m1_value(const uint32_t code) {
  const uint32_t mag = code & 7u;
  const float lvl = mag < 2 ? 0.5f * mag : (mag < 4 ? 1.0f + 0.5f * (mag - 2) : (mag < 6 ? 2.0f + (mag - 4) : (mag == 6 ? 4.0f : 6.0f)));
  return (code & 8u) ? -lvl : lvl;
}

// By a whole warp: lane l holds channels l*C ... l*C + C-1 of the group's (smoothed) rows in x.  m receives the slot of the
// group mean, row(j, r) is called with the residual of token j; returns lambda of slot `lane` (0 in the mean slot and
// beyond the group).
template <int C, class Row>
__device__ __forceinline__ float pack_group(const float (&x)[kGroup][C], const int lane, float (&m)[C], Row&& row) {
  constexpr int kLanesPerBlock = 16 / C;            // lanes that share one 16-channel scale block
  // ---- group mean -> bf16 -> block-scaled FP4 round trip along the head dimension (16-channel blocks)
  float amax = 0.f;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < kGroup; ++j) sum += x[j][c];
    m[c] = __bfloat162float(__float2bfloat16(__fdiv_rn(sum, (float)kGroup)));
    amax = fmaxf(amax, fabsf(m[c]));
  }
#pragma unroll
  for (int o = 1; o < kLanesPerBlock; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = e4m3_to_f32(f32_to_e4m3(__fdiv_rn(amax, 6.0f)));
  const float inv = scale == 0.f ? 0.f : __frcp_rn(scale);
  {
    float sc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < C; ++c) sc[c] = __fmul_rn(m[c], inv);
    // E2M1 round-to-nearest-even with saturation, then back to fp32 through the 8 magnitudes
    uint32_t codes = f32x8_to_e2m1x8(sc[0], sc[1], sc[2], sc[3], 0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      m[c] = __bfloat162float(__float2bfloat16(__fmul_rn(e2m1_value((codes >> (4 * c)) & 0xFu), scale)));
    }
  }
  // ---- direction = m / |m|^2
  float nsq = 0.f;
#pragma unroll
  for (int c = 0; c < C; ++c) nsq = fmaf(m[c], m[c], nsq);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nsq += __shfl_xor_sync(0xffffffffu, nsq, o);
  float dir[C];
#pragma unroll
  for (int c = 0; c < C; ++c) dir[c] = nsq > 0.f ? __fdiv_rn(m[c], nsq) : 0.f;
  // ---- lambda and residual of every token
  float my_lam = 0.f;                               // lane s keeps lambda of slot s
#pragma unroll
  for (int j = 0; j < kGroup; ++j) {
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) dot = fmaf(x[j][c], dir[c], dot);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (lane == j + 1) my_lam = dot;
    float r[C];
#pragma unroll
    for (int c = 0; c < C; ++c) r[c] = __fsub_rn(x[j][c], __fmul_rn(dot, m[c]));
    row(j, r);
  }
  return my_lam;
}

// "Split first" V layout, one channel: v is the group's first value and amax the group's largest magnitude.  v becomes what
// the V^T quantiser will make of it (one scale over the group's 16 slots, slot 0 still zero; emulation arithmetic of
// api.py:77-110: true division, round to nearest even); returns the remainder, which goes to slot 0.
__device__ __forceinline__ float split_first_value(float& v, const float amax) {
  const float scale = e4m3_to_f32(f32_to_e4m3(__fdiv_rn(amax, 6.0f)));
  const float inv = scale == 0.f ? 0.f : __frcp_rn(scale);
  const uint32_t code = f32x8_to_e2m1x8(__fmul_rn(v, inv), 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f) & 0xFu;
  const float hi = __bfloat162float(__float2bfloat16(__fmul_rn(e2m1_value(code), scale)));
  const float lo = __fsub_rn(v, hi);
  v = hi;
  return lo;
}

}  // namespace sage3
