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
  for (int c = 0; c < C; c += 2) {
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kGroup; ++j) sum = fadd2(sum, make_float2(x[j][c], x[j][c + 1]));
    m[c] = __bfloat162float(__float2bfloat16(__fdiv_rn(sum.x, (float)kGroup)));
    m[c + 1] = __bfloat162float(__float2bfloat16(__fdiv_rn(sum.y, (float)kGroup)));
    amax = fmaxf(fmaxf(amax, fabsf(m[c])), fabsf(m[c + 1]));
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
  // ---- lambda of every token: 16 sums over the warp at once, each step of the exchange leaving a lane half of them - token
  // lane / 2 in the end.  The pairs of lanes that are added are those of an exchange of every sum on its own, and so are the bits.
  // (On its own, 75 shuffles instead of 31, K pass of B4 H32 N2048 D128 65.9 us; now 64.2.)
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    v[j] = 0.f;
    if (j < kGroup)
#pragma unroll
      for (int c = 0; c < C; ++c) v[j] = fmaf(x[j][c], dir[c], v[j]);
  }
#pragma unroll
  for (int step = 0; step < 4; ++step) {
    const int o = 16 >> step, n = 8 >> step;
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float give = upper ? v[i] : v[n + i], own = upper ? v[n + i] : v[i];
      v[i] = own + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  const float lam = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
  // ---- residuals
#pragma unroll
  for (int j = 0; j < kGroup; ++j) {
    const float dot = __shfl_sync(0xffffffffu, lam, 2 * j);
    float r[C];
#pragma unroll
    // the product rounded by itself: a packed multiplication and addition (mul.rn.f32x2, add.rn.f32x2) came out as one
    // fused operation, and residuals and codes with it
    for (int c = 0; c < C; ++c) r[c] = __fsub_rn(x[j][c], __fmul_rn(dot, m[c]));
    row(j, r);
  }
  const float my_lam = __shfl_sync(0xffffffffu, lam, (2 * lane - 2) & 31);   // lane s: lambda of slot s
  return lane >= 1 && lane <= kGroup ? my_lam : 0.f;
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
