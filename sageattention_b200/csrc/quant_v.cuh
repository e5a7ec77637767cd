// NVFP4 quantisation of V along tokens, shared by the fused quantisation kernel (quant.cu) and the scores kernel of few query rows per
// head (decode.cu): 4 channels of one 16-token block in registers.
#pragma once

#include "common.cuh"
#include "pack_group.cuh"

namespace sage3 {

// x[i] = channels d ... d + 3 of token i of block `blk`; codes: the tile's [channel][64 bytes]; sf: its two atoms.
// split_first (K-packing mode): token 0 takes what FP4 leaves of token 1.
__device__ __forceinline__ void quant_v_block(const uint2 (&x)[16], const int d, const int blk, const bool split_first,
                                              uint8_t* __restrict__ codes, uint8_t* __restrict__ sf) {
  // largest magnitudes of the 4 channels, two at a time (bf16 comparisons are exact)
  uint32_t m01 = habsmax2(x[0].x, x[1].x), m23 = habsmax2(x[0].y, x[1].y);
#pragma unroll
  for (int i = 2; i < 16; ++i) { m01 = habsmax2(m01, x[i].x); m23 = habsmax2(m23, x[i].y); }
  m01 = abs2(m01); m23 = abs2(m23);
  // four channels from a multiple of 4 on: rows of an atom 16 bytes apart
  uint8_t* const sf_row = sf + (blk >> 2) * 512 + sf_atom_offset(d, blk & 3);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float f[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t wv = (j < 2) ? x[i].x : x[i].y;
      f[i] = (j & 1) ? bf16_hi(wv) : bf16_lo(wv);
    }
    const uint32_t mv = j < 2 ? m01 : m23;
    float amax = (j & 1) ? bf16_hi(mv) : bf16_lo(mv);
    if (split_first) {
      f[0] = __bfloat162float(__float2bfloat16_rn(split_first_value(f[1], amax)));
      amax = fmaxf(fabsf(f[0]), fabsf(f[1]));
#pragma unroll
      for (int i = 2; i < 16; ++i) amax = fmaxf(amax, fabsf(f[i]));
    }
    uint32_t sfb; float inv;
    block_scale(amax, sfb, inv);
    const float2 inv2 = make_float2(inv, inv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 y = mul2_ftz(make_float2(f[2 * i], f[2 * i + 1]), inv2);
      f[2 * i] = y.x; f[2 * i + 1] = y.y;
    }
    *reinterpret_cast<uint2*>(codes + (d + j) * 64 + blk * 8) =
        make_uint2(f32x8_to_e2m1x8(f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]),
                   f32x8_to_e2m1x8(f[8], f[9], f[10], f[11], f[12], f[13], f[14], f[15]));
    sf_row[j * 16] = (uint8_t)sfb;
  }
}

}  // namespace sage3
