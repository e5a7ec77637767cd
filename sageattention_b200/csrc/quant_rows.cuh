// Row-wise NVFP4 quantisation of one 128-token tile held in registers, shared by the fused quantisation kernel
// (quant.cu, Q and K roles) and the K quantisation + delta_s kernel (delta_s.cu).
#pragma once

#include "common.cuh"

namespace sage3 {

constexpr int kTile = 128;
constexpr int kThreads = 256;

// The 8 channels of this thread (chunk threadIdx.x % (D/8)) of a head's K mean: from `km` where it is given, else from
// the partial sums, by the whole CTA; also written to km_out if that is not null.  `stage`: shared memory for kMaxChunks
// partial rows - they are fetched all at once, so that the CTA waits for memory once and not once per few rows (the K
// kernel at B1 H40 N32760: 328 us, 356 with a chain of loads).
constexpr int kMaxChunks = 64;             // at most so many partial rows per head (pick_chunk_tokens, quant.cu)
template <int D>
__device__ __forceinline__ void k_mean(const __nv_bfloat16* __restrict__ km, const float* __restrict__ partial, const int nchunks,
                                       const float divisor, const int64_t bh, float* stage, __nv_bfloat16* km_out,
                                       float (&mean)[8]) {
  const int t = threadIdx.x, c = t % (D / 8);
  if (km != nullptr) {
    const uint4 m = *reinterpret_cast<const uint4*>(km + bh * D + c * 8);
    mean[0] = bf16_lo(m.x); mean[1] = bf16_hi(m.x); mean[2] = bf16_lo(m.y); mean[3] = bf16_hi(m.y);
    mean[4] = bf16_lo(m.z); mean[5] = bf16_hi(m.z); mean[6] = bf16_lo(m.w); mean[7] = bf16_hi(m.w);
    return;
  }
  constexpr int V = kMaxChunks * D / 4 / kThreads;
  const int nv = nchunks * D / 4;
  float4 x[V];
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (i * kThreads + t < nv) x[i] = __ldcg(reinterpret_cast<const float4*>(partial) + i * kThreads + t);
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (i * kThreads + t < nv) reinterpret_cast<float4*>(stage)[i * kThreads + t] = x[i];
  __syncthreads();
  float s = 0.f;
  if (t < D)
    for (int i = 0; i < nchunks; ++i) s += stage[i * D + t];
  __syncthreads();
  if (t < D) {
    const __nv_bfloat16 m = __float2bfloat16_rn(s / divisor);
    stage[t] = __bfloat162float(m);
    if (km_out != nullptr) km_out[bh * D + t] = m;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) mean[i] = stage[c * 8 + i];
}

// Row-wise quantisation of one 128-token tile held in registers (Q and K roles).
// Thread t owns 8 consecutive channels (chunk c) of rows rl, rl+RPP, ... ; w[p] = 4 packed bf16x2.
// ------------------------------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void quant_rows_store(const uint4 (&w)[kTile / (kThreads / (D / 8))],
                                                 uint8_t* __restrict__ codes_tile, uint8_t* __restrict__ sf_tile,
                                                 uint8_t* sf_smem) {
  constexpr int CH = D / 8, RPP = kThreads / CH, NP = kTile / RPP;
  const int t = threadIdx.x, c = t % CH, rl = t / CH;
  // scale of block c / 2 in row p * RPP + rl: sf_atom_offset with what depends on p taken out as a constant (rl < RPP <= 32; written as
  // such, the addresses were 15 % of the instructions)
  uint8_t* const sf_row = sf_smem + (c >> 3) * 512 + ((c >> 1) & 3) + rl * 16;
  uint8_t* const out = codes_tile + rl * (D / 2) + c * 4;
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const uint32_t m2 = abs2(habsmax2(habsmax2(w[p].x, w[p].y), habsmax2(w[p].z, w[p].w)));
    float amax = fmaxf(bf16_lo(m2), bf16_hi(m2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));       // 16-element block = 2 threads
    uint32_t sfb; float inv;
    block_scale(amax, sfb, inv);
    const float2 inv2 = make_float2(inv, inv);
    const float2 f0 = mul2_ftz(bf16x2_to_f32(w[p].x), inv2), f1 = mul2_ftz(bf16x2_to_f32(w[p].y), inv2);
    const float2 f2 = mul2_ftz(bf16x2_to_f32(w[p].z), inv2), f3 = mul2_ftz(bf16x2_to_f32(w[p].w), inv2);
    const uint32_t code = f32x8_to_e2m1x8(f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y);
    *reinterpret_cast<uint32_t*>(out + p * (RPP * D / 2)) = code;
    static_assert(RPP == 16 || RPP == 32, "rows of a pass");
    if ((c & 1) == 0) sf_row[RPP == 16 ? (p & 1) * 256 + (p >> 1) * 4 : p * 4] = (uint8_t)sfb;
  }
  __syncthreads();
  constexpr int SFV = (D / 64) * 512 / 16;                           // 16-byte vectors of scales
  if (t < SFV) reinterpret_cast<uint4*>(sf_tile)[t] = reinterpret_cast<const uint4*>(sf_smem)[t];
}


}  // namespace sage3
