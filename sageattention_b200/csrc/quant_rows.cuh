// Row-wise NVFP4 quantisation of one 128-token tile held in registers, shared by the fused quantisation kernel
// (quant.cu, Q and K roles) and the K quantisation + delta_s kernel (delta_s.cu).
#pragma once

#include "common.cuh"

namespace sage3 {

constexpr int kTile = 128;
constexpr int kThreads = 256;

// Row-wise quantisation of one 128-token tile held in registers (Q and K roles).  Thread t owns the 16 channels 16 block(t) ... of
// rows row(t), + kStep, ...: whole quantisation blocks, so that scales need no exchange and are worked out once.  (With 8 channels a
// thread, two threads to a block: B1 H40 N32760 228 -> 219 us, K pass 321 -> 292.)
// Which lane has which: its bits kBlockBits are the block, the others the row.  D=128: so that 8 lanes' 16-byte stores of the K pass
// (delta_s.cu), 4128 bytes from block to block and 16 from row to row, meet different banks.
// kHalves (Q): bit 4 is the half of the tile (rows 0 ... 63 or 64 ... 127), which the order of the block sums asks for (tile_sums in
// quant.cu); else a warp has rows next to one another (K pass of B1 H40 N32760 280 us, 299 with kHalves).
// ------------------------------------------------------------------------------------------------
template <int D, bool kHalves>
struct RowTile {
  static constexpr int kPerRow = D / 16, kPasses = kTile * kPerRow / kThreads, kStep = kTile / kPasses / (kHalves ? 2 : 1);
  static constexpr int kBlockBits = D == 128 ? 11 : 3;     // bits of the lane that are the block
  static __device__ __forceinline__ int block(const int t) { return D == 128 ? (t & 3) | ((t >> 1) & 4) : t & 3; }
  static __device__ __forceinline__ int row(const int t) {
    if (!kHalves) return D == 128 ? ((t >> 2) & 1) | ((t >> 4) << 1) : t >> 2;
    return (D == 128 ? ((t >> 2) & 1) | ((t >> 5) << 1) : ((t >> 2) & 3) | ((t >> 5) << 2)) + ((t >> 4) & 1) * (kTile / 2);
  }
  static_assert(kStep == kThreads / (kHalves ? 2 : 1) / kPerRow, "every row once");
};
__device__ __forceinline__ void bf16x16_to_f32(const __nv_bfloat16* p, float (&x)[16]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint4 m = reinterpret_cast<const uint4*>(p)[i];
    x[8 * i] = bf16_lo(m.x); x[8 * i + 1] = bf16_hi(m.x); x[8 * i + 2] = bf16_lo(m.y); x[8 * i + 3] = bf16_hi(m.y);
    x[8 * i + 4] = bf16_lo(m.z); x[8 * i + 5] = bf16_hi(m.z); x[8 * i + 6] = bf16_lo(m.w); x[8 * i + 7] = bf16_hi(m.w);
  }
}

// The 16 channels of this thread (16 block(threadIdx.x) ...) of a head's K mean: from `km` where it is given, else from
// the partial sums, by the whole CTA; also written to km_out if that is not null.  `stage`: shared memory for kMaxChunks
// partial rows - they are fetched all at once, so that the CTA waits for memory once and not once per few rows (the K
// kernel of that time at B1 H40 N32760: 328 us, 356 with a chain of loads; by now 281).
constexpr int kMaxChunks = 64;             // at most so many partial rows per head (pick_chunk_tokens, quant.cu)
template <int D>
__device__ __forceinline__ void k_mean(const __nv_bfloat16* __restrict__ km, const float* __restrict__ partial, const int nchunks,
                                       const float divisor, const int64_t bh, float* stage, __nv_bfloat16* km_out,
                                       uint4 (&mean)[2]) {
  const int t = threadIdx.x, c = RowTile<D, false>::block(t);
  if (km != nullptr) {
    mean[0] = reinterpret_cast<const uint4*>(km + bh * D + c * 16)[0];
    mean[1] = reinterpret_cast<const uint4*>(km + bh * D + c * 16)[1];
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
    reinterpret_cast<__nv_bfloat16*>(stage)[t] = m;
    if (km_out != nullptr) km_out[bh * D + t] = m;
  }
  __syncthreads();
  mean[0] = reinterpret_cast<const uint4*>(stage)[2 * c];
  mean[1] = reinterpret_cast<const uint4*>(stage)[2 * c + 1];
}

template <int D, bool kHalves>
__device__ __forceinline__ void quant_rows_store(const uint4 (&w)[RowTile<D, kHalves>::kPasses][2], uint8_t* __restrict__ codes_tile,
                                                 uint8_t* __restrict__ sf_tile, uint8_t* sf_smem) {
  using R = RowTile<D, kHalves>;
  const int t = threadIdx.x, c = R::block(t), rl = R::row(t);
  // sf_atom_offset of row rl + p * kStep is the sum of both offsets, the second a constant (left to the compiler, the addresses were
  // 15 % of the instructions)
  uint8_t* const sf_row = sf_smem + (c >> 2) * 512 + sf_atom_offset(rl, c & 3);
  uint8_t* const out = codes_tile + rl * (D / 2) + c * 8;
#pragma unroll
  for (int p = 0; p < R::kPasses; ++p) {
    uint32_t m2 = habsmax2(habsmax2(w[p][0].x, w[p][0].y), habsmax2(w[p][0].z, w[p][0].w));
    m2 = abs2(habsmax2(m2, habsmax2(habsmax2(w[p][1].x, w[p][1].y), habsmax2(w[p][1].z, w[p][1].w))));
    uint32_t sfb; float inv;
    block_scale(fmaxf(bf16_lo(m2), bf16_hi(m2)), sfb, inv);
    const float2 inv2 = make_float2(inv, inv);
    uint32_t code[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 f0 = mul2_ftz(bf16x2_to_f32(w[p][i].x), inv2), f1 = mul2_ftz(bf16x2_to_f32(w[p][i].y), inv2);
      const float2 f2 = mul2_ftz(bf16x2_to_f32(w[p][i].z), inv2), f3 = mul2_ftz(bf16x2_to_f32(w[p][i].w), inv2);
      code[i] = f32x8_to_e2m1x8(f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y);
    }
    *reinterpret_cast<uint2*>(out + p * (R::kStep * D / 2)) = make_uint2(code[0], code[1]);
    sf_row[sf_atom_offset(p * R::kStep, 0)] = (uint8_t)sfb;
  }
  __syncthreads();
  constexpr int SFV = (D / 64) * 512 / 16;                           // 16-byte vectors of scales
  if (t < SFV) reinterpret_cast<uint4*>(sf_tile)[t] = reinterpret_cast<const uint4*>(sf_smem)[t];
}


}  // namespace sage3
