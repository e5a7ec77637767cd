// K quantisation + delta_s in one pass over K:
//   ks            = bf16(k - km)                                       sageattn4/api.py:184
//   K codes / SF  = NVFP4(ks), 128-token tiles                         quantization/fp4_quantization_4d.cu:492-569
//   delta_s[b, hq, qb, n] = bf16( sum_d qm[b, hq, qb, d] * ks[b, hkv, n, d] )   api.py:201
//
// The reference computes delta_s with a bf16 GEMM (fp32 accumulation, bf16 result) that it then widens to fp32.
// It stays bf16 here - the same values in half the bytes - because the attention kernel feeds each row to the
// tensor core as a bf16 operand (rank-1 update of the score accumulator), which restores the Q block mean that
// was removed before quantisation.
//
// One CTA per (128-key tile, kv head): the K tile is read from HBM ONCE, smoothed in registers, quantised (the
// same device function as the fused quantisation kernel, so codes and scales are bit-identical) and laid out
// in shared memory as the B operand of tcgen05.mma kind::f16; the Q block means of every query head of the GQA
// group (contiguous in memory, so the group counts as one list of rows of A, 128 at a time: the four heads of a decode
// step are one MMA instead of four) are multiplied against it with the accumulator in tensor
// memory; the [128 query blocks x 128 keys] result goes as bf16 through a swizzled staging tile in shared memory
// and leaves with two TMA stores (whole 128-byte lines; rows beyond the last query block are clipped by the
// tensor map).  HBM-bound: the output ([Tq x 128] bf16 per CTA and query head) dominates the traffic, in a chain of
// dependent steps per CTA.  So a CTA walks several key tiles of a head: tensor memory, barrier and K means are set up once, and
// the next tile's rows are on their way (in the registers that the quantised tile leaves) during the MMAs and stores of the
// present one (B4 H32 N4096 D64 52 -> 45 us, B1 H40 N9450 66 -> 57 us, B1 H40 N32760 327 -> 314 us, by now 282; one tile per CTA with three
// CTAs per SM was the best without that).  Up to 128 rows of A (kMulti = false) A is loaded once per CTA; with more, the next
// 128 wait in registers during a round (390 us without).
//
// kPack: K-packing mode (pack.cu) on the way in - a tile is 8 groups of 16 slots, its 120 tokens are smoothed, laid out
// and turned into mean and residuals by one warp per group, in place in the operand tile; the lambdas leave from here.
// (B4 H32 N2048 D128: a packing kernel in front, whose output this one and the V quantiser read back, took 111 us.)
//
// Operand layout in shared memory (K-major, no swizzle): 8-row x 16-byte core matrices; the 16 row groups of one
// 8-channel chunk are contiguous (128 B apart), chunks are kChunk bytes apart - 16 bytes more than their size so
// that the lanes which write one row's chunks hit different banks (A: 16 of them, K: as RowTile deals them out).
#include <cuda.h>

#include <atomic>
#include <cstdint>

#include "common.cuh"
#include "kernels.h"
#include "pack_group.cuh"
#include "quant_rows.cuh"
#include "tensor_map.h"

namespace sage3 {

namespace {

constexpr uint32_t kChunk = 128 * 16 + 16;            // one 8-channel chunk of 128 rows (+ bank skew)

struct KDsParams {
  const __nv_bfloat16 *qm, *k, *km;
  const float* partial;                                // K channel sums when km is null (both null: no smoothing)
  __nv_bfloat16* km_out;
  int chunks;
  int64_t k_sb, k_sh, k_sn;
  uint8_t *k_codes, *k_sf;                             // null: K is quantised elsewhere
  __nv_bfloat16* ds;
  int* status;                                         // optional device status word
  float* lam;                                          // kPack: fp32 [B,Hkv,Tk*128]
  int Hkv, rows, Tk, Nk;                               // rows = query heads per kv head x query blocks per head
  const int* cu_k;
  int d_in;                                            // channels the K rows really have; the rest are zero
  int run;                                             // key tiles per CTA
};

constexpr int kDsStageBytes = 2 * 128 * 128;          // output staging: [2 key halves][128 rows x 128 bytes], 128-byte swizzle
template <int D, bool kMulti, bool kPack>
__global__ void __launch_bounds__(kThreads, 2) k_quant_delta_s_kernel(const __grid_constant__ CUtensorMap tm_ds,
                                                                      const KDsParams P) {
  constexpr int CH = D / 8, RPP = kThreads / CH, NP = kTile / RPP;
  constexpr uint32_t kTileBytes = CH * kChunk;
  extern __shared__ uint8_t dyn_raw[];
  uint8_t* dyn_smem = dyn_raw + ((1024u - (smem_u32(dyn_raw) & 1023u)) & 1023u);   // the swizzled staging tile needs it
  uint8_t* stage = dyn_smem;                           // output staging (first: 1024-byte aligned)
  uint8_t* sA = dyn_smem + kDsStageBytes;              // 128 Q block means [CH][kChunk]
  uint8_t* sB = sA + kTileBytes;                       // smoothed K tile  [CH][kChunk]
  uint8_t* sf_smem = sB + kTileBytes;                  // 2048 B
  uint8_t* misc = sf_smem + 2048;                      // mbarrier (8 B), tensor-memory slot (4 B), from byte 16 on the K means
  const uint32_t bar = smem_u32(misc), slot = smem_u32(misc + 8);
  const int first = blockIdx.x * P.run, bh = blockIdx.y, b = bh / P.Hkv, hkv = bh % P.Hkv;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, c = t % CH, rl = t / CH;

  // ---- the K tile: load, smooth, quantise, lay out as the B operand
  int Nk = P.Nk;
  if (P.cu_k != nullptr) {
    Nk = min(P.cu_k[b + 1] - P.cu_k[b], Nk);           // a packed batch: this sequence, cut at max_seqlen
    if (first * kTile >= Nk) {                          // beyond the sequence: nothing reads this tile or its delta_s
      pdl_wait();                                      // (this grid never ends before the one it follows)
      return;
    }
  }
  using R = RowTile<D, false>;
  const int kc = R::block(t), krl = R::row(t);          // K rows: 16 channels a thread (A rows, c and rl: 8)
  const __nv_bfloat16* src = P.k + (P.cu_k ? (int64_t)P.cu_k[b] * P.k_sn : b * P.k_sb) + hkv * P.k_sh + kc * 16;
  auto place = [&](const int p, const int i) {          // of channels 8 i ... of this thread's row p in sB
    const int row = p * R::kStep + krl;
    return reinterpret_cast<uint4*>(sB + (2 * kc + i) * kChunk + (row >> 3) * 128 + (row & 7) * 16);
  };
  const int end = min(first + P.run, P.cu_k != nullptr ? (Nk + kTile - 1) / kTile : P.Tk);
  // token in slot `row` of a tile (kPack: 16 slots hold 15 tokens, none the first)
  auto token_of = [&](const int tile, const int row) {
    if (!kPack) return tile * kTile + row;
    return (row & 15) == 0 ? -1 : (tile * (kTile / 16) + (row >> 4)) * kGroup + (row & 15) - 1;
  };
  uint4 w[R::kPasses][2];
  auto load = [&](const int tile) {
#pragma unroll
    for (int p = 0; p < R::kPasses; ++p) {             // all loads in flight before the first use
      const int n = token_of(tile, p * R::kStep + krl);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        w[p][i] = (n >= 0 && n < Nk && kc * 16 + 8 * i < P.d_in) ? *reinterpret_cast<const uint4*>(src + (int64_t)n * P.k_sn + 8 * i)
                                                                 : make_uint4(0, 0, 0, 0);
    }
  };
  load(first);
  if (t == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(slot, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(misc + 8);
  // only now: the attention kernel that may come in takes all of tensor memory, and waits for this grid
  pdl_launch_dependents();
  pdl_wait();                                          // the sums and block means of the launch before
  // A: Q block means of rows round*128 ... +127 (zeros beyond the last one)
  const __nv_bfloat16* qm_g = P.qm + (int64_t)bh * P.rows * D + c * 8;
  uint4 a_next[kMulti ? NP : 1];
  auto load_a = [&](const int round) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int row = p * RPP + rl, m = round * 128 + row;
      if constexpr (kMulti)
        a_next[p] = m < P.rows ? __ldcg(reinterpret_cast<const uint4*>(qm_g + (int64_t)m * D)) : make_uint4(0, 0, 0, 0);
      else
        cp_async16(smem_u32(sA) + c * kChunk + (row >> 3) * 128 + (row & 7) * 16, qm_g + (int64_t)min(m, P.rows - 1) * D, m < P.rows);
    }
  };
  if (!kMulti) load_a(0);
  const bool smooth = P.km != nullptr || P.partial != nullptr;
  // this thread's means: in registers, or (kMulti, where the waiting A rows take them) in shared memory
  uint4 mean[2];
  uint4* const mean_s = reinterpret_cast<uint4*>(misc + 16) + 2 * kc;
  if (smooth) {
    static_assert(kMaxChunks * D * 4 <= (int)kTileBytes, "partial rows of the K mean");
    k_mean<D>(P.km, P.partial + (int64_t)bh * P.chunks * D, P.chunks, (float)max(Nk, 1), bh, reinterpret_cast<float*>(sB),
              first == 0 ? P.km_out : nullptr, mean);
    if (kMulti && krl == 0) { mean_s[0] = mean[0]; mean_s[1] = mean[1]; }
    __syncthreads();                                   // every thread has its means: sB takes the K tile
  }
  bool ok = true;
  uint32_t done = 0;                                   // rounds so far, of all tiles
#pragma unroll 1
  for (int tile = first; tile < end && ok; ++tile) {
  if (smooth) {
    if (kMulti) { mean[0] = mean_s[0]; mean[1] = mean_s[1]; }
#pragma unroll
    for (int p = 0; p < R::kPasses; ++p)
      if (const int n = token_of(tile, p * R::kStep + krl); n >= 0 && n < Nk) {   // padding rows stay zero (the reference subtracts before padding)
        w[p][0] = subtract_mean(w[p][0], mean[0]);
        w[p][1] = subtract_mean(w[p][1], mean[1]);
      }
  }
#pragma unroll
  for (int p = 0; p < R::kPasses; ++p) { *place(p, 0) = w[p][0]; *place(p, 1) = w[p][1]; }
  if constexpr (kPack) {
    // one warp per group: rows 16 warp ... +15 of the tile, lane l channels l*C ... (8-channel chunks of sB)
    constexpr int C = D / 32;
    __syncthreads();
    uint8_t* grp = sB + (lane * C / 8) * kChunk + (lane * C % 8) * 2 + warp * 256;
    auto at = [&](const int slot) { return grp + (slot >> 3) * 128 + (slot & 7) * 16; };
    auto put = [&](const int slot, const float (&r)[C]) {
      if constexpr (C == 4) *reinterpret_cast<uint2*>(at(slot)) = make_uint2(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]));
      else                  *reinterpret_cast<uint32_t*>(at(slot)) = pack_bf16(r[0], r[1]);
    };
    float x[kGroup][C], m[C];
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      if constexpr (C == 4) {
        const uint2 raw = *reinterpret_cast<const uint2*>(at(j + 1));
        x[j][0] = bf16_lo(raw.x); x[j][1] = bf16_hi(raw.x); x[j][2] = bf16_lo(raw.y); x[j][3] = bf16_hi(raw.y);
      } else {
        const uint32_t raw = *reinterpret_cast<const uint32_t*>(at(j + 1));
        x[j][0] = bf16_lo(raw); x[j][1] = bf16_hi(raw);
      }
    }
    const float my_lam = pack_group<C>(x, lane, m, [&](const int j, const float (&r)[C]) { put(j + 1, r); });
    put(0, m);
    if (lane < 16) P.lam[((int64_t)bh * P.Tk + tile) * kTile + warp * 16 + lane] = my_lam;
    __syncthreads();
#pragma unroll
    for (int p = 0; p < R::kPasses; ++p) { w[p][0] = *place(p, 0); w[p][1] = *place(p, 1); }
  }
  if (P.k_codes != nullptr) {
    const int64_t kt = (int64_t)bh * P.Tk + tile;
    quant_rows_store<D, false>(w, P.k_codes + kt * (kTile * D / 2), P.k_sf + kt * ((D / 64) * 512), sf_smem);
  }
  if (tile + 1 < end) load(tile + 1);
  // ---- delta_s: for the query blocks of all heads of the group, 128 at a time
  constexpr uint32_t idesc = make_idesc_bf16(128, 128);
  constexpr uint32_t HI = (128u >> 4) | (1u << 14);                     // 8-row groups 128 B apart, no swizzle
  const uint32_t a_lo = (smem_u32(sA) >> 4) | ((kChunk >> 4) << 16);    // leading (K) offset = one chunk
  const uint32_t b_lo = (smem_u32(sB) >> 4) | ((kChunk >> 4) << 16);
  const int rounds = kMulti ? (P.rows + 127) / 128 : 1;
  if (kMulti) load_a(0);
  for (int round = 0; round < rounds && ok; ++round, ++done) {
    if constexpr (kMulti) {
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int row = p * RPP + rl;
        *reinterpret_cast<uint4*>(sA + c * kChunk + (row >> 3) * 128 + (row & 7) * 16) = a_next[p];
      }
    } else {
      cp_async_wait_all();
    }
    if (t == 0) bulk_wait_read0();                     // the previous round's stores have left the staging tile
    fence_proxy_async_smem();
    __syncthreads();
    if (t == 0) {
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)              // K = 16 per instruction = two chunks
        tc_mma_bf16(tmem, a_lo + kk * (2 * kChunk >> 4), HI, b_lo + kk * (2 * kChunk >> 4), HI, idesc, kk > 0 ? 1u : 0u);
      tc_commit(bar);
    }
    if (kMulti && round + 1 < rounds) load_a(round + 1);
    // bounded: a few microseconds normally; gives up after about a second.  (One vote behind the loop: 0.3 us of the
    // operator at B1 H32/8 N128 less than a vote on every poll, unlike in the attention kernel.)
    ok = __all_sync(0xffffffffu, mbar_wait(bar, done & 1, 1u << 18));
    if (!ok && P.status != nullptr && lane == 0) atomicCAS(P.status, 0, 50);
    tc_fence_after();
    if (ok) {
      // lane = query block (row of the staging tile), 64 keys per thread: warps 0-3 the tile's keys 0-63, warps 4-7
      // keys 64-127 (= the two 128-byte-wide store boxes)
      const int row = (warp & 3) * 32 + lane, half = warp >> 2;
      const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)half * 64;
      uint8_t* srow = stage + half * (128 * 128) + row * 128;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t r[32];
        tmem_ld32(taddr + 32 * part, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(srow + (((4 * part + i) ^ (row & 7)) << 4)) =
              make_uint4(pack_bf16(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1])),
                         pack_bf16(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3])),
                         pack_bf16(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5])),
                         pack_bf16(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7])));
      }
      fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();                                   // the staging tile is complete (and the accumulator read)
    if (ok && t == 0) {
      tma_store_3d(&tm_ds, smem_u32(stage), tile * kTile, round * 128, bh);
      tma_store_3d(&tm_ds, smem_u32(stage) + 128 * 128, tile * kTile + 64, round * 128, bh);
      bulk_commit_group();
    }
    // the accumulator and the A tile are rewritten by the next round; every thread leaves the loop together
    tc_fence_before();
    ok = __syncthreads_and(ok);
  }
  }
  if (t == 0) bulk_wait_read0();                       // the last stores have read the staging tile before the CTA ends
  if (!ok && t == 0) {
    // the MMAs issued last may still be running: give them time to drain before tensor memory is freed
    mbar_wait(bar, (done - 1) & 1, 1u << 16);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

}  // namespace

cudaError_t launch_delta_s(const DeltaSArgs& a, cudaStream_t stream) {
  KDsParams P;
  P.qm = (const __nv_bfloat16*)a.qm; P.k = (const __nv_bfloat16*)a.k; P.km = (const __nv_bfloat16*)a.km;
  P.k_sb = a.k_sb; P.k_sh = a.k_sh; P.k_sn = a.k_sn;
  P.k_codes = (uint8_t*)a.k_codes; P.k_sf = (uint8_t*)a.k_sf;
  P.ds = (__nv_bfloat16*)a.ds; P.status = a.status;
  P.partial = (const float*)a.partial; P.km_out = (__nv_bfloat16*)a.km_out;
  int chunk_tokens;
  quant_chunks(a.B * a.Hkv, a.Nk, &P.chunks, &chunk_tokens);
  P.Hkv = a.Hkv; P.rows = a.Hq / a.Hkv * a.Tq; P.Nk = a.Nk; P.lam = a.k_lambda;
  P.Tk = ((a.k_lambda ? (a.Nk + kGroup - 1) / kGroup * 16 : a.Nk) + 127) / 128;
  P.cu_k = a.cu_k;
  P.d_in = (a.d_in > 0 && a.d_in <= a.D) ? a.d_in : a.D;
  // key tiles per CTA: the fewest tile times on SMs with two CTAs each, a CTA's start counted as one; at most two where
  // lengths vary, since a CTA that has begun is not given to another sequence (16 prompts: 486 us, 500 with up to 16)
  int sms;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  int64_t best = INT64_MAX;
  for (int run = 1; run <= (a.cu_k != nullptr ? 2 : 16); ++run) {
    const int64_t ctas = (int64_t)((P.Tk + run - 1) / run) * a.B * a.Hkv, cost = (ctas + 2 * sms - 1) / (2 * sms) * (run + 1);
    if (cost < best) { best = cost; P.run = run; }
  }
  const dim3 grid((P.Tk + P.run - 1) / P.run, a.B * a.Hkv);
  // delta_s as a 3-D bf16 tensor (key, query block of the GQA group, batch x kv head); store boxes of 64 keys x 128 rows
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return cudaErrorInvalidValue;
  CUtensorMap tm;
  {
    const cuuint64_t nk_pad = (cuuint64_t)P.Tk * kTile;
    cuuint64_t dims[3] = {nk_pad, (cuuint64_t)P.rows, (cuuint64_t)a.B * a.Hkv};
    cuuint64_t strides[2] = {nk_pad * 2, nk_pad * 2 * (cuuint64_t)P.rows};
    cuuint32_t box[3] = {64, 128, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    if (enc(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, a.ds, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
  }
  const bool multi = P.rows > 128;
  const int smem = kDsStageBytes + 2 * (a.D / 8) * (int)kChunk + 2048 + 16 + a.D * 2 + 1024;
  static std::atomic<unsigned long long> ready[8];      // per kernel: devices on which the shared memory was asked for
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  using Kern = void (*)(CUtensorMap, KDsParams);
  static const Kern kerns[8] = {k_quant_delta_s_kernel<64, false, false>,  k_quant_delta_s_kernel<64, true, false>,
                                k_quant_delta_s_kernel<128, false, false>, k_quant_delta_s_kernel<128, true, false>,
                                k_quant_delta_s_kernel<64, false, true>,   k_quant_delta_s_kernel<64, true, true>,
                                k_quant_delta_s_kernel<128, false, true>,  k_quant_delta_s_kernel<128, true, true>};
  const int which = (a.k_lambda ? 4 : 0) + (a.D == 128 ? 2 : 0) + (multi ? 1 : 0);
  const Kern kern = kerns[which];
  auto& done = ready[which];
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev >= 64 || !(done.load(std::memory_order_acquire) & bit)) {
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    if (dev < 64) done.fetch_or(bit, std::memory_order_release);
  }
  return launch_pdl(kern, grid, kThreads, smem, stream, a.after_quant, tm, P);
}

}  // namespace sage3
