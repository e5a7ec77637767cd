// Attention of a few query rows per head (decoding): the operands, the arithmetic of the softmax and the rounding of P are
// those of attn.cu, the work is split over the keys instead of the query rows.  There a tile of 128 query rows is worked on
// whole, and its key tiles one after another: P is rounded relative to the running row maximum, so a tile has to know the
// maximum of all tiles before it.  Here that maximum comes from a pass of its own:
//   decode_scores_kernel   a CTA walks key tiles: K is smoothed and quantised on the way, scores of all rows that share the kv
//                          head (with delta_s) -> memory, and their tile maxima
//   decode_output_kernel   one warp per run of key tiles: running maximum before the run from the tile maxima, P^, P^.V^;
//                          partial outputs; the last CTA of a kv head to finish adds them up
// The FP4 rows that are long - keys, channels of V^T - are the 16-row operand of mma.m16n8k16, the query rows the 8 columns:
// tcgen05's smallest tile has 128 rows of the other kind, and its operands would have to go through shared and tensor
// memory.  Values are expanded to halves together with their block scale, which is exact (2 + 4 significant bits, 2^-10 ...
// 2688), products are exact and sums fp32.  The order of elements along the contraction is free as long as both operands have
// the same: a lane takes whole quantisation blocks of a row, so that maxima, scales and codes need no exchange between lanes.
// What bounds it: on a full chip the conversions between the formats and their latencies (half of the issue slots in use,
// the tensor pipe 5 % busy, K at 2.7 TB/s), on few heads a chain of a few dependent loads.  Whole operator on the device,
// against tiles of 128 query rows: B8 H32/8 Nk4096 131 -> 63 us, B1 70 -> 19, B3 H32/4 Nk16384 258 -> 56.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.h"
#include "quant_v.cuh"

namespace sage3 {

namespace {

constexpr int kTile = 128;
constexpr int kWarps = 4, kThreads = 32 * kWarps;        // output kernel
constexpr int kScoreThreads = 256;
constexpr int kMaxChunks = 64;                           // CTAs of the output kernel per kv head
constexpr int kMaxRows = 64;                             // query rows per kv head

struct DecodeParams {
  const uint8_t *q_codes, *q_sf;
  uint8_t *vt_codes, *vt_sf;
  const __nv_bfloat16* v;                                // scores kernel with kV: V as it is
  int64_t v_sb, v_sh, v_sn;
  const __nv_bfloat16 *k, *qm, *km;                      // km: the K mean, or
  const float* partial;                                  // its partial sums, [kv][mean_chunks][D], or neither
  __nv_bfloat16* km_out;
  int64_t k_sb, k_sh, k_sn;
  int Hkv, mean_chunks, d_in;
  bool smooth;
  __nv_bfloat16* out;
  float* lse;
  const float* lse_add;
  int64_t o_sb, o_sh, o_sn;
  int kvs, Hq, G, Nq, Nk, Tk, rows;                      // kv heads of the batch; rows = G * Nq query rows share one
  int causal, d_out;
  int score_run;                                         // scores kernel: key tiles per CTA
  int run, chunks;                                       // output kernel: key tiles per warp, CTAs per kv head
  float scale_log2, sm_scale;
  float *scores, *tile_max, *o_part, *l_part, *m_part;   // [kv][rows][Tk*128], [kv][rows][Tk], [kv][rows][chunks] ([D])
  int* counter;                                          // [kv][rows]: CTAs of the output kernel that are done with a group of rows
};

__device__ __forceinline__ uint32_t e2m1x2_to_half2(const float lo, const float hi) {   // rounded to E2M1, as halves
  uint32_t r;
  asm("{\n"
      ".reg .b8 b;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b, %2, %1;\n"
      "cvt.rn.f16x2.e2m1x2 %0, b;\n"
      "}"
      : "=r"(r)
      : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint32_t hmul2(const uint32_t a, const uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// 8 E2M1 codes times a scale (twice in a half pair) -> 4 half pairs, in order
__device__ __forceinline__ void expand8(const uint32_t w, const uint32_t scale2, uint32_t* h) {
  asm("{\n"
      ".reg .b8 b0, b1, b2, b3;\n"
      "mov.b32 {b0, b1, b2, b3}, %4;\n"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n"
      "}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(w));
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = hmul2(h[i], scale2);
}
// two E4M3 bytes -> a half pair each
__device__ __forceinline__ void scales2(const uint32_t bytes, uint32_t& lo2, uint32_t& hi2) {
  uint32_t h;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"((uint16_t)bytes));
  lo2 = __byte_perm(h, h, 0x1010);
  hi2 = __byte_perm(h, h, 0x3232);
}
// What lane `tg` of the four that share a row holds of it, as words of two codes or values:
//   V^T, P (128 keys)   keys 32 tg ... + 31: one 16-byte load of codes
//   Q, K (D channels)   16-channel blocks tg and (D=128) tg + 4: the four lanes' loads of bf16 K fall into one line, which
//                       is what the L1 is short of (a quarter of a row per lane: two lines, 88 -> 85 us for the whole operator at B8 H32/8 Nk4096)
struct RawRow { uint32_t w[4], sf; };
__device__ __forceinline__ RawRow raw_keys(const uint8_t* codes, const uint8_t* sf, const int row, const int tg) {
  const uint4 v = *reinterpret_cast<const uint4*>(codes + row * 64 + tg * 16);
  return {{v.x, v.y, v.z, v.w}, *reinterpret_cast<const uint16_t*>(sf + (tg >> 1) * 512 + sf_atom_offset(row, (tg & 1) * 2))};
}
template <int D>
__device__ __forceinline__ RawRow raw_channels(const uint8_t* codes, const uint8_t* sf, const int row, const int tg) {
  RawRow x = {};
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    const uint2 v = *reinterpret_cast<const uint2*>(codes + row * (D / 2) + (tg + 4 * i) * 8);
    x.w[2 * i] = v.x; x.w[2 * i + 1] = v.y;
    x.sf |= (uint32_t)sf[i * 512 + sf_atom_offset(row, tg)] << (8 * i);
  }
  return x;
}
template <int W>
__device__ __forceinline__ void expand_row(const RawRow& x, uint32_t (&h)[W]) {
  uint32_t s0, s1;
  scales2(x.sf, s0, s1);
#pragma unroll
  for (int i = 0; i < W / 4; ++i) expand8(x.w[i], i < 2 ? s0 : s1, &h[4 * i]);
}
template <bool kBf16>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t a0, const uint32_t a1, const uint32_t a2, const uint32_t a3,
                                         const uint32_t b0, const uint32_t b1) {
  if (kBf16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 keys (parts of rows in registers) times 8 query rows (parts as vectors, 32 lanes apart, in shared memory)
template <bool kBf16, int W>
__device__ __forceinline__ void product(float (&s)[4], const uint32_t (&k)[2][W], const uint4* f) {
#pragma unroll
  for (int j = 0; j < W / 4; ++j) {
    const uint4 b = f[j * 32];
    mma16816<kBf16>(s, k[0][4 * j], k[1][4 * j], k[0][4 * j + 1], k[1][4 * j + 1], b.x, b.y);
    mma16816<kBf16>(s, k[0][4 * j + 2], k[1][4 * j + 2], k[0][4 * j + 3], k[1][4 * j + 3], b.z, b.w);
  }
}

// Where the score of key `k` of a tile lies: key 32 a + 4 b + c at 16 b + 4 a + c, so that the output kernel's four lanes
// read 64 contiguous bytes.
__device__ __forceinline__ constexpr int score_place(const int k) { return (k & 28) * 4 + (k >> 5) * 4 + (k & 3); }

// A CTA takes `score_run` key tiles one after another, each warp 16 keys of a tile, and fetches the rows of the next while it
// works on the present one.  K is smoothed, quantised and multiplied where it was loaded, so neither its codes nor delta_s
// exist in memory.  kOne: at most 8 query rows; the quantised rows then take the registers of the smoothed ones.
// (One tile per CTA of four warps, 32 keys each: 47 us at B8 H32/8 Nk4096, so 26; with V beside it 35, for 18 us less in the launch
// before.)
// kV: V of the same key tile comes through shared memory meanwhile and is quantised behind the scores: the conversions of K leave most
// of the memory's time unused, and K, of which the launch before has just taken the sums, is still in L2 where V has not been read in
// between.
// (D=128 only, see decode_takes_v.)
constexpr int kVRowsBytes = kTile * 128 * 2 + 8 * 16;    // 16-token blocks 16 bytes further apart, for the banks
template <int D, bool kOne, bool kV>
__global__ __launch_bounds__(kScoreThreads, D == 128 ? 2 : 3) void decode_scores_kernel(const DecodeParams P) {
  static_assert(!kV || D == 128, "8 warps of 16 channels each");
  constexpr int W = D / 8;                               // words of a lane's part of a row, as halves or bf16
  extern __shared__ __align__(16) uint32_t frag[];       // [groups of 8 query rows][W / 4][32 lanes][4]: Q^, then their Q means
  __shared__ __align__(16) __nv_bfloat16 mean_s[D];
  __shared__ float tmax[2][8][kOne ? 8 : kMaxRows];
  __shared__ __align__(16) uint8_t v_sf[kV ? 1024 : 16];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tg = lane & 3;
  const int kv = blockIdx.y, groups = kOne ? 1 : (P.rows + 7) / 8;
  const int first = blockIdx.x * P.score_run, end = min(first + P.score_run, P.Tk);
  pdl_launch_dependents();
  const __nv_bfloat16* src = P.k + kv / P.Hkv * P.k_sb + kv % P.Hkv * P.k_sh;
  auto channel = [](const int quarter, const int j) { return 16 * (quarter + 4 * (j >> 1)) + 8 * (j & 1); };   // first of 8
  uint4 w[2][W / 4];                                     // rows 16 warp + g and + 8 of the tile
  auto load = [&](const int tile) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int key = tile * kTile + 16 * warp + g + 8 * i;
#pragma unroll
      for (int j = 0; j < W / 4; ++j)
        w[i][j] = key < P.Nk && channel(tg, j) < P.d_in ? *reinterpret_cast<const uint4*>(src + (int64_t)key * P.k_sn + channel(tg, j))
                                                        : make_uint4(0, 0, 0, 0);
    }
  };
  load(first);
  uint8_t* const v_rows = reinterpret_cast<uint8_t*>(frag) + groups * 2 * 32 * W * 4;
  auto load_v = [&](const int tile) {                    // 16-byte pieces of whole rows; zeros beyond the keys and channels there are
    constexpr int CH = D / 8, RPP = kScoreThreads / CH;
    const __nv_bfloat16* v = P.v + kv / P.Hkv * P.v_sb + kv % P.Hkv * P.v_sh + t % CH * 8;
#pragma unroll
    for (int p = 0; p < kTile / RPP; ++p) {
      const int row = p * RPP + t / CH, key = tile * kTile + row;
      cp_async16(smem_u32(v_rows) + row * D * 2 + (row >> 4) * 16 + t % CH * 16, v + (int64_t)min(key, P.Nk - 1) * P.v_sn,
                 key < P.Nk && t % CH * 8 < P.d_in);
    }
  };
  if (kV) load_v(first);
  pdl_wait();
  if (blockIdx.x == 0 && t < P.rows) P.counter[kv * P.rows + t] = 0;
  for (int i = t; i < groups * 64; i += kScoreThreads) {
    const int n = i >> 6, r = 8 * n + ((i & 31) >> 2), quarter = i & 3;      // (threads of a warp: all Q^ or all means)
    const int64_t head = (int64_t)kv * P.G + min(r, P.rows - 1) / P.Nq;
    uint32_t x[W];
    if ((i & 32) == 0) {
      RawRow raw = {};
      if (r < P.rows) raw = raw_channels<D>(P.q_codes + head * kTile * (D / 2), P.q_sf + head * (D / 64) * 512, r % P.Nq, quarter);
      expand_row(raw, x);
    } else {
#pragma unroll
      for (int j = 0; j < W / 4; ++j)
        reinterpret_cast<uint4*>(x)[j] = __ldcg(reinterpret_cast<const uint4*>(P.qm + head * D + channel(quarter, j)));
    }
#pragma unroll
    for (int j = 0; j < W / 4; ++j)
      reinterpret_cast<uint4*>(frag)[((i >> 5) * (W / 4) + j) * 32 + (i & 31)] = make_uint4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
  }
  if (t >= kScoreThreads - D) {
    // the mean: given, or from the partial sums (same order and rounding as in the other K kernel), or none
    const int d = t - (kScoreThreads - D);
    __nv_bfloat16 m = __float2bfloat16_rn(0.f);
    if (P.km != nullptr) {
      m = P.km[(int64_t)kv * D + d];
    } else if (P.partial != nullptr) {
      const float* p = P.partial + (int64_t)kv * P.mean_chunks * D + d;
      float s = 0.f;
#pragma unroll 16
      for (int i = 0; i < P.mean_chunks; ++i) s += __ldcg(p + i * D);
      m = __float2bfloat16_rn(s / (float)P.Nk);
      if (blockIdx.x == 0 && P.km_out != nullptr) P.km_out[(int64_t)kv * D + d] = m;
    }
    mean_s[d] = m;
  }
  __syncthreads();
  const int64_t ld = (int64_t)P.Tk * kTile;
#pragma unroll 1
  for (int tile = first; tile < end; ++tile) {
    uint32_t kb[2][W];                                   // smoothed rows
    uint32_t amax[2][W / 4];
    const int key = tile * kTile + 16 * warp + g;
#pragma unroll
    for (int j = 0; j < W / 4; ++j) {
      const uint4 mean = *reinterpret_cast<const uint4*>(&mean_s[channel(tg, j)]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint4 x = w[i][j];
        if (P.smooth && key + 8 * i < P.Nk) x = subtract_mean(x, mean);    // padding rows stay zero
        kb[i][4 * j] = x.x; kb[i][4 * j + 1] = x.y; kb[i][4 * j + 2] = x.z; kb[i][4 * j + 3] = x.w;
        amax[i][j] = habsmax2(habsmax2(x.x, x.y), habsmax2(x.z, x.w));
      }
    }
    if (tile + 1 < end) load(tile + 1);
    // scores start from delta_s
    auto delta_s = [&](float (&s)[4], const int n) {
      s[0] = s[1] = s[2] = s[3] = 0.f;
      product<true, W>(s, kb, reinterpret_cast<const uint4*>(frag) + (2 * n + 1) * (W / 4) * 32 + lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = __bfloat162float(__float2bfloat16_rn(s[i]));
    };
    auto quantise = [&](uint32_t (&kq)[2][W]) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int blk = 0; blk < W / 8; ++blk) {
          const uint32_t m2 = abs2(habsmax2(amax[i][2 * blk], amax[i][2 * blk + 1]));
          uint32_t sfb, sf2, unused;
          float inv;
          block_scale(fmaxf(bf16_lo(m2), bf16_hi(m2)), sfb, inv);
          scales2(sfb, sf2, unused);
          const float2 inv2 = make_float2(inv, inv);
#pragma unroll
          for (int j = 8 * blk; j < 8 * blk + 8; ++j) {
            const float2 x = mul2_ftz(bf16x2_to_f32(kb[i][j]), inv2);
            kq[i][j] = hmul2(e2m1x2_to_half2(x.x, x.y), sf2);
          }
        }
      }
    };
    auto scores = [&](float (&s)[4], const uint32_t (&kq)[2][W], const int n) {
      product<false, W>(s, kq, reinterpret_cast<const uint4*>(frag) + 2 * n * (W / 4) * 32 + lane);
      // columns: query rows 8 n + 2 tg and + 1, rows: keys `key` and + 8
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = 8 * n + 2 * tg + j;
        const int lim = P.causal ? min(P.Nk - 1, r % P.Nq + P.Nk - P.Nq) : P.Nk - 1;       // last visible key
        const float lo = key <= lim ? s[j] : __uint_as_float(0xff800000u), hi = key + 8 <= lim ? s[2 + j] : __uint_as_float(0xff800000u);
        if (r < P.rows) {
          float* row = P.scores + ((int64_t)kv * P.rows + r) * ld + tile * kTile + score_place(16 * warp + g);
          row[0] = lo;
          row[score_place(8)] = hi;
        }
        float m = fmaxf(fmaxf(lo, hi), kNoMax);
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
        if (g == 0) tmax[tile & 1][warp][r] = m;
      }
    };
    float s[4];
    if constexpr (kOne) {
      delta_s(s, 0);
      quantise(kb);
      scores(s, kb, 0);
    } else {
      uint32_t kq[2][W];
      quantise(kq);
#pragma unroll 1
      for (int n = 0; n < groups; ++n) {
        delta_s(s, n);
        scores(s, kq, n);
      }
    }
    if (kV) cp_async_wait_all();
    __syncthreads();                                     // (the other half of tmax is written next)
    if (t < P.rows) {
      float m = tmax[tile & 1][0][t];
#pragma unroll
      for (int i = 1; i < 8; ++i) m = fmaxf(m, tmax[tile & 1][i][t]);
      P.tile_max[((int64_t)kv * P.rows + t) * P.Tk + tile] = m;
    }
    if constexpr (kV) {
      const int64_t vt = (int64_t)kv * P.Tk + tile;
      const int d = (warp * 4 + (lane >> 3)) * 4, blk = lane & 7;
      uint2 x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = *reinterpret_cast<const uint2*>(v_rows + (blk * 16 + i) * D * 2 + blk * 16 + d * 2);
      quant_v_block(x, d, blk, false, P.vt_codes + vt * (D * 64), v_sf);
      __syncthreads();                                   // the rows have been read, the scales are complete
      if (tile + 1 < end) load_v(tile + 1);
      if (t < 64) reinterpret_cast<uint4*>(P.vt_sf + vt * 1024)[t] = reinterpret_cast<const uint4*>(v_sf)[t];
    }
  }
}

// Key tiles from the last to the first, as in attn.cu; a warp takes `run` of them, a CTA 4 * run.
template <int D, int NT>
__global__ __launch_bounds__(kThreads, NT == 1 ? 4 : 3) void decode_output_kernel(const DecodeParams P) {
  constexpr int MT = D / 16, RO = 8 * NT;
  __shared__ __align__(16) float o_s[kWarps][RO][D + 4];
  __shared__ float m_s[kWarps][RO], l_s[kWarps][RO];
  __shared__ float fac[RO][kMaxChunks];
  __shared__ int last_s;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, tg = lane & 3;
  const int chunk = blockIdx.x % P.chunks, kv = blockIdx.x / P.chunks;
  const int r0 = blockIdx.y * RO, nr = min(RO, P.rows - r0);
  const int end = (chunk * kWarps + warp) * P.run, first = min(end + P.run, P.Tk) - 1;    // tiles first ... end, or none
  const float c = P.scale_log2;
  const int64_t row0 = (int64_t)kv * P.rows + r0, ld = (int64_t)P.Tk * kTile;
  float m_run[NT], l[NT], o[NT][MT][4];
  pdl_wait();
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    float m = kNoMax;
    if (8 * n + g < nr)
      for (int i = max(first, end - 1) + 1 + tg; i < P.Tk; i += 4) m = fmaxf(m, P.tile_max[(row0 + 8 * n + g) * P.Tk + i]);
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m_run[n] = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    l[n] = 0.f;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[n][mt][i] = 0.f;
  }
#pragma unroll 1
  for (int tile = first; tile >= end; --tile) {
    const uint8_t* vc = P.vt_codes + ((int64_t)kv * P.Tk + tile) * (D * 64);
    const uint8_t* vs = P.vt_sf + ((int64_t)kv * P.Tk + tile) * 1024;
    // V of this tile on its way during the softmax: D lines of 64 bytes of codes, 1 KB of scales (B32 H32 Nk2000: operator 430 ->
    // 420 us; registers for it would cost a CTA per SM: 128 -> 96 for five instead of four is 3 to 7 % slower)
#pragma unroll
    for (int i = 0; i < D / 64; ++i) asm volatile("prefetch.global.L1 [%0];" ::"l"(vc + (i * 32 + lane) * 128));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(vs + (lane & 7) * 128));
    uint32_t p[NT][16];                                  // keys 32 tg ... + 31 of query g
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const bool live = 8 * n + g < nr;
      const int64_t row = row0 + 8 * n + g;
      float4 s[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float off = __uint_as_float(0xff800000u);
        s[i] = live ? *reinterpret_cast<const float4*>(P.scores + row * ld + tile * kTile + 16 * i + 4 * tg)
                    : make_float4(off, off, off, off);
      }
      const float m_new = fmaxf(m_run[n], live ? P.tile_max[row * P.Tk + tile] : kNoMax);
      const float alpha = ex2_approx((m_run[n] - m_new) * c);
      m_run[n] = m_new;
      l[n] *= alpha;
      const float offset = fmaf(m_new, c, kLog2Inv2688);
#pragma unroll
      for (int blk = 0; blk < 2; ++blk) {
        float bm = kNoMax;
#pragma unroll
        for (int i = 4 * blk; i < 4 * blk + 4; ++i) bm = fmaxf(fmaxf(fmaxf(bm, s[i].x), fmaxf(s[i].y, s[i].z)), s[i].w);
        const float e = fmaf(bm, c, kLog2Inv6);
        const float sb = ex2_approx(e - offset);         // unrounded block scale
        uint32_t sb2, unused;
        scales2(f32_to_e4m3(sb), sb2, unused);
        float sum = 0.f;
#pragma unroll
        for (int i = 4 * blk; i < 4 * blk + 4; ++i) {    // P / block scale in [0, 6]
          const float x = ex2_approx(fmaf(s[i].x, c, -e)), y = ex2_approx(fmaf(s[i].y, c, -e));
          const float z = ex2_approx(fmaf(s[i].z, c, -e)), w = ex2_approx(fmaf(s[i].w, c, -e));
          sum += (x + y) + (z + w);
          p[n][2 * i] = hmul2(e2m1x2_to_half2(x, y), sb2);
          p[n][2 * i + 1] = hmul2(e2m1x2_to_half2(z, w), sb2);
        }
        l[n] = fmaf(sum, sb, l[n]);
      }
      // columns of the accumulator fragment: queries 2 tg and 2 tg + 1, whose factors lanes 8 tg and 8 tg + 4 have
      const float a0 = __shfl_sync(0xffffffffu, alpha, 8 * tg), a1 = __shfl_sync(0xffffffffu, alpha, 8 * tg + 4);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        o[n][mt][0] *= a0; o[n][mt][1] *= a1; o[n][mt][2] *= a0; o[n][mt][3] *= a1;
      }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      uint32_t v0[16], v1[16];
      expand_row(raw_keys(vc, vs, 16 * mt + g, tg), v0);
      expand_row(raw_keys(vc, vs, 16 * mt + g + 8, tg), v1);
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 8; ++j) mma16816<false>(o[n][mt], v0[2 * j], v1[2 * j], v0[2 * j + 1], v1[2 * j + 1], p[n][2 * j], p[n][2 * j + 1]);
    }
  }

  // ---- the four warps together: warp 0 has the lowest tiles, i.e. the largest maximum so far (or no other has any)
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    l[n] += __shfl_xor_sync(0xffffffffu, l[n], 1);
    l[n] += __shfl_xor_sync(0xffffffffu, l[n], 2);
    if (tg == 0) { m_s[warp][8 * n + g] = m_run[n]; l_s[warp][8 * n + g] = l[n]; }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 4; ++i) o_s[warp][8 * n + 2 * tg + (i & 1)][16 * mt + g + (i >> 1) * 8] = o[n][mt][i];
  }
  __syncthreads();
  if (t < nr * kWarps) {                                 // factors of the warps
    const int r = t / kWarps, w = t % kWarps;
    fac[r][w] = ex2_approx((m_s[w][r] - m_s[0][r]) * c);
  }
  __syncthreads();
#pragma unroll 4
  for (int i = t; i < nr * (D / 4); i += kThreads) {
    const int r = i / (D / 4), d = i % (D / 4) * 4;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float4 x = *reinterpret_cast<const float4*>(&o_s[w][r][d]);
      const float y = fac[r][w];
      sum.x = fmaf(x.x, y, sum.x); sum.y = fmaf(x.y, y, sum.y); sum.z = fmaf(x.z, y, sum.z); sum.w = fmaf(x.w, y, sum.w);
    }
    *reinterpret_cast<float4*>(P.o_part + ((row0 + r) * P.chunks + chunk) * D + d) = sum;
  }
  if (t < nr) {
    float sum = l_s[0][t];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) sum = fmaf(l_s[w][t], fac[t][w], sum);
    P.l_part[(row0 + t) * P.chunks + chunk] = sum;
    P.m_part[(row0 + t) * P.chunks + chunk] = m_s[0][t];
  }
  // ---- the last CTA of the kv head to get here adds all up, in a fixed order
  if (P.chunks > 1) {
    __threadfence();
    __syncthreads();
    if (t == 0) last_s = atomicAdd(P.counter + kv * P.rows + blockIdx.y, 1) == P.chunks - 1;
    __syncthreads();
    if (!last_s) return;
    __threadfence();
  } else {
    __syncthreads();
  }
#pragma unroll 2
  for (int r = warp; r < nr; r += kWarps) {              // factors of the chunks, row sum
    const int64_t i = (row0 + r) * P.chunks;
    float m[kMaxChunks / 32], ls[kMaxChunks / 32], sum = 0.f;
    const float top = __ldcg(P.m_part + i);              // chunk 0 has the maximum of the whole row
#pragma unroll
    for (int j = 0; j < kMaxChunks / 32; ++j) {
      const bool is = lane + 32 * j < P.chunks;
      m[j] = is ? __ldcg(P.m_part + i + lane + 32 * j) : kNoMax;
      ls[j] = is ? __ldcg(P.l_part + i + lane + 32 * j) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kMaxChunks / 32; ++j) {
      const float x = ex2_approx((m[j] - top) * c);
      fac[r][lane + 32 * j] = x;
      sum = fmaf(ls[j], x, sum);
    }
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
    if (lane == 0) {
      const bool keyless = top == kNoMax;                // a row that sees no key: zeros, LSE -inf
      l_s[0][r] = (keyless || sum != sum) ? 0.f : 1.0f / sum;
      if (P.lse != nullptr) {
        const int q = r0 + r;
        const int64_t li = ((int64_t)kv * P.G + q / P.Nq) * P.Nq + q % P.Nq;
        float v = keyless ? -INFINITY : (top * c + log2f(sum) + kLog2Inv2688) * (1.0f / kLog2e);
        if (P.lse_add != nullptr) v = fmaf(P.lse_add[li], P.sm_scale, v);
        P.lse[li] = v;
      }
    }
  }
  __syncthreads();
#pragma unroll 2
  for (int i = t; i < nr * (D / 4); i += kThreads) {
    const int r = i / (D / 4), d = i % (D / 4) * 4, q = r0 + r;
    const float* part = P.o_part + (row0 + r) * P.chunks * D + d;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int ch = 0; ch < P.chunks; ++ch) {
      const float4 x = __ldcg(reinterpret_cast<const float4*>(part + (int64_t)ch * D));
      const float y = fac[r][ch];
      sum.x = fmaf(x.x, y, sum.x); sum.y = fmaf(x.y, y, sum.y); sum.z = fmaf(x.z, y, sum.z); sum.w = fmaf(x.w, y, sum.w);
    }
    const int head = kv * P.G + q / P.Nq;
    const float inv = l_s[0][r];
    if (d < P.d_out)
      *reinterpret_cast<uint2*>(P.out + head / P.Hq * P.o_sb + head % P.Hq * P.o_sh + q % P.Nq * P.o_sn + d) =
          make_uint2(pack_bf16(sum.x * inv, sum.y * inv), pack_bf16(sum.z * inv, sum.w * inv));
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

template <int D, int NT>
cudaError_t launch(DecodeParams P, bool overlap, cudaStream_t stream) {
  int sms;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  const int groups = (P.rows + 8 * NT - 1) / (8 * NT), units = P.kvs * P.Tk;
  // runs: 16 warps per SM, at most kMaxChunks CTAs per kv head
  const int even = (int)(((int64_t)units * groups + sms * 16 - 1) / (sms * 16)), most = (P.Tk + kWarps * kMaxChunks - 1) / (kWarps * kMaxChunks);
  P.run = even > most ? even : most;
  P.chunks = (P.Tk + kWarps * P.run - 1) / (kWarps * P.run);
  const size_t frag = (size_t)(P.rows + 7) / 8 * 2 * 32 * (D / 8) * 4;         // 32 KB at most
  // key tiles per CTA of the scores kernel: the fewest tile times, a CTA's start counted as one
  const int slots = sms * (D == 128 ? 2 : 3);
  int64_t best = INT64_MAX;
  for (int run = 1; run <= 16; ++run) {
    const int64_t ctas = (int64_t)((P.Tk + run - 1) / run) * P.kvs, cost = (ctas + slots - 1) / slots * (run + 1);
    if (cost < best) { best = cost; P.score_run = run; }
  }
  const dim3 grid((P.Tk + P.score_run - 1) / P.score_run, P.kvs);
  constexpr bool kV = D == 128;
  if (kV && P.v != nullptr)
    e = launch_pdl(decode_scores_kernel<D, true, kV>, grid, kScoreThreads, frag + kVRowsBytes, stream, overlap, P);
  else
    e = launch_pdl(P.rows <= 8 ? decode_scores_kernel<D, true, false> : decode_scores_kernel<D, false, false>, grid, kScoreThreads, frag,
                   stream, overlap, P);
  if (e != cudaSuccess) return e;
  return launch_pdl(decode_output_kernel<D, NT>, dim3((unsigned)(P.kvs * P.chunks), groups), kThreads, 0, stream, true, P);
}

}  // namespace

// Against the tile kernels, whole operator (us): Nq=1 H32/8 Nk700 25 -> 14, Nk4096 70 -> 19; B16 H32/8 Nk4096, Nq=4 258 -> 166,
// Nq=8 260 -> 212, but Nq=16 (64 rows) 262 -> 315; B4 H32 Nq=16 (16 rows) Nk4000 181 -> 163, Nk700 26 -> 27.  With two or three
// key tiles there is nothing to split.
bool decode_fits(int Hq, int Hkv, int Nq, int Nk) {
  const int rows = Hq / Hkv * Nq;
  return Nk > 3 * kTile && rows <= kMaxRows && (Nq <= 8 || (Nq <= 16 && rows <= 32 && Nk > 1024));
}

// Only the kernels of one group of rows and D=128 (D=64 keeps half the warps busy with V: B8 H32 Nk2000 63.1 -> 64.1 us), and not where
// a launch is a chain of latencies anyhow (device time without / with, B1 H32/8: 32 tiles 11.3 / 11.7 us, 64 13.5 / 13.9, 96 16.6 / 15.8,
// 128 17.3 / 17.4, 160 18.7 / 18.6, 192 21.7 / 19.5, 256 16.8 / 16.2; B2 and B4, 128 tiles 16.6 / 15.8 and 15.1 / 14.3; B8, 2048 tiles
// 58.2 / 55.6; B32 224 / 202; B16 H32 Nk8000 779 / 679).
bool decode_takes_v(int B, int Hq, int Hkv, int Nq, int Nk, int D) {
  return D == 128 && Hq / Hkv * Nq <= 8 && (int64_t)B * Hkv * ((Nk + kTile - 1) / kTile) >= 128;
}

size_t decode_scratch_bytes(int B, int Hq, int Hkv, int Nq, int Nk, int D) {
  if (!decode_fits(Hq, Hkv, Nq, Nk)) return 0;
  const size_t Tk = (Nk + kTile - 1) / kTile, rows = (size_t)B * Hq * Nq, chunks = Tk < kMaxChunks ? Tk : kMaxChunks;
  return align256(rows * Tk * kTile * 4) + align256(rows * Tk * 4) + align256(rows * chunks * D * 4) +
         2 * align256(rows * chunks * 4) + align256(rows * 4);
}

cudaError_t launch_attn_decode(const AttnArgs& a, const DeltaSArgs& k, void* scratch, cudaStream_t stream) {
  if ((a.D != 128 && a.D != 64) || !decode_fits(a.Hq, a.Hkv, a.Nq, a.Nk)) return cudaErrorInvalidValue;
  DecodeParams P;
  P.q_codes = (const uint8_t*)a.q_codes; P.q_sf = (const uint8_t*)a.q_sf;
  P.vt_codes = (uint8_t*)a.vt_codes; P.vt_sf = (uint8_t*)a.vt_sf;
  P.v = (const __nv_bfloat16*)k.v; P.v_sb = k.v_sb; P.v_sh = k.v_sh; P.v_sn = k.v_sn;
  if ((P.v != nullptr) != decode_takes_v(a.B, a.Hq, a.Hkv, a.Nq, a.Nk, a.D)) return cudaErrorInvalidValue;
  P.k = (const __nv_bfloat16*)k.k; P.k_sb = k.k_sb; P.k_sh = k.k_sh; P.k_sn = k.k_sn;
  P.qm = (const __nv_bfloat16*)k.qm; P.km = (const __nv_bfloat16*)k.km; P.partial = (const float*)k.partial;
  P.km_out = (__nv_bfloat16*)k.km_out;
  P.smooth = P.km != nullptr || P.partial != nullptr;
  int chunk_tokens;
  quant_chunks(a.B * a.Hkv, a.Nk, &P.mean_chunks, &chunk_tokens);
  P.d_in = (k.d_in > 0 && k.d_in <= a.D) ? k.d_in : a.D;
  P.Hkv = a.Hkv;
  P.out = (__nv_bfloat16*)a.out; P.lse = a.lse; P.lse_add = a.lse_add;
  P.o_sb = a.o_sb; P.o_sh = a.o_sh; P.o_sn = a.o_sn;
  P.kvs = a.B * a.Hkv; P.Hq = a.Hq; P.G = a.Hq / a.Hkv; P.Nq = a.Nq; P.Nk = a.Nk; P.Tk = (a.Nk + kTile - 1) / kTile;
  P.rows = P.G * a.Nq;
  P.causal = a.causal;
  P.d_out = (a.d_out > 0 && a.d_out <= a.D) ? a.d_out : a.D;
  P.scale_log2 = a.sm_scale * kLog2e; P.sm_scale = a.sm_scale;
  const size_t rows = (size_t)P.kvs * P.rows, chunks = P.Tk < kMaxChunks ? P.Tk : kMaxChunks;
  char* w = reinterpret_cast<char*>(scratch);
  auto take = [&](size_t n) { char* p = w; w += align256(n); return p; };
  P.scores = (float*)take(rows * P.Tk * kTile * 4);
  P.tile_max = (float*)take(rows * P.Tk * 4);
  P.o_part = (float*)take(rows * chunks * a.D * 4);
  P.l_part = (float*)take(rows * chunks * 4);
  P.m_part = (float*)take(rows * chunks * 4);
  P.counter = (int*)take(rows * 4);
  if (a.D == 128) return P.rows <= 8 ? launch<128, 1>(P, k.after_quant, stream) : launch<128, 2>(P, k.after_quant, stream);
  return P.rows <= 8 ? launch<64, 1>(P, k.after_quant, stream) : launch<64, 2>(P, k.after_quant, stream);
}

}  // namespace sage3
