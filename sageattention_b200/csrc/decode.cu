// Attention of a few query rows per head (decoding): the operands, the arithmetic of the softmax and the rounding of P are
// those of attn.cu, the work is split over the keys instead of the query rows.  There a tile of 128 query rows is worked on
// whole, and its key tiles one after another: P is rounded relative to the running row maximum, so a tile has to know the
// maximum of all tiles before it.  Here that maximum comes from a pass of its own:
//   decode_scores_kernel   one warp per key tile: scores of all rows that share the kv head -> memory, and their tile maxima
//   decode_output_kernel   one warp per run of key tiles: running maximum before the run from the tile maxima, P^, P^.V^;
//                          partial outputs; the last CTA of a kv head to finish adds them up
// The FP4 rows that are long - keys, channels of V^T - are the 16-row operand of mma.m16n8k16, the query rows the 8 columns:
// tcgen05's smallest tile has 128 rows of the other kind, and its operands would have to go through shared and tensor
// memory.  Values are expanded to halves together with their block scale, which is exact (2 + 4 significant bits, 2^-10 ...
// 2688), products are exact and sums fp32.  The order of elements along the contraction is free as long as both operands have
// the same: a lane takes a quarter of a row, contiguous, so it loads it with one instruction - and of P a lane then holds 32
// keys of one query, i.e. whole quantisation blocks: their maxima, scales and codes need no exchange between lanes.
// What bounds it: on a full chip the expansion of the codes (32 instructions per row and lane, the MMA are 8), on few heads
// the latency of a few dependent loads.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.h"

namespace sage3 {

namespace {

constexpr int kTile = 128;
constexpr int kWarps = 4, kThreads = 32 * kWarps;
constexpr int kMaxChunks = 64;                           // CTAs of the output kernel per kv head

struct DecodeParams {
  const uint8_t *q_codes, *q_sf, *k_codes, *k_sf, *vt_codes, *vt_sf;
  const __nv_bfloat16* ds;
  __nv_bfloat16* out;
  float* lse;
  const float* lse_add;
  int64_t o_sb, o_sh, o_sn;
  int kvs, Hq, G, Nq, Nk, Tk, rows;                      // kv heads of the batch; rows = G * Nq query rows share one
  int causal, d_out;
  int run, chunks;                                       // output kernel: key tiles per warp, CTAs per kv head
  float scale_log2, sm_scale;
  float *scores, *tile_max, *o_part, *l_part, *m_part;   // [kv][rows][Tk*128], [kv][rows][Tk], [kv][rows][chunks] ([D])
  int* counter;                                          // [kv][groups of rows]
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
// Row of E values (E = 128 or 64) of the tile whose codes and scale atoms start at `codes`, `sf`: the quarter of lane `tg` of
// the four that share it, as E / 8 half pairs.  `raw` and `expand` apart: all loads of a tile go out first.
template <int E> struct RawRow { uint32_t w[E / 32], sf; };
template <int E>
__device__ __forceinline__ RawRow<E> raw_row(const uint8_t* codes, const uint8_t* sf, const int row, const int tg) {
  RawRow<E> x;
  const uint8_t* s = sf + (row & 31) * 16 + (row >> 5) * 4;
  if (E == 128) {
    const uint4 v = *reinterpret_cast<const uint4*>(codes + row * 64 + tg * 16);
    x.w[0] = v.x; x.w[1] = v.y; x.w[E / 32 - 2] = v.z; x.w[E / 32 - 1] = v.w;
    x.sf = *reinterpret_cast<const uint16_t*>(s + (tg >> 1) * 512 + (tg & 1) * 2);
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(codes + row * 32 + tg * 8);
    x.w[0] = v.x; x.w[1] = v.y;
    x.sf = s[tg];
  }
  return x;
}
template <int E>
__device__ __forceinline__ void expand_row(const RawRow<E>& x, uint32_t (&h)[E / 8]) {
  uint32_t s0, s1;
  scales2(x.sf, s0, s1);
#pragma unroll
  for (int i = 0; i < E / 32; ++i) expand8(x.w[i], i < 2 ? s0 : s1, &h[4 * i]);
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t a0, const uint32_t a1, const uint32_t a2, const uint32_t a3,
                                         const uint32_t b0, const uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT = groups of 8 query rows
template <int D, int NT>
__global__ __launch_bounds__(kThreads) void decode_scores_kernel(const DecodeParams P) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
  const int unit = blockIdx.x * kWarps + (threadIdx.x >> 5), r0 = blockIdx.y * 8 * NT;
  pdl_launch_dependents();
  if (unit >= P.kvs * P.Tk) return;
  const int kv = unit / P.Tk, tile = unit % P.Tk;
  // columns of the result fragment: queries 2 tg and 2 tg + 1 of each group.  Head of query row r, counted over the batch: kv
  // heads are numbered b * Hkv + h, so it is kv * G + r / Nq
  int64_t ds_row[NT][2];
  int lim[NT][2];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = r0 + 8 * n + 2 * tg + j, head = r < P.rows ? r / P.Nq : 0;
      ds_row[n][j] = ((int64_t)kv * P.G + head) * P.Tk * kTile;
      lim[n][j] = P.causal ? min(P.Nk - 1, r - head * P.Nq + P.Nk - P.Nq) : P.Nk - 1;      // last visible key
    }
  pdl_wait();
  if (tile == 0 && lane == 0) P.counter[kv * gridDim.y + blockIdx.y] = 0;
  const uint8_t* kc = P.k_codes + (int64_t)unit * kTile * (D / 2);
  const uint8_t* ks = P.k_sf + (int64_t)unit * (D / 64) * 512;
  uint32_t q[NT][D / 8];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int r = r0 + 8 * n + g;
    RawRow<D> x = {};
    if (r < P.rows) {
      const int64_t head = (int64_t)kv * P.G + r / P.Nq;
      x = raw_row<D>(P.q_codes + head * kTile * (D / 2), P.q_sf + head * (D / 64) * 512, r % P.Nq, tg);
    }
    expand_row<D>(x, q[n]);
  }
  float m[NT][2];
#pragma unroll
  for (int n = 0; n < NT; ++n) m[n][0] = m[n][1] = kNoMax;
  const int64_t ld = (int64_t)P.Tk * kTile;
#pragma unroll 4
  for (int mt = 0; mt < 8; ++mt) {
    const int row = 16 * mt + g, key = tile * kTile + row;
    uint32_t k0[D / 8], k1[D / 8];
    expand_row<D>(raw_row<D>(kc, ks, row, tg), k0);
    expand_row<D>(raw_row<D>(kc, ks, row + 8, tg), k1);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      if (P.ds != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = __bfloat162float(P.ds[ds_row[n][i & 1] + key + (i >> 1) * 8]);
      }
#pragma unroll
      for (int j = 0; j < D / 16; ++j) mma16816(s, k0[2 * j], k1[2 * j], k0[2 * j + 1], k1[2 * j + 1], q[n][2 * j], q[n][2 * j + 1]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + 8 * n + 2 * tg + (i & 1), kk = key + (i >> 1) * 8;
        if (kk > lim[n][i & 1]) s[i] = __uint_as_float(0xff800000u);
        if (r < P.rows) P.scores[((int64_t)kv * P.rows + r) * ld + kk] = s[i];
        m[n][i & 1] = fmaxf(m[n][i & 1], s[i]);
      }
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int x = 4; x < 32; x <<= 1) m[n][j] = fmaxf(m[n][j], __shfl_xor_sync(0xffffffffu, m[n][j], x));
      const int r = r0 + 8 * n + 2 * tg + j;
      if (g == 0 && r < P.rows) P.tile_max[((int64_t)kv * P.rows + r) * P.Tk + tile] = m[n][j];
    }
}

// Key tiles from the last to the first, as in attn.cu; a warp takes `run` of them, a CTA 4 * run.
template <int D, int NT>
__global__ __launch_bounds__(kThreads) void decode_output_kernel(const DecodeParams P) {
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
    uint32_t p[NT][16];                                  // keys 32 tg ... + 31 of query g
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const bool live = 8 * n + g < nr;
      const int64_t row = row0 + 8 * n + g;
      float4 s[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float off = __uint_as_float(0xff800000u);
        s[i] = live ? *reinterpret_cast<const float4*>(P.scores + row * ld + tile * kTile + 32 * tg + 4 * i)
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
      expand_row<128>(raw_row<128>(vc, vs, 16 * mt + g, tg), v0);
      expand_row<128>(raw_row<128>(vc, vs, 16 * mt + g + 8, tg), v1);
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 8; ++j) mma16816(o[n][mt], v0[2 * j], v1[2 * j], v0[2 * j + 1], v1[2 * j + 1], p[n][2 * j], p[n][2 * j + 1]);
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
    if (t == 0) last_s = atomicAdd(P.counter + kv * gridDim.y + blockIdx.y, 1) == P.chunks - 1;
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
  const int groups = (P.rows + 8 * NT - 1) / (8 * NT), units = P.kvs * P.Tk;
  // runs: 16 warps per SM of a B200, at most kMaxChunks CTAs per kv head
  const int even = (int)(((int64_t)units * groups + 148 * 16 - 1) / (148 * 16)), most = (P.Tk + kWarps * kMaxChunks - 1) / (kWarps * kMaxChunks);
  P.run = even > most ? even : most;
  P.chunks = (P.Tk + kWarps * P.run - 1) / (kWarps * P.run);
  cudaError_t e = launch_pdl(decode_scores_kernel<D, NT>, dim3((unsigned)((units + kWarps - 1) / kWarps), groups), kThreads, 0, stream,
                             overlap, P);
  if (e != cudaSuccess) return e;
  return launch_pdl(decode_output_kernel<D, NT>, dim3((unsigned)(P.kvs * P.chunks), groups), kThreads, 0, stream, true, P);
}

}  // namespace

bool decode_fits(int Hq, int Hkv, int Nq, int Nk) {
  const int rows = Hq / Hkv * Nq;
  return Nk > 7 * kTile && rows <= 128 && (Nq <= 4 || rows <= 8);
}

size_t decode_scratch_bytes(int B, int Hq, int Hkv, int Nq, int Nk, int D) {
  if (!decode_fits(Hq, Hkv, Nq, Nk)) return 0;
  const size_t Tk = (Nk + kTile - 1) / kTile, rows = (size_t)B * Hq * Nq, chunks = Tk < kMaxChunks ? Tk : kMaxChunks;
  return align256(rows * Tk * kTile * 4) + align256(rows * Tk * 4) + align256(rows * chunks * D * 4) +
         2 * align256(rows * chunks * 4) + align256(rows * 4);
}

cudaError_t launch_attn_decode(const AttnArgs& a, void* scratch, cudaStream_t stream) {
  if ((a.D != 128 && a.D != 64) || !decode_fits(a.Hq, a.Hkv, a.Nq, a.Nk)) return cudaErrorInvalidValue;
  DecodeParams P;
  P.q_codes = (const uint8_t*)a.q_codes; P.q_sf = (const uint8_t*)a.q_sf; P.k_codes = (const uint8_t*)a.k_codes;
  P.k_sf = (const uint8_t*)a.k_sf; P.vt_codes = (const uint8_t*)a.vt_codes; P.vt_sf = (const uint8_t*)a.vt_sf;
  P.ds = (const __nv_bfloat16*)a.ds; P.out = (__nv_bfloat16*)a.out; P.lse = a.lse; P.lse_add = a.lse_add;
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
  if (a.D == 128) return P.rows <= 8 ? launch<128, 1>(P, a.after_delta_s, stream) : launch<128, 2>(P, a.after_delta_s, stream);
  return P.rows <= 8 ? launch<64, 1>(P, a.after_delta_s, stream) : launch<64, 2>(P, a.after_delta_s, stream);
}

}  // namespace sage3
