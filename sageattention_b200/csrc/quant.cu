// Fused smoothing + NVFP4 quantisation of Q, K and V for the FP4 attention kernel (sm_100a).
//
// Replaces, in one launch (the K channel means are added up from its partial sums by the next one, or, where the means
// themselves are asked for, come from a reduction launch before it):
//   * K minus its per-channel mean over tokens        sageattn4/api.py:184
//   * Q zero-padded to 128 rows, minus per-128-row mean sageattn4/api.py:26-72,186-191
//   * NVFP4 quantisation of Q                          quantization/fp4_quantization_4d.cu:164-284,414-490
//   * NVFP4 quantisation of K (the reference permutes rows for its mma.sync fragment layout,
//     :146-162; tensor memory accumulators make that unnecessary, rows stay in token order)
//   * transpose + NVFP4 quantisation of V along tokens :286-412,571-648
//
// The arithmetic per 16-element block is the reference's, instruction for instruction
// (common.cuh: block_scale, f32x8_to_e2m1x8), so codes and scale bytes are bit-identical.
//
// Memory plan (HBM-bound): every thread issues all of its 128-bit loads for a 128-token tile
// before the first use (a whole 32 KB tile in flight per CTA) and owns whole 16-element blocks, codes
// leave as full 32-byte sectors and the scale bytes are staged in shared memory so that they leave as
// 16-byte vectors in the exact order the attention kernel's tcgen05.cp expects.  What paces it is instructions
// (about half of the issue slots, at 4.6 TB/s) as much as memory: 13 per element of Q, 12 of V with its share of the K sums.
//
// Output layouts (per batch b, head h; Np = tokens padded to a multiple of 128, T = Np/128):
//   codes  Q,K : [T][128 rows][D/2] bytes            (row-major, element 2i in the low nibble)
//   scales Q,K : [T][D/64][512] bytes                (SF atom, sf_atom_offset())
//   codes  V^T : [T][D rows][64] bytes               (row d holds the tile's 128 tokens)
//   scales V^T : [T][2][512] bytes                   (atom rows = d, columns = 16-token blocks)
//   qm         : [T][D] bf16 block means of Q;  km : [D] bf16 channel means of K
#include "common.cuh"
#include "kernels.h"
#include "pack_group.cuh"
#include "quant_rows.cuh"
#include "quant_v.cuh"

namespace sage3 {

// ------------------------------------------------------------------------------------------------
// Channel sums over tokens (K channel mean; also the whole-sequence Q mean when per_block_mean=0): fp32 sums of one
// chunk of tokens -> one partial row [D].  Rows of a head are always added in chunk order, so the mean is deterministic
// and does not depend on who adds them (this file's mean kernel, or k_mean in quant_rows.cuh).
// ------------------------------------------------------------------------------------------------
template <int D, int U>                // U = passes in flight
__device__ __forceinline__ void channel_partial(const __nv_bfloat16* __restrict__ base, const int64_t sn, const int N,
                                                const int chunk, const int chunk_tokens, const int d_in,
                                                float* __restrict__ prow, float* red) {
  constexpr int CH = D / 8;              // 16-byte chunks per row
  constexpr int RPP = kThreads / CH;     // rows per pass
  const int t = threadIdx.x, c = t % CH, rl = t / CH;
  base += c * 8;
  const int n0 = chunk * chunk_tokens;
  const int n1 = min(N, n0 + chunk_tokens);
  float2 acc[4] = {};
  for (int n = n0 + rl; n < n1; n += RPP * U) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      int nn = n + u * RPP;
      v[u] = (nn < n1 && c * 8 < d_in) ? *reinterpret_cast<const uint4*>(base + (int64_t)nn * sn) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) add_channels(acc, v[u]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<float2*>(red + rl * D + c * 8 + 2 * i) = acc[i];
  __syncthreads();
  if (t < D) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < RPP; ++r) s += red[r * D + t];
    prow[t] = s;
  }
}

// The sums and the mean in one launch: grid = (chunks, B*H), the last CTA of a (b,h) to finish adds the partial rows
// and writes mean = sum / divisor as bf16.
// scratch: partial[B*H][chunks][D] fp32 followed by counters[B*H] u32 (zeroed by the host).
// Eight rows in flight per thread and four CTAs per SM: B1 H40 N9450 34.6 -> 27.2 us (four rows and eight CTAs before; sixteen and
// three 30.0).
template <int D>
__global__ void __launch_bounds__(kThreads, 4) channel_mean_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t sb, int64_t sh, int64_t sn, int H, int N,
    int chunk_tokens, float divisor, float* __restrict__ partial, unsigned int* __restrict__ counters,
    __nv_bfloat16* __restrict__ mean_out, const int* __restrict__ cu, int d_in) {
  __shared__ __align__(16) float red[(kThreads / (D / 8)) * D];
  __shared__ bool is_last;
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  const int chunk = blockIdx.x, nchunks = gridDim.x, t = threadIdx.x;
  // variable-length batch: sequence b starts at token cu[b] of the packed tensor and has its own length
  if (cu != nullptr) {
    N = min(cu[b + 1] - cu[b], N);         // never beyond the caller's max_seqlen (the grid covers no more)
    divisor = (float)max(N, 1);
  }
  channel_partial<D, 8>(x + (cu ? (int64_t)cu[b] * sn : b * sb) + h * sh, sn, N, chunk, chunk_tokens, d_in,
                     partial + ((int64_t)bh * nchunks + chunk) * D, red);
  __threadfence();
  __syncthreads();
  if (t == 0) is_last = (atomicAdd(&counters[bh], 1u) == (unsigned)(nchunks - 1));
  __syncthreads();
  if (is_last) {
    __threadfence();
    if (t < D) {
      const float* p = partial + (int64_t)bh * nchunks * D + t;
      float s = 0.f;
#pragma unroll 8
      for (int i = 0; i < nchunks; ++i) s += __ldcg(p + (int64_t)i * D);
      mean_out[(int64_t)bh * D + t] = __float2bfloat16_rn(s / divisor);
    }
    if (t == 0) counters[bh] = 0;        // leave the scratch clean for the next call
  }
}

// Channel sums of a Q tile: those of the warps' rows, red[warp][D].  The order is fixed - rows r, r + kStep, ... of the whole tile
// one after another, then r and r + 1 (D=64: then the same of r + 2 and r + 3), the warps last, by the caller - because a block mean
// that rounds the other way is seen in 128 rows of delta_s.  So the two lanes that have rows 0 ... 63 and 64 ... 127 of the same
// kind swap half of their channels, and each adds all rows of 8.  (Launch of B1 H40 N32760 / B4 H32/8 N8192 / 16 prompts 218.8 / 96.8 /
// 69.4 us; sums handed on, each lane adding twice: 223 / 99 / 72; swapped as sums are needed, twice the shuffles: 225 / 102 / 69; in
// any order: 218.5 / 96.5 / 66.6.)
template <int D>
__device__ __forceinline__ void tile_sums(const uint4 (&w)[RowTile<D, true>::kPasses][2], const int t, const int c, float* red) {
  constexpr int kPasses = RowTile<D, true>::kPasses;
  const bool second = (t & 16) != 0;
  float2 a[4] = {};
  uint4 got[kPasses];                            // the first lane's channels 0 ... 7 of the other half, the second's 8 ... 15
#pragma unroll
  for (int p = 0; p < kPasses; ++p) {
    const uint4 give = second ? w[p][0] : w[p][1];
    got[p].x = __shfl_xor_sync(0xffffffffu, give.x, 16); got[p].y = __shfl_xor_sync(0xffffffffu, give.y, 16);
    got[p].z = __shfl_xor_sync(0xffffffffu, give.z, 16); got[p].w = __shfl_xor_sync(0xffffffffu, give.w, 16);
    add_channels(a, second ? got[p] : w[p][0]);
  }
#pragma unroll
  for (int p = 0; p < kPasses; ++p) add_channels(a, second ? w[p][1] : got[p]);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) { acc[2 * j] = a[j].x; acc[2 * j + 1] = a[j].y; }
  int first = c * 16 + (second ? 8 : 0);
#pragma unroll
  for (int step = 0; step < (D == 128 ? 1 : 2); ++step) {        // each step of the exchange leaves a lane half its channels
    const int o = 4 << step, n = 4 >> step;      // the lane's bits that are the row
    const bool upper = (t & o) != 0;
#pragma unroll
    for (int j = 0; j < n; ++j) {
      const float give = upper ? acc[j] : acc[n + j], own = upper ? acc[n + j] : acc[j];
      acc[j] = own + __shfl_xor_sync(0xffffffffu, give, o);
    }
    if (upper) first += n;
  }
#pragma unroll
  for (int j = 0; j < (D == 128 ? 4 : 2); ++j) red[(t >> 5) * D + first + j] = acc[j];
}

// Division by a number that the host knows, for 0 <= n < 2^31 (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994): the six of a CTA's index arithmetic were 10 % of the Q role's instructions.
struct Div {
  uint32_t d, mul, shift;
  void set(uint32_t by) {
    d = by;
    for (shift = 0; (1ull << shift) < by; ++shift) {}
    mul = (uint32_t)(((1ull << 32) * ((1ull << shift) - by)) / by + 1);
  }
  __device__ __forceinline__ int quot(int n) const { return (int)((__umulhi(mul, (uint32_t)n) + (uint32_t)n) >> shift); }
  __device__ __forceinline__ void split(int n, int& q, int& r) const { q = quot(n); r = n - q * (int)d; }
};

struct QuantLaunch {
  const __nv_bfloat16 *q, *k, *v;
  int64_t q_sb, q_sh, q_sn, k_sb, k_sh, k_sn, v_sb, v_sh, v_sn;
  int B, Hq, Hkv, Nq, Nk, Tq, Tk;        // T* = number of 128-token tiles
  int q_mean_mode;                       // 0 none, 1 per 128-token block, 2 whole sequence (mean given)
  const __nv_bfloat16* km;               // [B,Hkv,D] K channel means
  const __nv_bfloat16* q_mean_seq;       // [B,Hq,D] (mode 2)
  const float* qm_override;              // optional fp32 block means [B,Hq,Tq,D] (mode 1)
  uint8_t *q_codes, *q_sf, *k_codes, *k_sf, *vt_codes, *vt_sf;
  __nv_bfloat16* qm;                     // [B,Hq,Tq,D] (mode 1)
  int q_blocks, k_blocks, v_blocks;      // CTAs per role
  Div by_Tq, by_Tk, by_Hq, by_Hkv, by_chunks;
  int q_heads;                           // kVar: heads that a CTA of the Q role takes; by_Hq then divides by their groups
  const int *cu_q, *cu_k;                // variable-length batches (else null)
  int d_in;                              // channels the input rows really have (<= D, multiple of 8); the rest are zero
  int s_blocks, chunks, chunk_tokens;    // CTAs of the K channel-sum role (0: none), chunks per head, tokens per chunk
  int s_first;                           // the first of them among the CTAs: 0, or all others before them
  float* partial;                        // [B,Hkv,chunks,D] fp32 K channel sums, written by that role
  int* zero_status;                      // status word of the whole operator call, zeroed here (optional)
  bool pack, split_first;                // K-packing mode: Nk tokens in Tk tiles of slots; V layout of its two variants
  int o_blocks, causal;                  // 1: the work-order role of a variable-length batch runs
  int *order, *n_order;                  // its result: (sequence, pair of query tiles) entries and their number
  float* q_dot_km;                       // optional fp32 [B,Hq,Nq]: raw q . K channel mean of the row's kv head
  const __nv_bfloat16* km_for_q;         //   (the term K smoothing removes from every score of the row)
};

// Work order of a variable-length batch for the attention kernel's static schedule: the pairs of query tiles that exist,
// by falling number of key tiles they visit, as sequence * pairs + pair.  One CTA, counting sort (costs above the table
// are scaled into it); the order within a bin is whatever the atomics make it, the results do not depend on it.
// Without it the schedule dealt out items as if every sequence were the longest: 16 causal sequences of 187 to 3000
// tokens, 32 heads, took 452 us.
constexpr int kOrderBins = 2048;
__device__ __forceinline__ void varlen_order(const QuantLaunch& P, int* hist) {
  const int t = threadIdx.x, n_pairs = (P.Tq + 1) >> 1, n = P.B * n_pairs;
  const int scale = (2 * P.Tk + kOrderBins) / kOrderBins;       // costs 0 ... 2 Tk
  auto bin_of = [&](const int e) {                              // heaviest in bin 0; -1: no such query tiles
    const int b = e / n_pairs, q0 = (e % n_pairs) * 2 * kTile;
    const int nq = min(P.cu_q[b + 1] - P.cu_q[b], P.Nq), nk = min(P.cu_k[b + 1] - P.cu_k[b], P.Nk);
    if (q0 >= nq) return -1;
    int cost = 0;
    for (int s = 0; s < 2; ++s) {
      const int end = min(q0 + (s + 1) * kTile, nq);
      if (q0 + s * kTile >= nq) break;
      const int keys = P.causal ? min(nk, end + nk - nq) : nk;
      cost += keys <= 0 ? 0 : (keys + kTile - 1) / kTile;
    }
    return kOrderBins - 1 - cost / scale;
  };
  for (int i = t; i < kOrderBins; i += kThreads) hist[i] = 0;
  __syncthreads();
  for (int e = t; e < n; e += kThreads) {
    const int bin = bin_of(e);
    if (bin >= 0) atomicAdd(&hist[bin], 1);
  }
  __syncthreads();
  if (t < 32) {                                                 // exclusive prefix sum by one warp
    int base = 0;
    for (int i = t; i < kOrderBins; i += 32) {
      const int v = hist[i];
      int x = v;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (t >= o) x += y;
      }
      hist[i] = base + x - v;
      base += __shfl_sync(0xffffffffu, x, 31);
    }
    if (t == 0) *P.n_order = base;
  }
  __syncthreads();
  for (int e = t; e < n; e += kThreads) {
    const int bin = bin_of(e);
    if (bin >= 0) P.order[atomicAdd(&hist[bin], 1)] = e;
  }
}

// 64 registers: four CTAs per SM, each with a whole 32 KB tile in flight (B1 H40 N32760 D128, with the K sums: 219 us, 229 at three
// per SM; B4 H32/8 N8192 96, 105)
// kVar: variable-length batches, whose grid is sized for sequences of the greatest length.  A CTA of the Q role then takes its tile of
// up to four heads, so that there are a quarter of the CTAs for tiles that no sequence has, and one of the V role leaves at once
// (16 prompts of 187 to 3000 tokens, H32/8: 77.7 -> 66.5 us; operator with 31 prompts of 600 and 8000, D=64: 687 -> 650, with eight
// of 2000 each: 304 -> 299).
template <int D, bool kVar>
__global__ void __launch_bounds__(kThreads, 4) quant_qkv_kernel(const QuantLaunch P) {
  using R = RowTile<D, true>;
  __shared__ __align__(16) uint8_t sf_smem[2048];
  __shared__ __align__(16) float red[kThreads / (D / 8) * D];    // (what the K channel sums need; the Q means less)
  __shared__ __align__(16) float mean_s[D + D / 8];              // four words further every 32 channels, for the banks
  const int t = threadIdx.x, c = R::block(t), rl = R::row(t);
  int bid = blockIdx.x;
  pdl_launch_dependents();                 // the K kernel may come in and fetch its tiles as SMs fall idle
  if (bid == 0 && t == 0 && P.zero_status != nullptr) *P.zero_status = 0;

  if (bid < P.o_blocks) {
    static_assert(sizeof(red) >= kOrderBins * sizeof(int), "histogram");
    varlen_order(P, reinterpret_cast<int*>(red));
    return;
  }
  bid -= P.o_blocks;
  if (bid >= P.s_first && bid < P.s_first + P.s_blocks) {
    // ----------------------------------------------------------------------------- K channel-sum role
    bid -= P.s_first;
    int chunk, bh, b, h;
    P.by_chunks.split(bid, bh, chunk);
    P.by_Hkv.split(bh, b, h);
    const int N = P.cu_k ? min(P.cu_k[b + 1] - P.cu_k[b], P.Nk) : P.Nk;
    channel_partial<D, 8>(P.k + (P.cu_k ? (int64_t)P.cu_k[b] * P.k_sn : b * P.k_sb) + h * P.k_sh, P.k_sn, N, chunk, P.chunk_tokens,
                       P.d_in, P.partial + (int64_t)bid * D, red);
    return;
  }
  if (P.s_first == 0) bid -= P.s_blocks;

  if (bid < P.q_blocks + P.k_blocks) {
    // ----------------------------------------------------------------------------- Q / K roles
    const bool is_q = bid < P.q_blocks;
    if (!is_q) bid -= P.q_blocks;
    const int T = is_q ? P.Tq : P.Tk;
    int tile, bh, b, h;
    (is_q ? P.by_Tq : P.by_Tk).split(bid, bh, tile);
    (is_q ? P.by_Hq : P.by_Hkv).split(bh, b, h);
    const int heads = kVar && is_q ? P.q_heads : 1;
    if (kVar && is_q) { h *= heads; bh = b * P.Hq + h; }
#pragma unroll 1
    for (int i_head = 0; i_head < (kVar ? heads : 1); ++i_head, ++h, ++bh) {
    int N = is_q ? P.Nq : P.Nk;
    if (kVar && i_head > 0) __syncthreads();   // shared memory of the head before has been read
    const int64_t sn = is_q ? P.q_sn : P.k_sn;
    const int* cu = is_q ? P.cu_q : P.cu_k;
    const __nv_bfloat16* src = is_q ? P.q + b * P.q_sb + h * P.q_sh : P.k + b * P.k_sb + h * P.k_sh;
    if (cu != nullptr) {                   // sequence b of a packed [tokens, H, D] tensor
      N = min(cu[b + 1] - cu[b], N);       // cut at max_seqlen, which sizes the output layouts
      src = (is_q ? P.q + h * P.q_sh : P.k + h * P.k_sh) + (int64_t)cu[b] * sn;
      if (is_q && tile * kTile >= N) {     // beyond the sequence: only the block mean is read (for delta_s rows that no
        if (P.q_mean_mode == 1 && rl == 0)  //   query uses), so it must at least be a number
          for (int i = 0; i < 2; ++i)
            reinterpret_cast<uint4*>(P.qm + ((int64_t)bh * T + tile) * D + c * 16)[i] = make_uint4(0, 0, 0, 0);
        continue;
      }
    }
    uint4 w[R::kPasses][2];
    src += (int64_t)(tile * kTile + rl) * sn + c * 16;
    const int rows = N - tile * kTile - rl;      // this thread's rows are there below it
#pragma unroll
    for (int p = 0; p < R::kPasses; ++p) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        w[p][i] = (p * R::kStep < rows && c * 16 + 8 * i < P.d_in) ? *reinterpret_cast<const uint4*>(src + 8 * i) : make_uint4(0, 0, 0, 0);
      src += R::kStep * sn;
    }
    float mean[16];
    if (is_q && P.q_dot_km != nullptr) {
      // q . km in fp32 from the raw rows: what K smoothing took out of every score of the row; the attention
      // kernel adds sm_scale times it to the log-sum-exp (the pattern of sageattention/core.py:993-994)
      bf16x16_to_f32(P.km_for_q + ((int64_t)b * P.Hkv + h / (P.Hq / P.Hkv)) * D + c * 16, mean);
#pragma unroll
      for (int p = 0; p < R::kPasses; ++p) {
        float d8[2];                             // of 8 channels each, then of more and more: an order that the LSE's last bits show
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 x = w[p][i];
          const float* m = mean + 8 * i;
          float d = bf16_lo(x.x) * m[0];
          d = fmaf(bf16_hi(x.x), m[1], d); d = fmaf(bf16_lo(x.y), m[2], d); d = fmaf(bf16_hi(x.y), m[3], d);
          d = fmaf(bf16_lo(x.z), m[4], d); d = fmaf(bf16_hi(x.z), m[5], d); d = fmaf(bf16_lo(x.w), m[6], d);
          d8[i] = fmaf(bf16_hi(x.w), m[7], d);
        }
        float d = d8[0] + d8[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
          if (o & R::kBlockBits) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (c == 0 && p * R::kStep < rows) P.q_dot_km[(int64_t)bh * P.Nq + tile * kTile + p * R::kStep + rl] = d;
      }
    }
    bool subtract = true;
    if (is_q && P.q_mean_mode == 1) {
      if (P.qm_override != nullptr) {
        const float* mp = P.qm_override + ((int64_t)bh * T + tile) * D + c * 16;
#pragma unroll
        for (int i = 0; i < 16; ++i) mean[i] = mp[i];
      } else {
        // fp32 column sums over the tile's 128 rows (zero rows of the padding included), / 128
        tile_sums<D>(w, t, c, red);
        __syncthreads();
        if (t < D) {
          float s = 0.f;
#pragma unroll
          for (int r = 0; r < kThreads / 32; ++r) s += red[r * D + t];
          mean_s[t + (t >> 5) * 4] = s * (1.0f / kTile);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) mean[i] = mean_s[c * 16 + (c >> 1) * 4 + i];
      }
      if (rl == 0) {   // bf16 block mean, consumed by the delta_s kernel
#pragma unroll
        for (int i = 0; i < 2; ++i)
          reinterpret_cast<uint4*>(P.qm + ((int64_t)bh * T + tile) * D + c * 16)[i] =
              make_uint4(pack_bf16(mean[8 * i], mean[8 * i + 1]), pack_bf16(mean[8 * i + 2], mean[8 * i + 3]),
                         pack_bf16(mean[8 * i + 4], mean[8 * i + 5]), pack_bf16(mean[8 * i + 6], mean[8 * i + 7]));
      }
    } else if (is_q && P.q_mean_mode == 2) {
      bf16x16_to_f32(P.q_mean_seq + (int64_t)bh * D + c * 16, mean);
    } else if (!is_q && P.km != nullptr) {
      bf16x16_to_f32(P.km + (int64_t)bh * D + c * 16, mean);
    } else {
      subtract = false;
    }
    if (subtract) {
      // x - mean in fp32, rounded to bf16 (what a bf16 tensor subtraction does).  Q: padding rows
      // become -mean like the reference (it pads before subtracting); K: padding rows stay zero
      // (the reference subtracts before padding).
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 neg[4] = {{-mean[8 * i], -mean[8 * i + 1]}, {-mean[8 * i + 2], -mean[8 * i + 3]},
                               {-mean[8 * i + 4], -mean[8 * i + 5]}, {-mean[8 * i + 6], -mean[8 * i + 7]}};
#pragma unroll
        for (int p = 0; p < R::kPasses; ++p)
          if (is_q || p * R::kStep < rows) w[p][i] = subtract_mean(w[p][i], neg);
      }
    }
    uint8_t* codes = (is_q ? P.q_codes : P.k_codes) + ((int64_t)bh * T + tile) * (kTile * D / 2);
    uint8_t* sf = (is_q ? P.q_sf : P.k_sf) + ((int64_t)bh * T + tile) * ((D / 64) * 512);
    quant_rows_store<D, true>(w, codes, sf, sf_smem);
    }
    return;
  }

  // ------------------------------------------------------------------------------------- V role
  // One warp = 4 groups of 4 channels x the 8 token blocks of a tile; a thread loads 16 tokens x
  // 4 channels (8-byte loads; a warp load touches 8 rows x one full 32-byte sector) and emits,
  // per channel, 8 bytes of codes + 1 scale.  Eight lanes with the same channel write one
  // contiguous 64-byte row of the V^T tile.
  bid -= P.q_blocks + P.k_blocks;
  constexpr int WPT = D / 16;                    // warps per tile
  constexpr int TPB = (kThreads / 32) / WPT;     // tiles per CTA (1 for D=128, 2 for D=64)
  const int warp = t >> 5, lane = t & 31;
  const int tl = warp / WPT;                     // tile slot inside this CTA
  const int gt = bid * TPB + tl;                 // global tile index over (b, h, tile)
  const int total = P.B * P.Hkv * P.Tk;
  int tile, bh, b, h;
  P.by_Tk.split(gt, bh, tile);
  P.by_Hkv.split(bh, b, h);
  const int Nv = P.cu_k && gt < total ? min(P.cu_k[b + 1] - P.cu_k[b], P.Nk) : P.Nk;
  if (kVar && TPB == 1 && tile * kTile >= Nv) return;     // (nothing reads a V tile beyond its sequence)
  for (int i = t; i < 2048 / 16; i += kThreads) reinterpret_cast<uint4*>(sf_smem)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  if (gt < total && (P.pack || tile * kTile < Nv)) {      // (nothing reads a V tile beyond its sequence)
    const int c4 = (warp % WPT) * 4 + (lane >> 3);        // group of 4 channels
    const int blk = lane & 7;                              // 16-token block
    // K-packing mode: a block is a group, 15 tokens behind an empty slot
    const int n0 = P.pack ? (tile * 8 + blk) * kGroup - 1 : tile * kTile + blk * 16;
    const __nv_bfloat16* src = P.v + (P.cu_k ? (int64_t)P.cu_k[b] * P.v_sn : b * P.v_sb) + h * P.v_sh + c4 * 4 + (int64_t)n0 * P.v_sn;
    const int lim = c4 * 4 < P.d_in ? Nv - n0 : 0;         // slots of the block that there are
    uint2 x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      x[i] = (i < lim && !(i == 0 && P.pack)) ? __ldcs(reinterpret_cast<const uint2*>(src)) : make_uint2(0, 0);
      src += P.v_sn;
    }
    uint8_t* codes = P.vt_codes + (int64_t)gt * (D * 64);
    quant_v_block(x, c4 * 4, blk, P.split_first, codes, sf_smem + tl * 1024);
  }
  __syncthreads();
  // each tile's 1 KB of scales leaves as 64 x 16 bytes
  {
    const int slot = t / 64, vec = t % 64;
    const int g2 = bid * TPB + slot;
    if (slot < TPB && g2 < total)
      reinterpret_cast<uint4*>(P.vt_sf + (int64_t)g2 * 1024)[vec] = reinterpret_cast<const uint4*>(sf_smem + slot * 1024)[vec];
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
static int pick_chunk_tokens(int N, int BH) {
  // enough CTAs (8 per SM on 148 SMs) to keep the memory system full, but at most 64 partial rows per (b,h)
  int chunk = 4096;
  while (chunk > 256 && (int64_t)BH * ((N + chunk - 1) / chunk) < 1184) chunk >>= 1;
  while ((N + chunk - 1) / chunk > kMaxChunks) chunk <<= 1;
  return chunk;
}

size_t quant_scratch_bytes(int B, int H, int N, int D) {
  int chunk = pick_chunk_tokens(N, B * H);
  int nchunks = (N + chunk - 1) / chunk;
  size_t part = (size_t)B * H * nchunks * D * sizeof(float);
  part = (part + 255) & ~(size_t)255;
  return part + (size_t)B * H * sizeof(unsigned int);
}

cudaError_t launch_channel_mean(const void* x, int64_t sb, int64_t sh, int64_t sn, int B, int H, int N, int D,
                                float divisor, void* scratch, void* mean_out, cudaStream_t stream, const int* cu,
                                int d_in) {
  if (d_in <= 0 || d_in > D) d_in = D;
  int chunk = pick_chunk_tokens(N, B * H);
  int nchunks = (N + chunk - 1) / chunk;
  size_t part = (size_t)B * H * nchunks * D * sizeof(float);
  part = (part + 255) & ~(size_t)255;
  float* partial = reinterpret_cast<float*>(scratch);
  unsigned int* counters = reinterpret_cast<unsigned int*>(reinterpret_cast<char*>(scratch) + part);
  cudaError_t e = cudaMemsetAsync(counters, 0, (size_t)B * H * sizeof(unsigned int), stream);
  if (e != cudaSuccess) return e;
  dim3 grid(nchunks, B * H);
  if (D == 128)
    channel_mean_kernel<128><<<grid, kThreads, 0, stream>>>((const __nv_bfloat16*)x, sb, sh, sn, H, N, chunk, divisor,
                                                            partial, counters, (__nv_bfloat16*)mean_out, cu, d_in);
  else
    channel_mean_kernel<64><<<grid, kThreads, 0, stream>>>((const __nv_bfloat16*)x, sb, sh, sn, H, N, chunk, divisor,
                                                           partial, counters, (__nv_bfloat16*)mean_out, cu, d_in);
  return cudaGetLastError();
}

void quant_chunks(int BH, int N, int* chunks, int* chunk_tokens) {
  *chunk_tokens = pick_chunk_tokens(N, BH);
  *chunks = (N + *chunk_tokens - 1) / *chunk_tokens;
}

// Fewest CTAs of the Q role of a variable-length batch that sharing one among heads may leave: two waves of four CTAs on each of 148
// SMs.  (Below, a chain of four heads is what counts: two prompts of 64 and 30 tokens 15.7 us, 19.0 with four heads to a CTA.)
constexpr int64_t kVarCtas = 1184;

cudaError_t launch_quant_qkv(const QuantArgs& a, cudaStream_t stream) {
  QuantLaunch P;
  P.q = (const __nv_bfloat16*)a.q; P.k = (const __nv_bfloat16*)a.k; P.v = (const __nv_bfloat16*)a.v;
  P.q_sb = a.q_sb; P.q_sh = a.q_sh; P.q_sn = a.q_sn;
  P.k_sb = a.k_sb; P.k_sh = a.k_sh; P.k_sn = a.k_sn;
  P.v_sb = a.v_sb; P.v_sh = a.v_sh; P.v_sn = a.v_sn;
  P.B = a.B; P.Hq = a.Hq; P.Hkv = a.Hkv; P.Nq = a.Nq; P.Nk = a.Nk;
  P.Tq = (a.Nq + kTile - 1) / kTile; P.pack = a.pack; P.split_first = a.pack && a.split_first;
  P.Tk = ((a.pack ? (a.Nk + kGroup - 1) / kGroup * 16 : a.Nk) + kTile - 1) / kTile;
  P.q_mean_mode = a.q_mean_mode;
  P.km = (const __nv_bfloat16*)a.km; P.q_mean_seq = (const __nv_bfloat16*)a.q_mean_seq;
  P.qm_override = (const float*)a.qm_override;
  P.q_codes = (uint8_t*)a.q_codes; P.q_sf = (uint8_t*)a.q_sf;
  P.k_codes = (uint8_t*)a.k_codes; P.k_sf = (uint8_t*)a.k_sf;
  P.vt_codes = (uint8_t*)a.vt_codes; P.vt_sf = (uint8_t*)a.vt_sf;
  P.qm = (__nv_bfloat16*)a.qm;
  P.cu_q = a.cu_q; P.cu_k = a.cu_k;
  P.d_in = (a.d_in > 0 && a.d_in <= a.D) ? a.d_in : a.D;
  P.partial = (float*)a.partial;
  P.zero_status = a.zero_status;
  quant_chunks(a.B * a.Hkv, a.Nk, &P.chunks, &P.chunk_tokens);
  P.s_blocks = a.partial != nullptr ? a.B * a.Hkv * P.chunks : 0;
  P.q_dot_km = (a.q_dot_km != nullptr && a.km != nullptr && a.cu_q == nullptr) ? (float*)a.q_dot_km : nullptr;
  P.km_for_q = (const __nv_bfloat16*)a.km;
  const bool var = a.cu_q != nullptr || a.cu_k != nullptr;
  P.q_heads = !var ? 1 : (a.Hq % 4 == 0 ? 4 : (a.Hq % 2 == 0 ? 2 : 1));
  while (P.q_heads > 1 && (int64_t)a.B * (a.Hq / P.q_heads) * P.Tq < kVarCtas) P.q_heads >>= 1;
  P.q_blocks = a.q ? a.B * (a.Hq / P.q_heads) * P.Tq : 0;
  P.k_blocks = a.k && a.k_codes ? a.B * a.Hkv * P.Tk : 0;
  const int tpb = a.D == 128 ? 1 : 2;
  P.v_blocks = a.v ? (int)(((int64_t)a.B * a.Hkv * P.Tk + tpb - 1) / tpb) : 0;
  // K sums come last where K fits in L2, so that the K kernel finds it there (with V read past the L2's favour: K-packing
  // B4 H32 N2048 325 -> 320 us, 16 prompts 490 -> 486); else first, being the longest units (B1 H40 N32760 loses 10 us else),
  // as where K is so small that it is in L2 anyhow.  Of a variable-length batch the padded size counts: last, the sums also wait
  // for the CTAs of tiles beyond the sequences (by the keys there really are, 73 MB of 688: 2162 -> 2186 us, 53 MB of 999: 1110 ->
  // 1140)
  const int64_t k_bytes = (int64_t)a.B * a.Hkv * a.Nk * a.D * 2;
  const bool fits = k_bytes <= 96 << 20 && k_bytes >= 8 << 20;
  P.s_first = fits ? P.q_blocks + P.k_blocks + P.v_blocks : 0;
  P.by_Tq.set(P.Tq > 0 ? P.Tq : 1); P.by_Tk.set(P.Tk > 0 ? P.Tk : 1); P.by_Hq.set(a.Hq / P.q_heads); P.by_Hkv.set(a.Hkv); P.by_chunks.set(P.chunks > 0 ? P.chunks : 1);
  P.order = a.order; P.n_order = a.n_order; P.causal = a.causal;
  P.o_blocks = a.order != nullptr ? 1 : 0;
  const int grid = P.o_blocks + P.s_blocks + P.q_blocks + P.k_blocks + P.v_blocks;
  if (grid == 0) return cudaSuccess;
  if (var) {
    if (a.D == 128) quant_qkv_kernel<128, true><<<grid, kThreads, 0, stream>>>(P);
    else            quant_qkv_kernel<64, true><<<grid, kThreads, 0, stream>>>(P);
  } else {
    if (a.D == 128) quant_qkv_kernel<128, false><<<grid, kThreads, 0, stream>>>(P);
    else            quant_qkv_kernel<64, false><<<grid, kThreads, 0, stream>>>(P);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Channel means with the reduction scratch inside the library.
//
// Some hosts of this library may not call cudaMalloc at the point where they need the K means: an
// inference server that handed all device memory to its own pool at start-up, or a plug-in hook that
// runs where an allocation (which synchronises the device and can fail under memory pressure) is not
// acceptable.  For them the partial sums and arrival counters of channel_mean_kernel live in the
// fixed array below instead of a caller buffer.  Every GPU that loads the library holds the array
// (1 MiB + 8 KiB) until the process exits.
//
// In host code `g_static_scratch` is only a handle for the symbol, not a device address; the address
// on the current device comes from cudaGetSymbolAddress, once per device, on the first call made
// with that device current.
// ------------------------------------------------------------------------------------------------
constexpr int kStaticMaxRows = 2048;                                   // partial rows: B * H * chunks
constexpr int kStaticMaxHeads = 2048;                                  // arrival counters: B * H
constexpr size_t kStaticPartialBytes = (size_t)kStaticMaxRows * 128 * sizeof(float);
static __device__ __align__(256) unsigned char g_static_scratch[kStaticPartialBytes + kStaticMaxHeads * sizeof(unsigned int)];

cudaError_t launch_channel_mean_static(const void* x, int64_t sb, int64_t sh, int64_t sn, int B, int H, int N, int D,
                                       float divisor, void* mean_out, cudaStream_t stream, bool* too_large) {
  *too_large = false;
  const int chunk = pick_chunk_tokens(N, B * H);
  const int nchunks = (N + chunk - 1) / chunk;
  if ((int64_t)B * H * nchunks > kStaticMaxRows || (int64_t)B * H > kStaticMaxHeads) {
    *too_large = true;
    return cudaSuccess;
  }
  static void* base_of_device[64] = {};                                // device ordinal -> address of the array there
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  void* base = __atomic_load_n(&base_of_device[dev], __ATOMIC_ACQUIRE);
  if (base == nullptr) {
    e = cudaGetSymbolAddress(&base, g_static_scratch);
    if (e != cudaSuccess) return e;
    __atomic_store_n(&base_of_device[dev], base, __ATOMIC_RELEASE);    // same value whoever stores first
  }
  float* partial = reinterpret_cast<float*>(base);
  unsigned int* counters = reinterpret_cast<unsigned int*>(reinterpret_cast<char*>(base) + kStaticPartialBytes);
  // The array keeps whatever the previous call left.  Partial rows are fully overwritten before they
  // are read; only the arrival counters must start at zero.
  e = cudaMemsetAsync(counters, 0, (size_t)B * H * sizeof(unsigned int), stream);
  if (e != cudaSuccess) return e;
  dim3 grid(nchunks, B * H);
  if (D == 128)
    channel_mean_kernel<128><<<grid, kThreads, 0, stream>>>((const __nv_bfloat16*)x, sb, sh, sn, H, N, chunk, divisor,
                                                            partial, counters, (__nv_bfloat16*)mean_out, nullptr, D);
  else
    channel_mean_kernel<64><<<grid, kThreads, 0, stream>>>((const __nv_bfloat16*)x, sb, sh, sn, H, N, chunk, divisor,
                                                           partial, counters, (__nv_bfloat16*)mean_out, nullptr, D);
  return cudaGetLastError();
}

}  // namespace sage3
