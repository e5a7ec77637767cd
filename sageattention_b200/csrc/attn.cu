// FP4 (NVFP4 block-scaled) flash-attention forward for B200 (sm_100a): TMA -> shared memory ->
// tcgen05.mma kind::mxf4nvf4 with accumulators in tensor memory -> online softmax in registers
// with two-level FP4 re-quantisation of P -> second block-scaled MMA for P.V, accumulated in tensor memory.
//
// Replaces the reference's sm_120-only mma.sync kernel (sageattn4/blackwell/fwd_kernel.cu:45-200,
// fwd_mainloop.cu:639-1125, softmax_fused.h:39-187, fwd_epilogue.cu:30-183) and its host launcher
// (fwd_kernel.cu:202-293).  Arithmetic follows the reference step by step:
//   S = delta_s + Q^ K^T                              fwd_mainloop.cu:766-794, 908-919
//   masks (key padding, bottom-right causal)          fwd_mainloop.cu:921-964
//   online softmax, per-16-key scale = blockmax/6 stored as E4M3, P/scale stored as E2M1
//                                                     softmax_fused.h:107-153, fwd_mainloop.cu:967-1002
//   O = sum over key tiles of P^ V^, rescaled when the row maximum moves     softmax_fused.h:175-187
//   O /= l, bf16                                      softmax_fused.h:156-173, fwd_epilogue.cu:103-147
// Key tiles are visited from the last to the first as the reference does (fwd_mainloop.cu:575).
//
// O lives in tensor memory and the P.V MMAs accumulate into it (the reference keeps O in registers and adds a
// fresh product per key tile); like the reference it is multiplied by 2^((m_old - m_new) c) whenever a row's
// maximum has moved - here in place in tensor memory, and only by the warps in which some row's maximum did move.
// P, its block scales and the row sum are the reference's value for value.
//
// One persistent CTA per SM walks a static list of work items (round r: item r*grid + i, odd rounds in
// reverse CTA order; causal items sorted by falling cost over all heads, those of variable-length batches by an order that
// the quantisation kernel made);
// an item is TWO adjacent 128-row query tiles of one head, which share every K / V tile.  All
// barrier phases keep counting across items, so the loads, the first Q.K^T and the first softmax of the next item are
// under way while the output of the current one is stored.  16 warps:
//   warps 0-3   softmax warpgroup of query tile 0: thread r owns score row r (tensor-memory lane r).  Per key
//               tile it copies its 128 scores from tensor memory into registers and releases the score buffer at
//               once (the Q.K^T of the other query tile is issued into it while this tile is worked on), then:
//               16-key block maxima, block scales, exponentials, E2M1 codes of P^ into tensor memory (the P.V MMA
//               takes its A operand from there; only the block scales go through shared memory).
//   warps 4-7   the same for query tile 1
//   warps 8-11  O: rescale it between two P.V MMAs where a row maximum moved, and at the end of an item write O / l as
//               bf16 (D=128: through a swizzled staging tile and TMA stores).  One warp per 32 rows, for both query
//               tiles in turn
//   warp  12    TMA producer (Q tiles per item, then a ring of K and V stages; scale factors and the
//               delta_s rows by plain bulk copies)
//   warp  13    QK issuer: scale-factor copies, rank-1 delta_s MMA and Q.K^T MMAs, both tiles in turn
//               into the ONE score buffer (D=64: one for each)
//   warp  14    turns each delta_s row (128 bf16) into the B operand of a rank-1 bf16 MMA
//               (ones x delta_s) that initialises the score accumulator, so the softmax warps never
//               touch delta_s
//   warp  15    PV issuer: scale-factor copies and P.V MMAs, O_t += P^_t V^
//
// What bounds it: the softmax warps' own instruction stream.  Two of them share a sub-partition (a score row in
// registers leaves room for no more), so whatever one waits for is idle time unless the other happens to be in its
// exponentials.  Hence: everything that is not softmax - the rescaling, the output - is other warps' work
// (B4 Hq32 Hkv8 N8192 D128 causal: 1.79 -> 1.61 ms; B4 H32 N4096 D64: 0.815 -> 0.79 ms); all 32 lanes of a role warp
// wait and one issues, because a wait executed by a single lane polls instead of parking and answers 40 cycles later;
// the poll loop is a handful of instructions in one asm block (left to the compiler it was unrolled at every wait) and uniform by
// a vote; 3 of 16 exponentials run on the FMA pipe, which takes the special-function unit from 1100 to 900 cycles per key tile (by
// count, at 16 a clock).
// A look at a barrier takes 150 to 200 cycles even where the phase is long complete, since it queues behind the other warp's
// exponentials, and so do the other hand-overs of a key tile (clock stamps).  So those of the softmax lie behind one another no
// more than they must: the next scores' barrier is looked at in the last exponentials, that of the last P.V before the first
// exponentials, whose codes wait in registers, and P^ is handed over while the next scores are on their way.  With it and with
// loops that are not unrolled in the issuers: B1 H10 N32760 D128 3.67 -> 3.47 ms (whole operator; by now 3.41), D64 3.59 -> 3.33
// (3.27), B4 H32/8 N8192 causal 1.66 -> 1.59 (1.56), 16 prompts 435 -> 408 us (376).  The arithmetic of the softmax alone, two warps
// per sub-partition with every barrier satisfied, took 1170 to 1250 cycles per key tile and 128 query rows in two measurements;
// the kernel takes 1410 (its time over the 35 rounds of B1 H40 N32760), and took 1530 before.
//
// Tensor memory (512 columns): O0 [0,D) O1 [D,2D) S [2D,2D+128) (D=64: one for each query tile, [2D,2D+256)); 56 columns of scale
// factors, P^0 and P^1 (16 columns each: 128 FP4 codes per row).
//
// Every wait on an mbarrier is bounded; if one gives up the CTA records its code in *status, waits
// (bounded) for its own copies and MMAs in flight, frees its tensor memory and returns.  The codes, one for each wait:
//   TMA producer 10 K stage free, 11 V stage free, 12 Q slot free; QK issuer 20 Q tile there, 21 K stage there, 23 score buffer
//   free, 25 delta_s operand there; PV issuer 24 V stage there, 26 P^ there; softmax 30 scores there, 31 last P.V done;
//   O 32 alpha there, 33 row sum there, 34 last P.V done; delta_s 40 K stage there
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "tensor_map.h"

// This file is compiled twice: as it is for dense batches, and once more through attn_varlen.cu with
// SAGE3_VARLEN_BUILD = 1 for variable-length batches (per-sequence offsets and lengths from cu_seqlens).  The
// dense build sees exactly the code it had before the second one existed: the kernel is paced by its softmax
// warps and even dead extra code moved their register allocation and timing by a few percent.
#ifndef SAGE3_VARLEN_BUILD
#define SAGE3_VARLEN_BUILD 0
#endif
// lengths of the sequence a work item `wk` belongs to, inside the softmax warps
#if SAGE3_VARLEN_BUILD
#define SEQ_NQ wk.Nq
#define SEQ_NK wk.Nk
#define SEQ_NK_LOG wk.Nk
#define SEQ_TILE_EXISTS (q0 < wk.Nq)
#else
#define SEQ_NQ P.Nq
#define SEQ_NK P.Nk
#define SEQ_NK_LOG P.Nk_log
#define SEQ_TILE_EXISTS (qt < P.Tq)
#endif

namespace sage3 {

namespace {

constexpr int kBlockM = 128;
constexpr int kBlockN = 128;
constexpr int kStages = 3;                              // K / V ring depth (4 and 5 measured the same or 1 % slower)
constexpr int kAttnThreads = 512;
// Register hand-over (setmaxnreg) moves registers inside the pool the CTA was LAUNCHED with; a request beyond
// it would block forever, so the split is checked here.  kLaunchRegs is what the compiler allocates under
// __launch_bounds__(512, 1).
constexpr int kLaunchRegs = 128;
struct RegSplit { static constexpr int softmax = 192, corr = 72, role = 56; };
static_assert(256 * RegSplit::softmax + 128 * (RegSplit::corr + RegSplit::role) <= kAttnThreads * kLaunchRegs,
              "setmaxnreg split exceeds the CTA's register pool");

template <int D>
struct Smem {
  static constexpr int kQBytes = kBlockM * D / 2;
  static constexpr int kKBytes = kBlockN * D / 2;
  static constexpr int kVBytes = D * kBlockN / 2;
  static constexpr int kSfRow = (D / 64) * 512;          // Q / K scales per tile
  static constexpr int kSfV = 1024;                       // V^T scales per tile
  static constexpr int q = 0;                             // [2]
  static constexpr int k = q + 2 * kQBytes;               // [kStages]
  static constexpr int v = k + kStages * kKBytes;         // [kStages]
  static constexpr int sfq = v + kStages * kVBytes;       // [2][1024]
  static constexpr int sfk = sfq + 2 * 1024;              // [kStages][1024]
  static constexpr int sfv = sfk + kStages * 1024;        // [kStages][1024]
  static constexpr int sfp = sfv + kStages * 1024;        // [2][1024]
  static constexpr int a1 = sfp + 2 * 1024;               // rank-1 A operand: column 0 = 1.0 (bf16)
  static constexpr int b1 = a1 + 2048;                    // [kStages][2][2048] rank-1 B operands
  static constexpr int zero = b1 + kStages * 2 * 2048;    // second K chunk of every rank-1 operand; it must lie
                                                          // ABOVE them: the descriptor offset to it is unsigned
  static constexpr int dsraw = zero + 2048;               // [kStages][2][256] delta_s rows as loaded
  static constexpr int lam = dsraw + kStages * 2 * 256;   // [2 * kStages][128] f32: lambda of the key slots (K-packing
                                                          // mode), arrives with the K stage; twice as many slots as
                                                          // stages because the softmax reads it after the stage is freed
  static constexpr int alpha = lam + 2 * kStages * 512;   // [2 query tiles][128] f32: factor of O where the row maximum moved
  static constexpr int lx = alpha + 1024;                 // [2 items][2 query tiles][l, m][128] f32
  static constexpr int bars = lx + 4096;
  // output staging for the TMA store: [2 tiles][4 warps][D/64 column halves][32 rows x 128 bytes], 128-byte swizzle
  static constexpr int kOStage = 32 * 128;
  static constexpr int ostage = (bars + 512 + 1023) / 1024 * 1024;
  static constexpr int total = ostage + ((!SAGE3_VARLEN_BUILD && D == 128) ? 8 * (D / 64) * kOStage : 0);
};

struct Bars {            // byte offsets inside the barrier block
  static constexpr int q_full = 0;                        // [2]
  static constexpr int q_empty = 16;                      // [2]
  static constexpr int k_full = 32;                       // [kStages]
  static constexpr int k_empty = k_full + 8 * kStages;
  static constexpr int v_full = k_empty + 8 * kStages;
  static constexpr int v_empty = v_full + 8 * kStages;
  static constexpr int ds_ready = v_empty + 8 * kStages;
  static constexpr int s_full = ds_ready + 8 * kStages;   // [2] Q.K^T of tile t is in the score buffer
  static constexpr int s_free = s_full + 16;              // [score buffers] the score buffer has been copied into registers
  static constexpr int p_full = s_free + 16;              // [2] P^ and its scales written (O rescaled if it had to be)
  static constexpr int pv_done = p_full + 16;             // [2] P.V MMAs of tile t complete: P^ may be rewritten, O_t is current
  static constexpr int drain = pv_done + 16;              // [2] the issuers' last commit when giving up
  static constexpr int corr = drain + 16;                 // [4 row quarters][2] alpha of a key tile is in shared memory, O_t may be rescaled
  static constexpr int tmem_slot = corr + 64;             // u32 written by tcgen05.alloc
  static constexpr int abort_flag = tmem_slot + 8;
  static constexpr int run_flag = abort_flag + 4;
};
static_assert(Bars::run_flag + 4 <= 512, "barrier block");

struct KParams {
  const uint8_t *q_sf, *k_sf, *vt_sf;
  const __nv_bfloat16* ds;
  __nv_bfloat16* out;
  float* lse;
  const float* lse_add;  // optional [B,Hq,Nq]: sm_scale * lse_add is added to the LSE (K-mean term removed by smoothing)
  int* status;
  int64_t o_sb, o_sh, o_sn;
  int B, Hq, Hkv, Nq, Nk, Tq, Tk, ds_rows;
  int list_tiles;        // kList: query tiles of the heads of a kv head
  int per_item;          // kList: how many of them make an item, 1 or 2, and
  int list_items;        //   how many items that are
  float scale_log2;      // sm_scale * log2(e)
  const float* lam;      // K-packing mode: lambda per key slot, fp32 [B,Hkv,Tk*128]; Nk is the packed length
  int Nk_log;            // number of key tokens (= Nk unless packed)
  int d_out;             // columns the output rows really have (<= D, multiple of 8)
  bool slot_first;       // K-packing mode: the mean slot takes the first token's score instead of being masked
  bool o_token_first;    // output tensor map: coordinates (d, token, head, batch) or (d, head, token, batch)
#if SAGE3_VARLEN_BUILD
  const int *cu_q, *cu_k; // token offsets of the sequences (device int32 [B+1]); Nq, Nk, Tq, Tk then describe the
                          // LONGEST sequence, i.e. the rectangular operand layouts
  const int *order, *n_order; // pairs of query tiles that exist (sequence * pairs + pair), heaviest first, and their number
#endif
};

// one arrival per warp: lane 0's, predicated instead of branched around
__device__ __forceinline__ void mbar_arrive_if(const bool who, const uint32_t bar) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %1, 0;\n@p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(bar), "r"((uint32_t)who) : "memory");
}
// ---- 3-input max
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float fmax3_nan(float a, float b, float c) {      // NaN if any of them is
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Largest of a 16-key block, NaNs left out.  `c` and `e` receive maxima over columns 6 to 8 and 12 to 14 that are NaN where
// one of those is: the columns that ex2_poly takes are among them (see nan_of_poly_columns).
__device__ __forceinline__ float max16(const uint32_t* r, float& c, float& e) {
  const float a = fmax3(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]));
  const float b = fmax3(__uint_as_float(r[3]), __uint_as_float(r[4]), __uint_as_float(r[5]));
  c = fmax3_nan(__uint_as_float(r[6]), __uint_as_float(r[7]), __uint_as_float(r[8]));
  const float d = fmax3(__uint_as_float(r[9]), __uint_as_float(r[10]), __uint_as_float(r[11]));
  e = fmax3_nan(__uint_as_float(r[12]), __uint_as_float(r[13]), __uint_as_float(r[14]));
  return fmax3(fmax3(a, b, c), fmax3(d, e, __uint_as_float(r[15])), kNoMax);
}

// The softmax of one key tile works on one score row (128 values) held in the registers of one thread; every
// loop below is fully unrolled so that the row never leaves the register file.

// K-packing mode (fwd_mainloop.cu:796-845, 878-881): a block of 16 keys is one group - slot 0 holds the
// score of the group mean, which every other score of the group gets added lambda times; the slot itself
// carries no token and is masked out.
__device__ __forceinline__ void apply_lambda(uint32_t* r, const float* lam16) {
  const float s0 = __uint_as_float(r[0]);
  const float2 s02 = make_float2(s0, s0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 l4 = reinterpret_cast<const float4*>(lam16)[i];
    const float2 a = ffma2(make_float2(l4.x, l4.y), s02, make_float2(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1])));
    const float2 b = ffma2(make_float2(l4.z, l4.w), s02, make_float2(__uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3])));
    r[4 * i] = __float_as_uint(a.x); r[4 * i + 1] = __float_as_uint(a.y);
    r[4 * i + 2] = __float_as_uint(b.x); r[4 * i + 3] = __float_as_uint(b.y);
  }
  r[0] = 0xff800000u;
}

// 2^x for two values on the FMA pipe (the special-function unit paces the softmax): x = n + r with n the nearest
// integer, found by adding and subtracting 1.5 * 2^23, |r| <= 1/2; 2^r by a polynomial of degree 5, minimax in the
// relative error (Remez exchange, computed for this file: 1.5e-7 with its coefficients rounded to fp32, 2.1e-7 = 2^-22.2 evaluated in
// fp32, the error bound of ex2.approx being 2^-22); n goes into the exponent bits.  x <= log2(6) here; below -125 (a
// masked score) the result is 2^-125: code 0, and nothing beside the 6 that the block's largest value adds to its sum.
// So is that of a NaN, which has to reach the row sum by another way: nan_of_poly_columns.
__device__ __forceinline__ float2 ex2_poly(float2 x) {
  const auto both = [](const float v) { return make_float2(v, v); };
  x.x = fmaxf(x.x, -125.f); x.y = fmaxf(x.y, -125.f);
  const float2 t = fadd2(x, both(12582912.f));
  const float2 r = ffma2(fadd2(t, both(-12582912.f)), both(-1.f), x);
  float2 p = ffma2(r, both(0.0013276472454890609f), both(0.009675540961325169f));
  p = ffma2(p, r, both(0.05550713092088699f));
  p = ffma2(p, r, both(0.24022120237350464f));
  p = ffma2(p, r, both(0.6931469440460205f));
  p = ffma2(p, r, both(1.0000001192092896f));
  p.x = __int_as_float(__float_as_int(p.x) + (__float_as_int(t.x) << 23));
  p.y = __int_as_float(__float_as_int(p.y) + (__float_as_int(t.y) << 23));
  return p;
}
// Which of the 8 pairs of a 16-key block take it: 3 in 16.  Whole operator for 0 / 2 / 3 / 4 of 16 on rows of 256 key tiles
// (B1 H10 N32760): D=128 3.55 / 3.42 / 3.41 / 3.45 ms, D=64 3.61 / 3.37 / 3.27 / 3.54 ms - more, and the 12
// instructions per pair cost more issue slots than the unit's cycles they save.
__device__ constexpr bool on_fma_pipe(const int blk, const int pair) { return pair == 3 || (pair == 6 && (blk & 1)); }
// A NaN if one of the columns that take it has a NaN score, else a finite number or +inf, from the maxima that max16 leaves:
// times 0 it goes into the row sum, so that such a row ends as one with a NaN in any other column does (its output zero, its
// LSE NaN) whatever the place of the key.  (A row with a score of +inf has that sum anyhow: inf - inf.)  7 instructions per key
// tile, 0.2 to 0.6 % of the kernel (B1 H40 N32760 D128 14.48 -> 14.57 ms); a select behind every polynomial would be 48.
__device__ __forceinline__ float nan_of_poly_columns(const float (&c)[8], const float (&e)[8]) {
  float x = kNoMax;
#pragma unroll
  for (int blk = 0; blk < 8; blk += 2) x = fmax3_nan(x, c[blk], c[blk + 1]);
  x = fmax3_nan(x, e[1], e[3]);
  return fmax3_nan(x, e[5], e[7]);
}

// Two 16-key blocks, 2 kPair and the next: P / blockscale = 2^(s*c - (bm*c + log2(1/6))) in [0, 6] -> E2M1 codes, 8 to a word in key
// order; they go into this row's 16 tensor-memory columns of P^, from where the P.V MMA reads its A operand.  To lsum, the row sum
// of the unquantised P, (sum of P/blockscale) * blockscale of each block is added (softmax_fused.h:135-153).
// neg_e[b] = -(bm_b*c + log2(1/6)), sb[b] = the block's unrounded scale.
// K-packing mode with slot_first: the first column of every block is the group's mean slot carrying a copy of the
// first token's score; its P^ goes to the MMA like any other, but it is no token and stays out of the row sum
// (softmax_fused.h:48-64).
template <bool kPacked, int kPair>
__device__ __forceinline__ void exp_quantise(const uint32_t (&s)[128], const float c, const float (&neg_e)[8], const float (&sb)[8],
                                             const bool slot_first, float& lsum, uint32_t (&code)[4]) {
  const float2 c2 = make_float2(c, c);
#pragma unroll
  for (int blk = 2 * kPair; blk < 2 * kPair + 2; ++blk) {
    const float2 nb2 = make_float2(neg_e[blk], neg_e[blk]);
    float2 e[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      e[i] = ffma2(make_float2(__uint_as_float(s[16 * blk + 2 * i]), __uint_as_float(s[16 * blk + 2 * i + 1])), c2, nb2);
      if (on_fma_pipe(blk, i)) e[i] = ex2_poly(e[i]);
      else { e[i].x = ex2_approx(e[i].x); e[i].y = ex2_approx(e[i].y); }
    }
    const float2 s4 = fadd2(fadd2(fadd2(e[0], e[1]), fadd2(e[2], e[3])), fadd2(fadd2(e[4], e[5]), fadd2(e[6], e[7])));
    float bsum = s4.x + s4.y;
    if (kPacked && slot_first) bsum -= e[0].x;
    lsum = fmaf(bsum, sb[blk], lsum);
    code[(blk & 1) * 2 + 0] = f32x8_to_e2m1x8(e[0].x, e[0].y, e[1].x, e[1].y, e[2].x, e[2].y, e[3].x, e[3].y);
    code[(blk & 1) * 2 + 1] = f32x8_to_e2m1x8(e[4].x, e[4].y, e[5].x, e[5].y, e[6].x, e[6].y, e[7].x, e[7].y);
  }
}

// K-packing mode: 15 tokens occupy 16 key slots (fwd_mainloop.cu:273-303).  Last slot that token `tok` or an
// earlier one occupies / number of slots the first `len` tokens occupy.
__device__ __forceinline__ int packed_slot_of_token(const int tok) { return (tok / 15) * 16 + tok % 15 + 1; }
__device__ __forceinline__ int packed_len_of(const int len) {
  return len <= 0 ? 0 : (len / 15) * 16 + (len % 15 == 0 ? 0 : len % 15 + 1);
}

// One unit of work of a CTA: two adjacent query tiles of one head - or, in the kList kernels, of the list of all query
// tiles of the heads that share a kv head: with an odd number of tiles every head would have an item of a single tile,
// which costs three quarters of a full one.
struct Work {
  int b, hq, hkv, pair;  // (kList: hq = first head of the list, pair = place in it)
#if SAGE3_VARLEN_BUILD
  int Nq, Nk;            // lengths of this item's sequence
  int q_base;            // first token of the sequence in the packed output
#endif
  int n_t[2];            // key tiles each query tile visits (0: none / tile does not exist)
  int n_max;
};

// Static schedule: in round r CTA i takes item r*G + i, odd rounds in reverse CTA order, so a CTA that got
// the heaviest item of one round gets the lightest of the next.  Returns -1 when the CTA is done.
__device__ __forceinline__ int work_at(const int r, const int total) {
  const int G = (int)gridDim.x, i = (int)blockIdx.x;
  const int w = r * G + ((r & 1) ? G - 1 - i : i);
  return w < total ? w : -1;
}

// head and query tile (>= Tq: there is none) of tile t of a work item
template <bool kList>
__device__ __forceinline__ int head_of(const KParams& P, const Work& k, const int t) {
  return kList ? k.hq + (P.per_item * k.pair + t) / P.Tq : k.hq;
}
template <bool kList>
__device__ __forceinline__ int tile_of(const KParams& P, const Work& k, const int t) {
  if (!kList) return 2 * k.pair + t;
  const int u = P.per_item * k.pair + t;
  return t < P.per_item && u < P.list_tiles ? u % P.Tq : P.Tq;
}

template <bool kCausal, bool kPacked, bool kList>
__device__ __forceinline__ Work get_work(const KParams& P, const int w) {
  Work k;
  const int n_pairs = kList ? P.list_items : (P.Tq + 1) >> 1;
  int bh;
#if SAGE3_VARLEN_BUILD
  const int entry = P.order[w / P.Hq];
  k.pair = entry % n_pairs;
  bh = entry / n_pairs * P.Hq + w % P.Hq;
#else
  if (kList) {
    // equal cost, as below
    k.pair = n_pairs - 1 - (w % n_pairs);
    bh = w / n_pairs * (P.Hq / P.Hkv);
  } else if (kCausal) {
    // item cost grows with the pair index: heaviest pairs of all heads first, so that the rounds of
    // the static schedule hand out work of falling, nearly equal cost
    const int n_bh = P.B * P.Hq;
    k.pair = n_pairs - 1 - w / n_bh;
    bh = w % n_bh;
  } else {
    // equal cost: keep the pairs of one head adjacent in time (they share K/V in L2)
    k.pair = n_pairs - 1 - (w % n_pairs);
    bh = w / n_pairs;
  }
#endif
  k.b = bh / P.Hq;
  k.hq = bh % P.Hq;
  k.hkv = k.hq / (P.Hq / P.Hkv);
#if SAGE3_VARLEN_BUILD
  k.q_base = P.cu_q[k.b];
  // a sequence longer than the caller's max_seqlen is cut there: the operand layouts (and the workspace) are
  // sized by max_seqlen, so tile indices beyond it must never be formed
  k.Nq = min(P.cu_q[k.b + 1] - k.q_base, P.Nq);
  k.Nk = min(P.cu_k[k.b + 1] - P.cu_k[k.b], P.Nk);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int qt = 2 * k.pair + t;
    int n = 0;
    if (qt * kBlockM < k.Nq) {
      const int Tk = (k.Nk + kBlockN - 1) / kBlockN;
      n = Tk;
      if (kCausal) {
        const int q_end = min((qt + 1) * kBlockM, k.Nq);
        const int lim = q_end + k.Nk - k.Nq;               // key tokens [0, lim) can be visible
        n = lim <= 0 ? 0 : min(Tk, (lim + kBlockN - 1) / kBlockN);
      }
    }
    k.n_t[t] = n;
  }
#else
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int qt = tile_of<kList>(P, k, t);
    int n = 0;
    if (qt < P.Tq) {
      n = P.Tk;
      if (kCausal) {
        const int q_end = min((qt + 1) * kBlockM, P.Nq);
        int lim = q_end + P.Nk_log - P.Nq;                 // key tokens [0, lim) can be visible
        if (kPacked) lim = packed_len_of(lim);             // ... which occupy this many key slots
        n = lim <= 0 ? 0 : min(P.Tk, (lim + kBlockN - 1) / kBlockN);
      }
    }
    k.n_t[t] = n;
  }
#endif
  k.n_max = max(k.n_t[0], k.n_t[1]);
  return k;
}

template <int D, bool kCausal, bool kPacked, bool kList>
__global__ void __launch_bounds__(kAttnThreads, 1) attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                                   const __grid_constant__ CUtensorMap tm_k,
                                                                   const __grid_constant__ CUtensorMap tm_v,
                                                                   const __grid_constant__ CUtensorMap tm_o,
                                                                   const KParams P) {
  using L = Smem<D>;
  // Score buffers in tensor memory: one for each query tile where there is room (D=64, one buffer / two: B4 H32 N4096 753 / 739 us, B4
  // H32/8 N8192 causal 1445 / 1408, B1 H10 N32760 3296 / 3273, B2 H16 N4100 Nk333 39.9 / 39.1, B8 H32 N1024 causal 115.5 / 113.0)
  constexpr int kSBufs = D == 64 ? 2 : 1;
  constexpr int kKB = D / 64;                              // K=64 blocks of the QK contraction
  constexpr uint32_t kSwzQK = (D == 128) ? 4u : 6u;        // 64-byte / 32-byte swizzle
  constexpr uint32_t kSboQK = (D == 128) ? 512u : 256u;
  constexpr bool kTmaStore = !SAGE3_VARLEN_BUILD && D == 128;   // see the epilogue
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // swizzled tiles need 1024-byte alignment
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bars = sbase + L::bars;
  volatile int* abort_s = reinterpret_cast<volatile int*>(smem + L::bars + Bars::abort_flag);
  // by a shuffle, so that the compiler knows it to be the same in all lanes: the roles' loops, branches and descriptors are then
  // uniform code (16 prompts 457 -> 435 us, K-packing B4 H32 N2048 306 -> 287, B4 H32/8 N8192 causal 1708 -> 1661)
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const bool has_ds = P.ds != nullptr;
#if !SAGE3_VARLEN_BUILD
  const int total_work = kList ? P.B * P.Hkv * P.list_items : P.B * P.Hq * ((P.Tq + 1) >> 1);
#endif

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) {
      mbar_init(bars + Bars::q_full + 8 * t, 1);
      mbar_init(bars + Bars::q_empty + 8 * t, 1);          // tcgen05.commit after the last QK that reads the tile
      mbar_init(bars + Bars::s_full + 8 * t, 1);           // tcgen05.commit
      mbar_init(bars + Bars::p_full + 8 * t, 8);           // the softmax warps of the tile and the four of O
      mbar_init(bars + Bars::pv_done + 8 * t, 1);          // tcgen05.commit
    }
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bars + Bars::k_full + 8 * s, 1);
      mbar_init(bars + Bars::k_empty + 8 * s, 1);          // tcgen05.commit
      mbar_init(bars + Bars::v_full + 8 * s, 1);
      mbar_init(bars + Bars::v_empty + 8 * s, 1);          // tcgen05.commit
      mbar_init(bars + Bars::ds_ready + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(bars + Bars::s_free + 8 * i, 4);
    for (int i = 0; i < 8; ++i) mbar_init(bars + Bars::corr + 8 * i, 1);
    mbar_init(bars + Bars::drain, 1);
    mbar_init(bars + Bars::drain + 8, 1);
    // the operands are there once the kernel before is complete (one thread waits for it, the barriers below pass that on)
    pdl_wait();
    // a failure reported by an earlier CTA (or an earlier launch that shares *status) stops new work
    const int bad = *reinterpret_cast<volatile int*>(P.status) != 0;
    *abort_s = bad;
    *reinterpret_cast<volatile int*>(smem + L::bars + Bars::run_flag) = !bad;
    fence_mbar_init();
  }
  // rank-1 operands: zero everything, then column 0 of A1 = 1.0
  for (int i = threadIdx.x; i < (L::dsraw - L::a1) / 16; i += kAttnThreads)
    reinterpret_cast<uint4*>(smem + L::a1)[i] = make_uint4(0, 0, 0, 0);
  if (warp == 13) {
    tmem_alloc(bars + Bars::tmem_slot, 512);
    tmem_relinquish();
  }
  __syncthreads();
  if (threadIdx.x < 128)
    *reinterpret_cast<__nv_bfloat16*>(smem + L::a1 + (threadIdx.x >> 3) * 128 + (threadIdx.x & 7) * 16) =
        __float2bfloat16(1.0f);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::bars + Bars::tmem_slot);
  // columns: O0 [0, D)  O1 [D, 2D)  S [2D, 2D + 128 kSBufs)  scale factors behind
  const uint32_t tm_Sbuf = tmem + 2 * D;
  const uint32_t tm_sfq = tm_Sbuf + 128 * kSBufs, tm_sfk = tm_sfq + 16, tm_sfp = tm_sfk + 16, tm_sfv = tm_sfp + 16;
  const uint32_t tm_P = tm_sfv + 8;                       // [2] P^ codes: the A operand of the P.V MMAs, 16 columns each

  // read once after the barrier: every warp takes the same branch, so the register hand-over
  // below (setmaxnreg) is always executed by whole warpgroups
  const bool run = *reinterpret_cast<volatile int*>(smem + L::bars + Bars::run_flag) != 0;
#if SAGE3_VARLEN_BUILD
  const int total_work = *P.n_order * P.Hq;
#endif
  // The CTA is persistent: every role walks the same static list of work items (blockIdx.x, +gridDim.x, ...)
  // and all barrier phases simply keep counting across items, so the loads, MMAs and softmax of the
  // next item start while the tail of the current one is still being finished.
  if (run) {
    if (warp >= 12) {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RegSplit::role));
      if (warp == 12) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) { prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_o); }
        int fail = 0;
        uint32_t g = 0;                       // K/V stages completely issued so far
        uint32_t gk = 0;                      // K stages issued so far (g or g + 1)
        uint32_t qn[2] = {0, 0};              // Q tiles loaded so far per slot
#pragma unroll 1
        for (int r = 0, w; fail == 0 && (w = work_at(r, total_work)) >= 0; ++r) {
          const Work wk = get_work<kCausal, kPacked, kList>(P, w);
          int64_t ds_row[2];
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int qt = (kList ? P.per_item : 2) * wk.pair + t;
            if (kList) ds_row[t] = ((int64_t)wk.b * P.Hq + head_of<kList>(P, wk, t)) * P.ds_rows + (P.ds_rows == 1 ? 0 : tile_of<kList>(P, wk, t));
            else ds_row[t] = ((int64_t)wk.b * P.Hq + wk.hq) * P.ds_rows + (P.ds_rows == 1 ? 0 : qt);
            if (fail == 0 && wk.n_t[t] > 0) {
              // the slot's previous Q tile must have been read by its last QK MMA
              if (qn[t] > 0 && (fail = wait_bar<12>(bars + Bars::q_empty + 8 * t, (qn[t] - 1) & 1)) != 0) break;
              const int64_t qtile = ((int64_t)wk.b * P.Hq + wk.hq) * P.Tq + qt;
              const uint32_t qb = bars + Bars::q_full + 8 * t;
              if (lane == 0) {
                mbar_arrive_expect_tx(qb, L::kQBytes + L::kSfRow);
                tma_load_2d(sbase + L::q + t * L::kQBytes, &tm_q, 0, (int)(qtile * kBlockM), qb);
                bulk_load(sbase + L::sfq + t * 1024, P.q_sf + qtile * L::kSfRow, L::kSfRow, qb);
              }
              __syncwarp();
              ++qn[t];
            }
          }
          const int64_t kvhead = ((int64_t)wk.b * P.Hkv + wk.hkv) * P.Tk;
#pragma unroll 1
          for (int it = 0; fail == 0 && it < wk.n_max; ++it, ++g) {
            const int j = wk.n_max - 1 - it, s = g % kStages;
            const uint32_t ph = ((g / kStages) & 1) ^ 1;
            if ((fail = wait_bar<10>(bars + Bars::k_empty + 8 * s, ph)) != 0) break;
            const uint32_t kb = bars + Bars::k_full + 8 * s;
            const int nds = has_ds ? (int)(j < wk.n_t[0]) + (int)(j < wk.n_t[1]) : 0;
            if (lane == 0) {
              mbar_arrive_expect_tx(kb, L::kKBytes + L::kSfRow + 256 * nds + (kPacked ? 512 : 0));
              if (kPacked) bulk_load(sbase + L::lam + (g % (2 * kStages)) * 512, P.lam + (kvhead + j) * kBlockN, 512, kb);
              tma_load_2d(sbase + L::k + s * L::kKBytes, &tm_k, 0, (int)((kvhead + j) * kBlockN), kb);
              bulk_load(sbase + L::sfk + s * 1024, P.k_sf + (kvhead + j) * L::kSfRow, L::kSfRow, kb);
              if (has_ds) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                  if (j < wk.n_t[t])
                    bulk_load(sbase + L::dsraw + (s * 2 + t) * 256, P.ds + (ds_row[t] * P.Tk + j) * kBlockN, 256, kb);
              }
            }
            __syncwarp();
            ++gk;
            if ((fail = wait_bar<11>(bars + Bars::v_empty + 8 * s, ph)) != 0) break;
            const uint32_t vb = bars + Bars::v_full + 8 * s;
            if (lane == 0) {
              mbar_arrive_expect_tx(vb, L::kVBytes + L::kSfV);
              tma_load_2d(sbase + L::v + s * L::kVBytes, &tm_v, 0, (int)((kvhead + j) * D), vb);
              bulk_load(sbase + L::sfv + s * 1024, P.vt_sf + (kvhead + j) * L::kSfV, L::kSfV, vb);
            }
            __syncwarp();
          }
        }
        if (fail != 0) give_up(abort_s, P.status, fail);
        if (__any_sync(0xffffffffu, *abort_s != 0)) {
          // giving up: the copies this thread started must land before the CTA may exit
          for (int t = 0; t < 2; ++t)
            if (qn[t] > 0) mbar_wait<true>(bars + Bars::q_full + 8 * t, (qn[t] - 1) & 1, 1u << 16);
          for (uint32_t i = (gk > (uint32_t)kStages ? gk - kStages : 0); i < gk; ++i)
            mbar_wait<true>(bars + Bars::k_full + 8 * (i % kStages), (i / kStages) & 1, 1u << 16);
          for (uint32_t i = (g > (uint32_t)kStages ? g - kStages : 0); i < g; ++i)
            mbar_wait<true>(bars + Bars::v_full + 8 * (i % kStages), (i / kStages) & 1, 1u << 16);
        }
      } else if (warp == 14 && has_ds) {
        // ---------------------------------------------------------------- delta_s -> rank-1 B operand
        // B1 is a K-major [128 keys x 16] bf16 operand in 8x16-byte core matrices: key n's first
        // element sits at (n/8)*128 + (n%8)*16; everything else stays zero.
        int fail = 0;
        uint32_t s = 0, ph = 0;
#pragma unroll 1
        for (int r = 0, w; fail == 0 && (w = work_at(r, total_work)) >= 0; ++r) {
          const Work wk = get_work<kCausal, kPacked, kList>(P, w);
#pragma unroll 1
          for (int j = wk.n_max - 1; j >= 0; --j) {
            if ((fail = wait_bar<40>(bars + Bars::k_full + 8 * s, ph)) != 0) break;
#pragma unroll 1
            for (int t = 0; t < 2; ++t) {
              if (j < (t == 0 ? wk.n_t[0] : wk.n_t[1])) {
                const uint16_t* raw = reinterpret_cast<const uint16_t*>(smem + L::dsraw + (s * 2 + t) * 256);
                uint8_t* dst = smem + L::b1 + (s * 2 + t) * 2048 + (lane >> 3) * 128 + (lane & 7) * 16;   // keys lane + 32 i
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<uint16_t*>(dst + i * 512) = raw[lane + 32 * i];
              }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + Bars::ds_ready + 8 * s);
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
        }
        if (fail != 0) give_up(abort_s, P.status, fail);
      } else if (warp == 13) {
        // ---------------------------------------------------------------- QK issuer
        // Its instruction stream is kept minimal: every shared-memory descriptor is a constant high word (stride /
        // swizzle / version bits) plus a low word (address >> 4, leading-offset field) that only needs an integer
        // add per use.  It waits with a suspend-time hint (1 % over all shapes).
        constexpr uint32_t idesc_qk = make_idesc_nvf4(kBlockM, kBlockN);
        constexpr uint32_t idesc_r1 = make_idesc_bf16(kBlockM, kBlockN);
        constexpr uint32_t HI_QK = (kSboQK >> 4) | (1u << 14) | (kSwzQK << 29);
        constexpr uint32_t HI_SF = (128u >> 4) | (1u << 14);          // 8x16-byte core matrices, no swizzle
        constexpr uint32_t LBO1 = 1u << 16;                            // leading offset field of swizzled operands
        const uint32_t q_lo = ((sbase + L::q) >> 4) | LBO1, k_lo = ((sbase + L::k) >> 4) | LBO1;
        const uint32_t sfq_lo = (sbase + L::sfq) >> 4, sfk_lo = (sbase + L::sfk) >> 4;
        const uint32_t a1_lo = ((sbase + L::a1) >> 4) | (((uint32_t)(L::zero - L::a1) >> 4) << 16);
        const uint32_t b1_lo = ((sbase + L::b1) >> 4) | (((uint32_t)(L::zero - L::b1) >> 4) << 16);
        int fail = 0;
        uint32_t s = 0, ph = 0;               // K stage and its parity
        uint32_t nqk = 0;                     // QK groups issued so far (= uses of the score buffer)
        uint32_t s_odd = 0;                   // K stages so far, odd or even
        uint32_t s_par = 0;                   // bit t: uses of tile t's own score buffer so far (kSBufs == 2), odd or even
        uint32_t q_par = 0;                   // bit t: parity of the Q tile to come in slot t
#pragma unroll 1
        for (int r = 0, w; fail == 0 && (w = work_at(r, total_work)) >= 0; ++r) {
          const Work wk = get_work<kCausal, kPacked, kList>(P, w);
#pragma unroll 1
          for (int j = wk.n_max - 1; fail == 0 && j >= 0; --j) {
            if ((fail = wait_bar_uniform<21>(bars + Bars::k_full + 8 * s, ph)) != 0) break;
            if (has_ds && (fail = wait_bar_uniform<25>(bars + Bars::ds_ready + 8 * s, ph)) != 0) break;
            // Its scale factors on their way before the score buffer is free, into the columns that the MMAs of the stage before do not
            // read (B1 H10 N32760 D128 3466 -> 3452 us; D=64 is within 0.3 % either way).  MMAs of two stages before have been seen complete by the waits for score
            // buffers; but where an item of both tiles is followed by one of tile 0 only, at D=64, whose tile 0 does not wait for
            // tile 1's buffer, it is the order in which the tensor pipe takes the copies and MMAs that one thread issues, as for
            // the columns of V's scale factors.
            const uint32_t tm_sfk_s = tm_sfk + 8 * (s_odd & 1);
            s_odd ^= 1;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int kb = 0; kb < kKB; ++kb) tc_cp_sf(tm_sfk_s + 4 * kb, sfk_lo + s * 64 + kb * 32, HI_SF);
            }
#pragma unroll 1
            for (int t = 0; t < 2; ++t) {
              const int n_t = t == 0 ? wk.n_t[0] : wk.n_t[1];
              if (j >= n_t) continue;
              // the score buffer must be free: the softmax warpgroup that got its last Q.K^T (the one buffer: of the other
              // query tile, or of this one in the previous key tile; a buffer for each: of this one) has copied it into
              // registers.  (Nothing to wait for: parity 1.)
              const uint32_t free_par = kSBufs == 1 ? (nqk - 1) & 1 : ((s_par >> t) & 1) ^ 1;
              if ((fail = wait_bar_uniform<23>(bars + Bars::s_free + 8 * (kSBufs - 1) * t, free_par)) != 0) break;
              if (kSBufs == 2) s_par ^= 1u << t;
              const uint32_t tm_S = tm_Sbuf + 128 * (kSBufs - 1) * t;
              if (j == n_t - 1) {                                  // first key tile of this query tile
                if ((fail = wait_bar_uniform<20>(bars + Bars::q_full + 8 * t, (q_par >> t) & 1)) != 0) break;
                q_par ^= 1u << t;
                tc_fence_after();
                if (elect_one())
#pragma unroll
                  for (int kb = 0; kb < kKB; ++kb) tc_cp_sf(tm_sfq + 8 * t + 4 * kb, sfq_lo + t * 64 + kb * 32, HI_SF);
              }
              tc_fence_after();
              if (elect_one()) {
                if (has_ds) {
                  // buffer i sits i*2048 bytes higher, so its distance to the shared zero chunk is i*2048 smaller
                  const uint32_t i = s * 2 + t;
                  tc_mma_bf16(tm_S, a1_lo, HI_SF, b1_lo + i * 128u - ((i * 128u) << 16), HI_SF, idesc_r1, 0);
                }
#pragma unroll
                for (int kb = 0; kb < kKB; ++kb)
                  tc_mma_nvf4(tm_S, q_lo + t * (L::kQBytes >> 4) + kb * 2, HI_QK, k_lo + s * (L::kKBytes >> 4) + kb * 2, HI_QK,
                              idesc_qk, tm_sfq + 8 * t + 4 * kb, tm_sfk_s + 4 * kb, (has_ds || kb > 0) ? 1u : 0u);
                tc_commit(bars + Bars::s_full + 8 * t);
                if (j == 0) tc_commit(bars + Bars::q_empty + 8 * t);   // last read of this Q tile
              }
              __syncwarp();
              ++nqk;
            }
            if (fail == 0 && elect_one()) tc_commit(bars + Bars::k_empty + 8 * s);
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
        }
        if (fail != 0) {
          give_up(abort_s, P.status, fail);
          // giving up: let every MMA / scale copy already issued finish before tensor memory is freed
          if (elect_one()) tc_commit(bars + Bars::drain);
          mbar_wait<true>(bars + Bars::drain, 0, 1u << 16);
        }
      } else if (warp == 15) {
        // ---------------------------------------------------------------- PV issuer
        // O_t += P^_t V^ for both tiles, from its own thread so that waiting for P^ never delays the next QK.
        // The first key tile of a work item overwrites O_t (no accumulate).
        constexpr uint32_t idesc_pv = make_idesc_nvf4(kBlockM, D);
        constexpr uint32_t HI_PV = (512u >> 4) | (1u << 14) | (4u << 29);
        constexpr uint32_t HI_SF = (128u >> 4) | (1u << 14);
        constexpr uint32_t LBO1 = 1u << 16;
        const uint32_t v_lo = ((sbase + L::v) >> 4) | LBO1;
        const uint32_t sfv_lo = (sbase + L::sfv) >> 4, sfp_lo = (sbase + L::sfp) >> 4;
        int fail = 0;
        uint32_t s = 0, ph = 0;               // V stage and its parity
        uint32_t p_par = 0;                   // bit t: parity of the P^ to come of tile t
#pragma unroll 1
        for (int r = 0, w; fail == 0 && (w = work_at(r, total_work)) >= 0; ++r) {
          const Work wk = get_work<kCausal, kPacked, kList>(P, w);
#pragma unroll 1
          for (int j = wk.n_max - 1; fail == 0 && j >= 0; --j) {
            // the V stage and its scale factors do not depend on the softmax: fetch them before waiting for P
            if ((fail = wait_bar<24>(bars + Bars::v_full + 8 * s, ph)) != 0) break;
            tc_fence_after();
            if (elect_one())
#pragma unroll
              for (int kb = 0; kb < 2; ++kb) tc_cp_sf(tm_sfv + 4 * kb, sfv_lo + s * 64 + kb * 32, HI_SF);
#pragma unroll 1
            for (int t = 0; t < 2; ++t) {
              const int n_t = t == 0 ? wk.n_t[0] : wk.n_t[1];
              if (j >= n_t) continue;
              if ((fail = wait_bar<26>(bars + Bars::p_full + 8 * t, (p_par >> t) & 1)) != 0) break;
              p_par ^= 1u << t;
              tc_fence_after();
              if (elect_one()) {
#pragma unroll
                for (int kb = 0; kb < 2; ++kb) tc_cp_sf(tm_sfp + 8 * t + 4 * kb, sfp_lo + t * 64 + kb * 32, HI_SF);
#pragma unroll
                for (int kb = 0; kb < 2; ++kb)
                  tc_mma_nvf4_ta(tmem + t * D, tm_P + 16 * t + 8 * kb, v_lo + s * (L::kVBytes >> 4) + kb * 2, HI_PV,
                                 idesc_pv, tm_sfp + 8 * t + 4 * kb, tm_sfv + 4 * kb, (j == n_t - 1 && kb == 0) ? 0u : 1u);
                tc_commit(bars + Bars::pv_done + 8 * t);
              }
              __syncwarp();
            }
            if (fail == 0 && elect_one()) tc_commit(bars + Bars::v_empty + 8 * s);
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
        }
        if (fail != 0) {
          give_up(abort_s, P.status, fail);
          if (elect_one()) tc_commit(bars + Bars::drain + 8);
          mbar_wait<true>(bars + Bars::drain + 8, 0, 1u << 16);
        }
      }
    } else {
      const int quarter = warp & 3;
      const int row = quarter * 32 + lane;                       // tensor-memory lane
      const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
      const float c = P.scale_log2;
      if (warp < 8) {
        // ---------------------------------------------------------------- softmax
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(RegSplit::softmax));
        // (which wait ran out as a flag and not, as elsewhere, as its code: B1 H40 N32760 13.47 -> 13.30 ms, D64 H10 3.33 -> 3.28)
        bool ok = true, late = false;
        const int t = warp >> 2;                                 // query tile slot of this warpgroup
        const uint32_t tm_S = tm_Sbuf + 128 * (kSBufs - 1) * t + lane_addr;
        const uint32_t bar_f = bars + Bars::s_free + 8 * (kSBufs - 1) * t;
        const uint32_t tm_Prow = tm_P + 16 * t + lane_addr;      // this row of P^: 16 columns of 8 codes
        uint32_t* sfp_row = reinterpret_cast<uint32_t*>(smem + L::sfp + t * 1024 + sf_atom_offset(row, 0));
        volatile float* alpha_row = reinterpret_cast<volatile float*>(smem + L::alpha) + t * 128 + row;
        volatile float* l_row = reinterpret_cast<volatile float*>(smem + L::lx) + t * 256 + row;   // [2 items][l, m]
        const uint32_t bar_s = bars + Bars::s_full + 8 * t, bar_p = bars + Bars::p_full + 8 * t;
        const uint32_t bar_pv = bars + Bars::pv_done + 8 * t, bar_c = bars + Bars::corr + 8 * (2 * quarter + t);
        uint32_t sc = 0;                                         // key tiles processed so far by this warpgroup
        uint32_t g0 = 0;                                         // K/V stages the CTA used before this work item
        uint32_t items = 0;
        bool s_ready = false;                                    // the next tile's scores were there when last looked at
        // P^ written: hand the tile to the PV issuer.  The codes went to tensor memory (tcgen05.st), their block
        // scales to shared memory for the issuer's tcgen05.cp.
        auto hand_over = [&](const bool there_is) {
          tmem_wait_st();
          tc_fence_before();
          fence_proxy_async_smem();
          __syncwarp();
          mbar_arrive_if(lane == 0 && there_is, bar_p);
        };
#pragma unroll 1
        for (int r = 0, w; ok && (w = work_at(r, total_work)) >= 0; ++r) {
          const Work wk = get_work<kCausal, kPacked, kList>(P, w);
          const int n_mine = t == 0 ? wk.n_t[0] : wk.n_t[1];
          const uint32_t g_first = g0 + (uint32_t)(wk.n_max - n_mine);   // stage counter of this tile's first key tile
          g0 += (uint32_t)wk.n_max;
          if (n_mine == 0) continue;
          const int q0 = tile_of<kList>(P, wk, t) * kBlockM, qpos = q0 + row;
          // last visible key (slot): key padding, and the bottom-right aligned causal diagonal - in K-packing mode
          // the slots of the tokens up to the diagonal one
          auto causal_limit = [&](const int qp) {
            const int tok = qp + SEQ_NK_LOG - SEQ_NQ;            // last visible key token
            if (!kPacked) return tok;
            return tok < 0 ? -1 : packed_slot_of_token(tok);
          };
          const int key_lim = min(SEQ_NK - 1, kCausal ? causal_limit(qpos) : 0x7fffffff);
          const int first_row_lim = kCausal ? causal_limit(q0) : 0x7fffffff;
          float m_run = kNoMax, l = 0.f;                         // row maximum so far (raw score units), row sum

#pragma unroll 1
          for (int it = 0; it < n_mine; ++it, ++sc) {
            const int n0 = (n_mine - 1 - it) * kBlockN;
            const bool need_mask = (n0 + kBlockN - 1 >= SEQ_NK) || (kCausal && n0 + kBlockN - 1 > first_row_lim);
            // the scores are usually there by now: then P^ of the tile before is handed over while they are on their way
            const bool ready = __all_sync(0xffffffffu, s_ready);
            if (!ready) {
              hand_over(it > 0);
              if (!(ok = wait_bar<30>(bar_s, sc & 1) == 0)) break;
            }
            tc_fence_after();
            uint32_t s[128];
            float bm[8], c6[8], c12[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) tmem_ld32(tm_S + 32 * q, *reinterpret_cast<uint32_t (*)[32]>(&s[32 * q]));
            if (ready) hand_over(it > 0);
            tmem_wait_ld();
            // the scores are in registers: the Q.K^T of the other query tile may overwrite the buffer
            tc_fence_before();
            mbar_arrive_if(lane == 0, bar_f);
            if (kPacked) {
              // lambda of this key tile arrived with its K stage, i.e. before the Q.K^T MMA whose completion was
              // awaited above.  Its slot is rewritten 2*kStages key tiles later, which the producer can only do
              // after the Q.K^T of tile g+kStages is complete - issued after both warpgroups finished tile g.
              const uint32_t g = g_first + (uint32_t)it;
              const float* lam_s = reinterpret_cast<const float*>(smem + L::lam) + (g % (2 * kStages)) * 128;
#pragma unroll
              for (int blk = 0; blk < 8; ++blk) apply_lambda(&s[16 * blk], lam_s + 16 * blk);
            }
            if (__builtin_expect(need_mask, 0)) {
              const int lim = key_lim - n0;                      // columns beyond it are masked
#pragma unroll
              for (int i = 0; i < 128; ++i) s[i] = (i > lim) ? 0xff800000u : s[i];
            }
            if (kPacked && P.slot_first) {
              // the other K-packing variant (fwd_mainloop.cu:847-891): the mean slot carries the (masked) score of the
              // group's first token - its V row holds that token's FP4 remainder - except, under the causal mask, in
              // the group of the diagonal token and beyond
              const int qk = qpos + SEQ_NK_LOG - SEQ_NQ;         // the diagonal key token of this row
              const int last_group = kCausal ? (qk < 0 ? -1 : qk / 15 - 1) : 0x7ffffff;   // last group whose slot may be used
#pragma unroll
              for (int blk = 0; blk < 8; ++blk) {
                const int col = n0 + 16 * blk;
                const bool usable = !kCausal || (col < SEQ_NK && (col >> 4) <= last_group);
                s[16 * blk] = usable ? s[16 * blk + 1] : 0xff800000u;
              }
            }
#pragma unroll
            for (int blk = 0; blk < 8; ++blk) bm[blk] = max16(&s[16 * blk], c6[blk], c12[blk]);
            const float m_loc = fmax3(fmax3(bm[0], bm[1], bm[2]), fmax3(bm[3], bm[4], bm[5]), fmaxf(bm[6], bm[7]));
            const float m_new = fmaxf(m_run, m_loc);
            const float alpha = ex2_approx((m_run - m_new) * c);
            l = fmaf(nan_of_poly_columns(c6, c12), 0.f, l);
            m_run = m_new;
            const float off = fmaf(m_new, c, kLog2Inv2688);       // P = 2^(s*c - off) in (0, 2688]
            float neg_e[8], sb[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float e = fmaf(bm[i], c, kLog2Inv6);
              sb[i] = ex2_approx(e - off);
              neg_e[i] = -e;
            }
            const bool pv_ready = mbar_test(bar_pv, (sc - 1) & 1);
            float lsum = 0.f;
            uint32_t code[4];
            exp_quantise<kPacked, 0>(s, c, neg_e, sb, P.slot_first, lsum, code);
            // the P.V MMAs of the previous key tile are complete: P^ and its scales may be rewritten, O rescaled
            if (!__all_sync(0xffffffffu, pv_ready) && !(ok = wait_bar<31>(bar_pv, (sc - 1) & 1) == 0)) {
              late = true;
              break;
            }
            tc_fence_after();
            *alpha_row = alpha;
            __syncwarp();
            mbar_arrive_if(lane == 0, bar_c);
            sfp_row[0] = f32x2_to_e4m3x2(sb[0], sb[1]) | (f32x2_to_e4m3x2(sb[2], sb[3]) << 16);     // keys 0-63 of the tile
            sfp_row[128] = f32x2_to_e4m3x2(sb[4], sb[5]) | (f32x2_to_e4m3x2(sb[6], sb[7]) << 16);   // keys 64-127
            tmem_st4(tm_Prow, code[0], code[1], code[2], code[3]);                                  // 32 keys = 4 columns
            exp_quantise<kPacked, 1>(s, c, neg_e, sb, P.slot_first, lsum, code);
            tmem_st4(tm_Prow + 4, code[0], code[1], code[2], code[3]);
            exp_quantise<kPacked, 2>(s, c, neg_e, sb, P.slot_first, lsum, code);
            tmem_st4(tm_Prow + 8, code[0], code[1], code[2], code[3]);
            exp_quantise<kPacked, 3>(s, c, neg_e, sb, P.slot_first, lsum, code);
            s_ready = mbar_test(bar_s, (sc + 1) & 1);
            tmem_st4(tm_Prow + 12, code[0], code[1], code[2], code[3]);
            l = fmaf(l, alpha, lsum);              // one rounding, whatever the compiler would make of a product and a sum
          }
          if (!ok) break;
          l_row[(items & 1) * 512] = l;
          l_row[(items & 1) * 512 + 128] = m_run;
          hand_over(true);
          ++items;
        }
        if (!ok) give_up(abort_s, P.status, late ? 31 : 30);
      } else {
        // ---------------------------------------------------------------- O: rescaling and output
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RegSplit::corr));
        int fail = 0;
        uint32_t sc[2] = {0, 0}, items[2] = {0, 0};              // key tiles / work items so far per query tile slot
#pragma unroll 1
        for (int r = 0, w; fail == 0 && (w = work_at(r, total_work)) >= 0; ++r) {
          const Work wk = get_work<kCausal, kPacked, kList>(P, w);
          // O_t *= alpha for the rows whose maximum moved, in place in tensor memory, between the P.V of the previous
          // key tile and that of this one; warps in which no row's maximum moved skip it.  The first key tile of an
          // item overwrites O_t: this arrival then says that the previous item's output has been read.
#pragma unroll 1
          for (int it = 0; fail == 0 && it < wk.n_max; ++it) {
#pragma unroll 1
            for (int t = 0; t < 2; ++t) {
              const int n_t = t == 0 ? wk.n_t[0] : wk.n_t[1];
              if (wk.n_max - 1 - it >= n_t) continue;
              uint32_t& cnt = t == 0 ? sc[0] : sc[1];
              if ((fail = wait_bar<32>(bars + Bars::corr + 8 * (2 * quarter + t), cnt & 1)) != 0) break;
              ++cnt;
              const float alpha = *(reinterpret_cast<volatile float*>(smem + L::alpha) + t * 128 + row);
              if (it != wk.n_max - n_t && __any_sync(0xffffffffu, alpha != 1.0f)) {
                tc_fence_after();
                const uint32_t tm_O = tmem + t * D + lane_addr;
                const float2 al2 = make_float2(alpha, alpha);
                uint32_t o[32];
#pragma unroll 1
                for (int ch = 0; ch < D / 32; ++ch) {
                  tmem_ld32(tm_O + ch * 32, o);
                  tmem_wait_ld();
#pragma unroll
                  for (int i = 0; i < 16; ++i) {
                    const float2 x = ffma2(make_float2(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1])), al2,
                                           make_float2(0.f, 0.f));
                    o[2 * i] = __float_as_uint(x.x); o[2 * i + 1] = __float_as_uint(x.y);
                  }
#pragma unroll
                  for (int h = 0; h < 2; ++h)
                    tmem_st16(tm_O + ch * 32 + 16 * h, *reinterpret_cast<const uint32_t (*)[16]>(&o[16 * h]));
                }
                tmem_wait_st();
                tc_fence_before();
              }
              __syncwarp();
              mbar_arrive_if(lane == 0, bars + Bars::p_full + 8 * t);
            }
          }
          if (fail != 0) break;

          // ---- output: O / l -> bf16 -> global.  D=128, dense batches: through a swizzled staging tile in shared
          // memory and two TMA stores per warp (32 rows x 64 columns) - a thread owns an output row, so direct
          // stores put 32 different rows into every store instruction.  D=64 (half the bytes) and packed
          // variable-length outputs (a tile must not spill into the next sequence) store directly.
#pragma unroll 1
          for (int t = 0; t < 2; ++t) {
            const int n_t = t == 0 ? wk.n_t[0] : wk.n_t[1];
            const int hq = head_of<kList>(P, wk, t), qt = tile_of<kList>(P, wk, t), q0 = qt * kBlockM, qpos = q0 + row;
            const bool live = SEQ_TILE_EXISTS && qpos < SEQ_NQ;
#if SAGE3_VARLEN_BUILD
            __nv_bfloat16* orow = P.out + hq * P.o_sh + (int64_t)(wk.q_base + qpos) * P.o_sn;   // packed output
#else
            __nv_bfloat16* orow = P.out + wk.b * P.o_sb + hq * P.o_sh + (int64_t)qpos * P.o_sn;
#endif
            const int64_t li = ((int64_t)wk.b * P.Hq + hq) * P.Nq + qpos;
            if (n_t == 0) {
              // query tile that sees no key at all (causal, more queries than keys): zeros, like the
              // reference's store_zero (fwd_epilogue.cu:150-183); nothing if the tile does not exist
              if (live) {
#pragma unroll 1
                for (int i = 0; i < P.d_out / 8; ++i) reinterpret_cast<uint4*>(orow)[i] = make_uint4(0, 0, 0, 0);
                if (P.lse) P.lse[li] = -INFINITY;
              }
              continue;
            }
            const uint32_t last = (t == 0 ? sc[0] : sc[1]) - 1;
            uint32_t& ni = t == 0 ? items[0] : items[1];
            // the last key tile's row sum is there, and its P.V has landed
            if ((fail = wait_bar<33>(bars + Bars::p_full + 8 * t, last & 1)) != 0) break;
            const volatile float* l_row = reinterpret_cast<const volatile float*>(smem + L::lx) + t * 256 + row + (ni & 1) * 512;
            const float l = l_row[0], m = l_row[128];
            ++ni;
            if ((fail = wait_bar<34>(bars + Bars::pv_done + 8 * t, last & 1)) != 0) break;
            tc_fence_after();
            const uint32_t tm_O = tmem + t * D + lane_addr;
            const bool keyless = m == kNoMax;                    // a row that has seen no key: zeros, LSE -inf
            const float inv = (keyless || l != l) ? 0.f : 1.0f / l;
            const float2 inv2 = make_float2(inv, inv);
            const uint32_t stage_off = L::ostage + (t * 4 + quarter) * (D / 64) * L::kOStage;
            uint8_t* stage = smem + stage_off + lane * 128;
            if (kTmaStore) {
              // the stores of this warp's previous output tiles must have left the staging tile
              if (lane == 0) bulk_wait_read0();
              __syncwarp();
            }
#pragma unroll 1
            for (int ch = 0; ch < D / 32; ++ch) {
              uint32_t o[32];
              tmem_ld32(tm_O + 32 * ch, o);
              tmem_wait_ld();
#pragma unroll
              for (int h = 0; h < 4; ++h) {
                uint4 v;
                float2 x;
                x = ffma2(make_float2(__uint_as_float(o[8 * h + 0]), __uint_as_float(o[8 * h + 1])), inv2, make_float2(0.f, 0.f));
                v.x = pack_bf16(x.x, x.y);
                x = ffma2(make_float2(__uint_as_float(o[8 * h + 2]), __uint_as_float(o[8 * h + 3])), inv2, make_float2(0.f, 0.f));
                v.y = pack_bf16(x.x, x.y);
                x = ffma2(make_float2(__uint_as_float(o[8 * h + 4]), __uint_as_float(o[8 * h + 5])), inv2, make_float2(0.f, 0.f));
                v.z = pack_bf16(x.x, x.y);
                x = ffma2(make_float2(__uint_as_float(o[8 * h + 6]), __uint_as_float(o[8 * h + 7])), inv2, make_float2(0.f, 0.f));
                v.w = pack_bf16(x.x, x.y);
                const int i = 4 * ch + h;                        // 16-byte chunk of the output row
                if (kTmaStore)
                  *reinterpret_cast<uint4*>(stage + (i >> 3) * L::kOStage + (((i & 7) ^ (lane & 7)) << 4)) = v;
                else if (live && 8 * i < P.d_out)
                  *reinterpret_cast<uint4*>(orow + 8 * i) = v;
              }
            }
            tc_fence_before();
            if (kTmaStore) {
              fence_proxy_async_smem();
              __syncwarp();
              const int n_row = q0 + 32 * quarter;
              if (lane == 0 && n_row < P.Nq) {
#pragma unroll
                for (int hcol = 0; hcol < D / 64; ++hcol)
                  if (64 * hcol < P.d_out)
                    tma_store_4d(&tm_o, sbase + stage_off + hcol * L::kOStage, 64 * hcol,
                                 P.o_token_first ? n_row : hq, P.o_token_first ? hq : n_row, wk.b);
                bulk_commit_group();
              }
            }
            if (live && P.lse) {
              // natural-log sum of exp(sm_scale * s) over the row (l carries the factor 2688)
              float v = keyless ? -INFINITY : (m * c + log2f(l) + kLog2Inv2688) * (1.0f / kLog2e);
              if (P.lse_add != nullptr) v = fmaf(P.lse_add[li], c * (1.0f / kLog2e), v);
              P.lse[li] = v;
            }
          }
        }
        if (fail != 0) give_up(abort_s, P.status, fail);
        if (kTmaStore && lane == 0) bulk_wait_read0();   // the last output tiles have left shared memory before the CTA ends
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 13) tmem_dealloc(tmem, 512);
}

// ------------------------------------------------------------------------------------------------
// host: tensor maps + launch
// ------------------------------------------------------------------------------------------------
// 2-D byte tensor [rows][row_bytes], box = [box_rows][row_bytes]
bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint32_t row_bytes, uint32_t box_rows,
              CUtensorMapSwizzle swz) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return false;
  cuuint64_t dims[2] = {row_bytes, rows};
  cuuint64_t strides[1] = {row_bytes};
  cuuint32_t box[2] = {row_bytes, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// bf16 output [B][Hq][Nq][D] with arbitrary element strides, box = 32 rows x 64 columns (128 bytes, swizzled).
// Tensor-map strides must grow with the dimension, so tokens and heads are ordered by their stride ("HND": D, N,
// H, B; "NHD": D, H, N, B); *n_dim tells the kernel which coordinate is the token.
bool make_out_map(CUtensorMap* m, const void* base, int B, int H, int N, int D, int64_t sb, int64_t sh, int64_t sn,
                  int* n_dim) {   // D = columns the rows really have: the 64-column boxes are clipped to it
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return false;
  // a dimension of extent 1 never advances; give it a stride that keeps the order valid
  const bool n_first = (H == 1) || (N > 1 && sn <= sh);
  *n_dim = n_first ? 1 : 2;
  cuuint64_t dims[4] = {(cuuint64_t)D, 0, 0, (cuuint64_t)B};
  cuuint64_t strides[3];
  cuuint32_t box[4] = {64, 1, 1, 1};
  const cuuint64_t s_n = (cuuint64_t)sn * 2, s_h = (cuuint64_t)sh * 2;
  if (n_first) {
    dims[1] = N; dims[2] = H; box[1] = 32;
    strides[0] = N > 1 ? s_n : (cuuint64_t)D * 2;
    strides[1] = H > 1 ? s_h : strides[0] * N;
  } else {
    dims[1] = H; dims[2] = N; box[2] = 32;
    strides[0] = s_h;
    strides[1] = N > 1 ? s_n : strides[0] * H;
  }
  strides[2] = B > 1 ? (cuuint64_t)sb * 2 : strides[1] * dims[2];
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// At most one query tile per CTA that may run: one per item then (kList kernels), since an item of one takes three quarters of
// the time of two (B1 H8 N1024 20.8 -> 16.4 us, B1 H32/8 N128 causal 10.2 -> 7.9 us).  CTAs, not SMs: with a margin and a tile
// count between the two, single tiles would take two rounds where pairs take one (B1 H32/8 N512, margin 25: 20.5 -> 16.4 us; B1
// H6/2 N3000, margin 8: 68 -> 49.6 us, but causal, where the second round is of lighter tiles, 39 -> 49).
bool few_query_tiles(const AttnArgs& a, const int ctas) { return (int64_t)a.B * a.Hq * ((a.Nq + 127) / 128) <= ctas; }

// CTAs of the persistent kernel: one per SM (registers and tensor memory allow exactly one) but for those left free
cudaError_t cta_count(const AttnArgs& a, int* ctas) {
  int sms = 0;
  const cudaError_t e = sm_count(&sms);
  *ctas = sms - a.sm_margin > 1 ? sms - a.sm_margin : 1;
  return e;
}

template <int D, bool kCausal, bool kPacked, bool kList>
cudaError_t launch(const AttnArgs& a, const int ctas, cudaStream_t stream) {
  using L = Smem<D>;
  const int Tq = (a.Nq + 127) / 128, Tk = (a.Nk + 127) / 128;
  CUtensorMap tq, tk, tv;
  const CUtensorMapSwizzle swz = D == 128 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
  if (!make_map(&tq, a.q_codes, (uint64_t)a.B * a.Hq * Tq * 128, D / 2, 128, swz)) return cudaErrorInvalidValue;
  if (!make_map(&tk, a.k_codes, (uint64_t)a.B * a.Hkv * Tk * 128, D / 2, 128, swz)) return cudaErrorInvalidValue;
  if (!make_map(&tv, a.vt_codes, (uint64_t)a.B * a.Hkv * Tk * D, 64, D, CU_TENSOR_MAP_SWIZZLE_64B))
    return cudaErrorInvalidValue;
  const int d_out = (a.d_out > 0 && a.d_out <= D) ? a.d_out : D;
  CUtensorMap to = tq;                       // only D=128 dense batches store through it
  int o_ndim = 1;
  if (!SAGE3_VARLEN_BUILD && D == 128 &&
      !make_out_map(&to, a.out, a.B, a.Hq, a.Nq, d_out, a.o_sb, a.o_sh, a.o_sn, &o_ndim))
    return cudaErrorInvalidValue;
  KParams P;
  P.q_sf = (const uint8_t*)a.q_sf; P.k_sf = (const uint8_t*)a.k_sf; P.vt_sf = (const uint8_t*)a.vt_sf;
  P.ds = (const __nv_bfloat16*)a.ds; P.out = (__nv_bfloat16*)a.out; P.lse = a.lse; P.lse_add = a.lse_add; P.status = a.status;
  P.o_sb = a.o_sb; P.o_sh = a.o_sh; P.o_sn = a.o_sn;
  P.B = a.B; P.Hq = a.Hq; P.Hkv = a.Hkv; P.Nq = a.Nq; P.Nk = a.Nk; P.Tq = Tq; P.Tk = Tk; P.ds_rows = a.ds_rows;
  P.scale_log2 = a.sm_scale * kLog2e;
  P.list_tiles = a.Hq / a.Hkv * Tq;
  P.per_item = few_query_tiles(a, ctas) ? 1 : 2;
  P.list_items = (P.list_tiles + P.per_item - 1) / P.per_item;
  P.o_token_first = o_ndim == 1;
  P.lam = a.k_lambda;
  P.slot_first = kPacked && a.slot_first != 0;
  P.d_out = d_out;
  // K-packing mode: Nk counts key slots; 16 slots hold 15 tokens, a partial group one slot more than its tokens
  P.Nk_log = kPacked ? (a.Nk / 16) * 15 + (a.Nk % 16 == 0 ? 0 : a.Nk % 16 - 1) : a.Nk;
#if SAGE3_VARLEN_BUILD
  P.cu_q = a.cu_q; P.cu_k = a.cu_k;
  P.order = a.order; P.n_order = a.n_order;
#endif
  auto kern = attn_fwd_kernel<D, kCausal, kPacked, kList>;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  // once per device and instantiation: opt in to the shared memory, and make sure the register hand-over inside the kernel
  // stays within the pool this build of it is launched with (it would block forever otherwise)
  static bool ready[64] = {};
  if (dev >= 64 || !__atomic_load_n(&ready[dev], __ATOMIC_ACQUIRE)) {
    cudaFuncAttributes fa;
    if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return e;
    if (fa.numRegs * kAttnThreads < 256 * RegSplit::softmax + 128 * (RegSplit::corr + RegSplit::role)) return cudaErrorLaunchOutOfResources;
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::total + 1024)) != cudaSuccess) return e;
    if (dev < 64) __atomic_store_n(&ready[dev], true, __ATOMIC_RELEASE);
  }
  const int64_t work = kList ? (int64_t)a.B * a.Hkv * P.list_items : (int64_t)a.B * a.Hq * ((Tq + 1) / 2);
  const int64_t grid = work < ctas ? work : ctas;
  return launch_pdl(kern, dim3((unsigned)grid), kAttnThreads, L::total + 1024, stream, a.after_delta_s, tq, tk, tv, to, P);
}

}  // namespace

#if SAGE3_VARLEN_BUILD
cudaError_t launch_attn_fwd_varlen(const AttnArgs& a, cudaStream_t stream) {
  // offsets come in pairs; no K-packing and no LSE for packed batches
  if (a.cu_q == nullptr || a.cu_k == nullptr || a.order == nullptr || a.n_order == nullptr || a.k_lambda != nullptr || a.lse != nullptr) return cudaErrorInvalidValue;
  int ctas;
  if (cudaError_t e = cta_count(a, &ctas); e != cudaSuccess) return e;
  if (a.D == 128) return a.causal ? launch<128, true, false, false>(a, ctas, stream) : launch<128, false, false, false>(a, ctas, stream);
  if (a.D == 64) return a.causal ? launch<64, true, false, false>(a, ctas, stream) : launch<64, false, false, false>(a, ctas, stream);
  return cudaErrorInvalidValue;
}
#else
cudaError_t launch_attn_fwd(const AttnArgs& a, cudaStream_t stream) {
  if (a.D != 128 && a.D != 64) return cudaErrorInvalidValue;
  int ctas;
  if (cudaError_t e = cta_count(a, &ctas); e != cudaSuccess) return e;
  if (a.k_lambda) {
    if (a.D == 128) return a.causal ? launch<128, true, true, false>(a, ctas, stream) : launch<128, false, true, false>(a, ctas, stream);
    return a.causal ? launch<64, true, true, false>(a, ctas, stream) : launch<64, false, true, false>(a, ctas, stream);
  }
  // Query tiles paired across the heads of a GQA group: where every head has an odd number of them, and the two of a pair
  // visit the same keys - one tile per head (decoding: B8 Hq32 Hkv8 Nk4096, 84 -> 62 us), or no causal mask.  (Kernels of
  // their own: the index arithmetic in the common ones cost those up to 5 %.)
  const int Tq = (a.Nq + 127) / 128;
  if ((a.Hq > a.Hkv && (Tq & 1) && (Tq == 1 || !a.causal)) || few_query_tiles(a, ctas)) {
    if (a.D == 128) return a.causal ? launch<128, true, false, true>(a, ctas, stream) : launch<128, false, false, true>(a, ctas, stream);
    return a.causal ? launch<64, true, false, true>(a, ctas, stream) : launch<64, false, false, true>(a, ctas, stream);
  }
  if (a.D == 128) return a.causal ? launch<128, true, false, false>(a, ctas, stream) : launch<128, false, false, false>(a, ctas, stream);
  return a.causal ? launch<64, true, false, false>(a, ctas, stream) : launch<64, false, false, false>(a, ctas, stream);
}

#endif

}  // namespace sage3
