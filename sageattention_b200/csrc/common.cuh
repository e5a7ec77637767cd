// Shared device helpers for the sm_100a kernels: numeric conversions that must match the
// reference's instruction forms bit for bit, and thin wrappers over the Blackwell PTX
// (mbarrier, TMA, tcgen05 / TMEM) used by the attention kernel.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sage3 {

// ---------------------------------------------------------------------------------------------
// Numerics.  The reference quantiser (sageattn4/quantization/fp4_quantization_4d.cu:224-251) is
// compiled with --use_fast_math, so `absmax / 6.0f` is div.approx.ftz, `1.0f / SF` is
// rcp.approx.ftz and the products are mul.ftz; the same PTX forms are issued here explicitly so
// that codes and scales come out bit-identical whatever flags this file is built with.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float div_approx_ftz(float a, float b) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float rcp_approx_ftz(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
// packed fp32x2 arithmetic: one issue slot for two elements, each rounded as by the scalar instruction
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}
__device__ __forceinline__ float2 mul2_ftz(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<uint64_t&>(d))
      : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
  return d;
}
__device__ __forceinline__ float ex2_approx(float a) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

constexpr float kNoMax = -1.0e30f;                     // row maximum where no key has been visible
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLog2Inv2688 = -11.392317422778762f;   // log2(1 / (448 * 6))  softmax_fused.h:33
constexpr float kLog2Inv6 = -2.584962500721156f;       // log2(1 / 6)          softmax_fused.h:34

// fp32 -> E4M3 (round to nearest even, saturate to 448); returns the byte.
__device__ __forceinline__ uint32_t f32_to_e4m3(float x) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(0.0f), "f"(x));
  return r & 0xFFu;
}
// two floats -> two E4M3 bytes, `lo` in bits 0-7
__device__ __forceinline__ uint32_t f32x2_to_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
// E4M3 byte -> fp32 (exact)
__device__ __forceinline__ float e4m3_to_f32(uint32_t b) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)b));
  return __half2float(__ushort_as_half((unsigned short)(h2 & 0xFFFFu)));
}

// 8 floats -> 8 E2M1 nibbles in one u32, element 0 in the lowest nibble
// (same operand order as fp32_vec_to_e2m1, fp4_quantization_4d.cu:77-99).
__device__ __forceinline__ uint32_t f32x8_to_e2m1x8(float a0, float a1, float a2, float a3,
                                                     float a4, float a5, float a6, float a7) {
  uint32_t v;
  asm("{\n"
      ".reg .b8 b0, b1, b2, b3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      "mov.b32 %0, {b0, b1, b2, b3};\n"
      "}"
      : "=r"(v)
      : "f"(a0), "f"(a1), "f"(a2), "f"(a3), "f"(a4), "f"(a5), "f"(a6), "f"(a7));
  return v;
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ float2 bf16x2_to_f32(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u)); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&p);
}
__device__ __forceinline__ uint32_t pack_bf16(float2 v) { return pack_bf16(v.x, v.y); }
// x - mean in fp32, rounded to bf16 (what a bf16 tensor subtraction does), for 8 channels; neg = -mean
__device__ __forceinline__ uint4 subtract_mean(const uint4& w, const float2 (&neg)[4]) {
  return make_uint4(pack_bf16(fadd2(bf16x2_to_f32(w.x), neg[0])), pack_bf16(fadd2(bf16x2_to_f32(w.y), neg[1])),
                    pack_bf16(fadd2(bf16x2_to_f32(w.z), neg[2])), pack_bf16(fadd2(bf16x2_to_f32(w.w), neg[3])));
}
// The same for a mean that is a bf16 value: the packed subtraction rounds the exact difference once.  Rounding to fp32 first, as above,
// never changes that: 24 bits of significand are at least twice 8 and 2 more, so the second rounding is harmless (Figueroa, "When is
// double rounding innocuous?", 1995); the formats share their exponents, so both overflow alike; and a difference below the
// normal numbers is a multiple of the smallest bf16 value, hence exact in both.
__device__ __forceinline__ uint4 subtract_mean(const uint4& w, const uint4& mean) {
  uint4 r;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r.x) : "r"(w.x), "r"(mean.x));
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r.y) : "r"(w.y), "r"(mean.y));
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r.z) : "r"(w.z), "r"(mean.z));
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r.w) : "r"(w.w), "r"(mean.w));
  return r;
}
__device__ __forceinline__ void add_channels(float2 (&acc)[4], const uint4& w) {
  acc[0] = fadd2(acc[0], bf16x2_to_f32(w.x)); acc[1] = fadd2(acc[1], bf16x2_to_f32(w.y));
  acc[2] = fadd2(acc[2], bf16x2_to_f32(w.z)); acc[3] = fadd2(acc[3], bf16x2_to_f32(w.w));
}
// Per half max(|a|, |b|), a NaN only where both are; the sign is of no meaning (xor of the two) until abs2 has cleared it.
__device__ __forceinline__ uint32_t habsmax2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t abs2(uint32_t a) { return a & 0x7fff7fffu; }

// Scale byte + reciprocal for one 16-element block whose absmax (a bf16 value) is `amax`
// (fp4_quantization_4d.cu:224-230).
__device__ __forceinline__ void block_scale(float amax, uint32_t& sf_byte, float& inv) {
  float sf = div_approx_ftz(amax, 6.0f);
  sf_byte = f32_to_e4m3(sf);
  float sfq = e4m3_to_f32(sf_byte);
  inv = (sfq == 0.0f) ? 0.0f : rcp_approx_ftz(sfq);
}

// Byte offset of the scale for (row, k16-block) inside a 512-byte "SF atom": 128 rows x 4 scales
// (= 64 elements of the contraction dim).  This is the order tcgen05.cp.32x128b.warpx4 moves
// into tensor memory for a block-scaled MMA: row r sits in lane r%32, 32-bit column r/32,
// byte = block index.
__host__ __device__ __forceinline__ int sf_atom_offset(int row, int blk4) {
  return (row & 31) * 16 + (row >> 5) * 4 + blk4;
}

// ---------------------------------------------------------------------------------------------
// PTX wrappers (sm_100a)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One look at an mbarrier phase, without parking.  (Measured on B200: 7 ns on an idle SM, 150 to 200 cycles beside a warp that
// keeps the special-function unit busy, so it is issued well before its result is needed; a failing try_wait of a whole warp returns after 4 us,
// with and without a suspend-time hint.  A parked thread resumes as soon as the phase completes.)
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: polls until the phase completes, at most `limit` times, and says whether it did.  The loop is one asm
// block of a handful of instructions: left to the compiler it was unrolled at every one of the kernels' many waits,
// and the instruction cache paid for it.  kWarp: by all 32 lanes of a warp, which leave it together and with the same answer,
// each poll being a vote.
// Returns 0, or kCode where the limit is reached.
template <bool kWarp, int kCode>
__device__ __forceinline__ int mbar_wait_or(uint32_t bar, uint32_t parity, uint32_t limit) {
  int fail;
#define SAGE3_WAIT(VOTE)                                                                        \
  "{\n.reg .pred p;\n.reg .b32 n;\nmov.b32 n, %3;\nPOLL:\n"                                    \
  "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n" VOTE                                \
  "@p bra DONE;\nadd.u32 n, n, -1;\nsetp.ne.u32 p, n, 0;\n@p bra POLL;\nDONE:\nselp.s32 %0, 0, %4, p;\n}"
  if constexpr (kWarp)
    asm volatile(SAGE3_WAIT("vote.sync.all.pred p, p, 0xffffffff;\n")
                 : "=r"(fail) : "r"(bar), "r"(parity), "r"(limit), "n"(kCode) : "memory");
  else
    asm volatile(SAGE3_WAIT("") : "=r"(fail) : "r"(bar), "r"(parity), "r"(limit), "n"(kCode) : "memory");
#undef SAGE3_WAIT
  return fail;
}
template <bool kWarp = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  return mbar_wait_or<kWarp, 1>(bar, parity, limit) == 0;
}

// Bounded wait of a whole warp of one of the kernels' roles: 0, or kCode where it ran out.  Then the caller leaves its loops, calls
// give_up with that code and unwinds instead of hanging the SM.  (The code comes out of the instruction that told success from
// failure, so knowing which wait it was costs nothing.)
//
// The warp goes on to warp-wide instructions (tcgen05.ld / st, __syncwarp), so it must never split on a wait that ran out for
// some of its lanes only: each poll is a vote.  That also lets the compiler treat the loops as uniform, without the code that
// brings diverged lanes together again.
//
// The limit.  A failing poll takes 80 ns (a busy CTA) to 4 us (a parked warp): the default gives up after 0.02 to 1.05
// seconds, where the longest wait of a working kernel is some 10 us.  A warp that waits does not look whether another
// has given up: all of them wait for one another, so each runs out its own limit at about the same time, and that is why it
// is not longer.
template <int kCode, uint32_t kPolls = (1u << 18)>
__device__ __forceinline__ int wait_bar(uint32_t bar, uint32_t parity) {
  return mbar_wait_or<true, kCode>(bar, parity, kPolls);
}

// The same as a loop that the compiler sees, so that it knows the answer to be the warp's, and with a suspend-time hint: for
// the QK issuer (all four forms measured for each role, within 1 % of one another; this one was the best over all shapes).
template <int kCode>
__device__ __forceinline__ int wait_bar_uniform(uint32_t bar, uint32_t parity) {
#pragma unroll 1
  for (uint32_t n = 1u << 18; n != 0; --n) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    if (__all_sync(0xffffffffu, ok)) return 0;
  }
  return kCode;
}

// A wait of this warp ran out: raises the CTA's abort flag and records its code in *status (first writer wins).
__device__ __forceinline__ void give_up(volatile int* abort_s, int* status, int code) {
  *abort_s = 1;
  atomicCAS(status, 0, code);
}

// Programmatic dependent launch: let the next kernel of the stream start its prologue / wait until the previous one is
// complete and its writes are visible.  Both do nothing in a kernel that was launched without the attribute.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 16 bytes global -> shared without a register in between; zeros if !valid
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// shared -> global tile store through a 4-D tensor map (rows outside the tensor are clipped by the hardware);
// completion is tracked in bulk groups of the issuing thread
__device__ __forceinline__ void tma_store_4d(const void* tmap, uint32_t src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
               :: "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(w), "r"(src) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
               :: "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(src) : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// all bulk groups of this thread have finished READING shared memory (their source may be reused)
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar) : "memory");
}
// plain bulk copy global -> shared (16-byte aligned addresses and size)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// --- tensor memory / tcgen05 ---
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// One lane of the (whole) warp, always the same one.  The compiler knows that one lane is left where this is the condition, and
// issues the tcgen05 instructions there as they are; behind `lane == 0` it takes 730 instead of 380 cycles to issue the copies and
// MMAs of a score tile, 520 instead of 210 for those of P.V (B2 H16 N4100 Nk333 D96 58.0 -> 56.2 us, 16 prompts 478 -> 457).
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(r));
  return r != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 lanes x 16 columns of 32-bit values from registers into tensor memory; tmem_wait_st() before a load
// of the same columns
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
         "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 4 words of this thread's TMEM lane (e.g. 32 FP4 codes of an A operand kept in tensor memory).
__device__ __forceinline__ void tmem_st4(uint32_t taddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" :: "r"(taddr), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Operations on operands in shared memory take each 64-bit descriptor as (low word, high word): the issuing thread then only
// does 32-bit adds on the low word.
// 32 rows x 16 bytes of scale factors: shared -> tensor memory, replicated into all four
// 32-lane quarters (what block-scaled MMAs expect).
__device__ __forceinline__ void tc_cp_sf(uint32_t taddr, uint32_t lo, uint32_t hi) {
  asm volatile("{\n.reg .b64 d;\nmov.b64 d, {%1, %2};\ntcgen05.cp.cta_group::1.32x128b.warpx4 [%0], d;\n}"
               ::"r"(taddr), "r"(lo), "r"(hi) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], E2M1 operands with one UE4M3 scale per 16 elements, K = 64.
__device__ __forceinline__ void tc_mma_nvf4(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                            uint32_t idesc, uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 da, db;\n"
      "setp.ne.b32 p, %6, 0;\nmov.b64 da, {%1, %2};\nmov.b64 db, {%3, %4};\n"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], da, db, %5, [%7], [%8], p;\n}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// The same with the A operand in tensor memory: lane = row, 8 columns per K block of 64, word c of a lane = the row's
// codes 8c ... 8c+7 (low nibble first) - the byte order of the shared-memory operand.
__device__ __forceinline__ void tc_mma_nvf4_ta(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                               uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 db;\n"
      "setp.ne.b32 p, %5, 0;\nmov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], [%1], db, %4, [%6], [%7], p;\n}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], bf16 operands, K = 16.
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 da, db;\n"
      "setp.ne.b32 p, %6, 0;\nmov.b64 da, {%1, %2};\nmov.b64 db, {%3, %4};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// A shared-memory descriptor's low word: address >> 4, leading offset >> 4 in bits 16 on (the distance between the two 16-byte
// K chunks where there is no swizzle, 1 else); its high word: distance between groups of 8 rows >> 4, version 1 in bit 14,
// swizzle from bit 29 (0 none, 6 = 32 bytes, 4 = 64, 2 = 128).

// Instruction descriptor for kind::mxf4nvf4, scale_vec::4X: E2M1 x E2M1 -> fp32, UE4M3 scales,
// both operands K-major, M x N tile, K = 64.
__host__ __device__ constexpr uint32_t make_idesc_nvf4(int M, int N) {
  return (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | (0u << 23) | ((uint32_t)(M >> 4) << 24);
}
// Instruction descriptor for kind::f16 with bf16 operands, fp32 accumulate, K-major A and B.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// 32 consecutive fp32 columns of this thread's TMEM lane -> registers.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}

}  // namespace sage3
