// PTX wrappers shared by the tcgen05 convolution kernels: mbarriers with bounded waits,
// tcgen05 fences / commit, shared-memory operand descriptors, TF32 rounding.
#pragma once
#include "ssc_common.cuh"

namespace ssc {

constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false when the limit ran out or another thread already gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// Bounded wait used on the way out after another wait has already given up: it neither reads nor
// sets the abort flag.  Lets work that is still in flight (tensor-core instructions, bulk copies)
// finish before tensor memory is freed and the CTA exits.
__device__ __forceinline__ bool mbar_wait_drain(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < (kSpinLimit >> 2); ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    __nanosleep(64);
  }
  return false;
}
// Warp-collective bounded wait: lane 0 polls (one shared-memory access per poll instead of
// 32), the outcome is broadcast.  Must be called by all 32 lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, abort_flag) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  return ok != 0;
}
// Bounded waits for the roles that are NOT on the critical path: after a few polls the thread
// sleeps `ns` between polls, which leaves the issue slots and the barrier unit to the threads
// that are.  Same contract as mbar_wait / mbar_wait_warp.
__device__ __forceinline__ bool mbar_wait_backoff(uint32_t bar, uint32_t parity, volatile int *abort_flag, uint32_t ns) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (i >= 4u) __nanosleep(ns);
    if ((i & 255u) == 255u && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ bool mbar_wait_warp_backoff(uint32_t bar, uint32_t parity, volatile int *abort_flag, uint32_t ns) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait_backoff(bar, parity, abort_flag, ns) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  return ok != 0;
}
// Roles that issue tensor-core instructions run as a whole warp with warp-uniform control flow, and one elected
// lane issues: the instructions take their operands from uniform registers, and inside a branch on
// the lane number the compiler moves every operand there one by one - 150 cycles per tcgen05.mma
// whatever its size, against 39 (N = 16), 55 (N = 80) and 128 (N = 256) in this form.
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}
// Bounded wait of a whole warp; the result is a vote, i.e. warp-uniform.
__device__ __forceinline__ bool mbar_wait_uniform(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 1023u) == 1023u && __any_sync(0xffffffffu, *abort_flag)) return false;
  }
  *abort_flag = 1;
  return false;
}
// The same for a loop without a way out in the middle, which costs the issuing warp more than the wait itself: after a wait has
// failed the next ones look once, and fail too unless the barrier is ready.  What a loop still copies until its end goes to slots that nobody
// reads any more and is waited for, like all copies, before the CTA leaves.
__device__ __forceinline__ bool mbar_wait_straight(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  uint32_t i = 0;
  bool ok;
  do { ok = __all_sync(0xffffffffu, mbar_try_wait(bar, parity)); } while (!ok && ++i < kSpinLimit && !__any_sync(0xffffffffu, *abort_flag));
  if (!ok) *abort_flag = 1;
  return ok;
}
// Pairs of CTAs (a cluster of two): the address of the same place in CTA `rank`'s shared memory, the store that tells the other CTA
// something, and the wait that sees it (mbar_wait_straight at cluster scope).
//
// Why what the second CTA tells of is visible to the tensor core that the first one's issuing warp starts.  The rows of a slot
// are other warps' copies (cp.async) and a bulk copy of filters; all of them count on the slot's barrier in the second CTA
// when they have landed.  One warp there waits for that barrier, which orders them before what it does next, and then orders them
// for the async proxy (fence_async_smem).  Behind both, in program order, it issues st_async_v4: its 16 bytes count on the
// first CTA's barrier, and that completion is a release at cluster scope (PTX ISA, st.async).  The issuing warp's wait on that barrier acquires at cluster
// scope, and causality passes through a release and an acquire to everything the releasing side had seen, by whatever
// thread it was done.  tcgen05.fence::after_thread_sync then stands between that wait and the products, which read both CTAs' slots.  Accumulators
// go the same way: tcgen05.ld, tcgen05.wait::ld, tcgen05.fence::before_thread_sync, the warp's lanes together, the store.
// (A store and a released remote arrival say the same in two operations, at 2100 cycles a step.)
__device__ __forceinline__ uint32_t peer_address(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint4 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_wait_straight_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  uint32_t i = 0, got;
  bool ok;
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(got)
        : "r"(bar), "r"(parity)
        : "memory");
    ok = __all_sync(0xffffffffu, got != 0);
  } while (!ok && ++i < kSpinLimit && !__any_sync(0xffffffffu, *abort_flag));
  if (!ok) *abort_flag = 1;
  return ok;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 accumulator columns of the warp's 32 TMEM lanes (warp-collective; tcgen05.wait::ld before the values are used).
__device__ __forceinline__ void tmem_ld16(uint32_t *q, uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]),
        "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
// Two floats -> two fp16 in one word (lo = a), round to nearest even, finite overflow saturates.
__device__ __forceinline__ uint32_t pack_f16x2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
// Two floats -> two bf16 in one word (lo = a), round to nearest even.
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
// A 16-byte piece of a staged row: four channels as TF32, eight in 16 bits.
__device__ __forceinline__ uint4 stage_piece(float4 v) { return make_uint4(to_tf32(v.x), to_tf32(v.y), to_tf32(v.z), to_tf32(v.w)); }
__device__ __forceinline__ uint4 stage_piece_16(float4 a, float4 b, bool bf16) {
  return bf16 ? make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w))
              : make_uint4(pack_f16x2(a.x, a.y), pack_f16x2(a.z, a.w), pack_f16x2(b.x, b.y), pack_f16x2(b.z, b.w));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bulk asynchronous copy global -> shared; completes `bytes` on the mbarrier.  Both addresses
// 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// out[0..3] += v (one 16-byte reduction at L2; address 16-byte aligned)
__device__ __forceinline__ void red_add_v4(float *p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// Shared-memory operand descriptor split into its two 32-bit halves.  The high half is the same
// for every K-major, 128-byte-swizzled operand; the low half is (address >> 4) | (1 << 16), so
// stepping 32 bytes along K adds 2 and stepping to another slot adds (slot bytes >> 4).
// High half: stride of 1024 bytes between groups of eight rows, descriptor version 1 (sm_100), 128-byte swizzle.
constexpr uint32_t kDescHi = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }

// D[tmem] (+)= A[smem desc] * B[smem desc], accumulate selects += or =.
__device__ __forceinline__ void mma_tf32_ss(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %3, {%6, %6, %6, %6}, p;\n\t}"
      :
      : "r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHi), "r"(0u)
      : "memory");
}
// D[tmem] += A * B for the rows whose bit in `off` (x = rows 0-31 ... w = rows 96-127) is clear;
// rows whose bit is set keep their accumulator value (disable-output-lane mask).
__device__ __forceinline__ void mma_tf32_ss_masked(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint4 off) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %3, {%6, %7, %8, %9}, p;\n\t}"
      :
      : "r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(1u), "r"(kDescHi), "r"(off.x), "r"(off.y), "r"(off.z), "r"(off.w)
      : "memory");
}
// The same for a pair of CTAs, 256 rows: rows 0-127 (off) and half of B's rows in this one, the others at the same addresses in
// the second.
template <bool F16>
__device__ __forceinline__ void mma_pair_masked(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint4 off, uint4 off2) {
  if (F16)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, {%6, %7, %8, %9, %10, %11, %12, %13}, p;\n\t}" ::"r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc),
        "r"(1u), "r"(kDescHi), "r"(off.x), "r"(off.y), "r"(off.z), "r"(off.w), "r"(off2.x), "r"(off2.y), "r"(off2.z), "r"(off2.w)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], da, db, %3, {%6, %7, %8, %9, %10, %11, %12, %13}, p;\n\t}" ::"r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc),
        "r"(1u), "r"(kDescHi), "r"(off.x), "r"(off.y), "r"(off.z), "r"(off.w), "r"(off2.x), "r"(off2.y), "r"(off2.z), "r"(off2.w)
        : "memory");
}
// D (+)= A * B of a pair, all rows.
template <bool F16>
__device__ __forceinline__ void mma_pair(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  if (F16)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, {%6, %6, %6, %6, %6, %6, %6, %6}, p;\n\t}" ::"r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc),
        "r"(accumulate), "r"(kDescHi), "r"(0u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], da, db, %3, {%6, %6, %6, %6, %6, %6, %6, %6}, p;\n\t}" ::"r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc),
        "r"(accumulate), "r"(kDescHi), "r"(0u)
        : "memory");
}
// The pair's commit arrives on the barrier at this address in both CTAs.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// The same for fp16 operands (kind::f16, 16 elements = 32 bytes along K per instruction).
__device__ __forceinline__ void mma_f16_ss_masked(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint4 off) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%6, %7, %8, %9}, p;\n\t}"
      :
      : "r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(1u), "r"(kDescHi), "r"(off.x), "r"(off.y), "r"(off.z), "r"(off.w)
      : "memory");
}
// D[tmem] (+)= A * B with 16-bit operands (kind::f16: fp16 or bf16, chosen by the instruction
// descriptor), 16 elements = 32 bytes along K per instruction.
__device__ __forceinline__ void mma_f16_ss(uint32_t tmem_c, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%6, %6, %6, %6}, p;\n\t}"
      :
      : "r"(tmem_c), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHi), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async16_cg(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most n of this thread's most recent copy groups are still in flight.
__device__ __forceinline__ void cp_async_wait(int n) {
  switch (n) {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
    case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
  }
}
// All of the thread's copies, committed to a group or not (copies that arrive on a barrier by themselves never are).
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The two 16-byte pieces a lane copies of each of its four rows (none where `from` is negative), P bytes into the row; its part of the
// slot is eight rows on for each.  Predicated instead of branched around: the instructions around the copies are what the producers' time goes into.
template <int P>
__device__ __forceinline__ void copy_rows(const int *from, const char *const *at, uint32_t dst0, uint32_t dst1) {
#define SSC_ROW(I, OFF) \
  asm volatile( \
      "{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %0, 0;\n\t" \
      "@p cp.async.cg.shared.global [%1+%4], [%3+%5], 16;\n\t" \
      "@p cp.async.cg.shared.global [%2+%4], [%3+%6], 16;\n\t}" ::"r"(from[I]), "r"(dst0), "r"(dst1), "l"(at[I]), "n"(OFF), "n"(P), "n"(P + 64) \
      : "memory")
  SSC_ROW(0, 0);
  SSC_ROW(1, 1024);
  SSC_ROW(2, 2048);
  SSC_ROW(3, 3072);
#undef SSC_ROW
}
// The same where a piece may lie past the row's end: it is zero-filled then, and its (base, stride) lead somewhere valid.
template <int OFF>
__device__ __forceinline__ void copy_row_ends(int from, uint32_t dst0, uint32_t dst1, const char *base0, uint32_t stride0, uint32_t bytes0,
                                              const char *base1, uint32_t stride1, uint32_t bytes1) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ge.s32 p, %0, 0;\n\tmad.wide.u32 a, %0, %4, %3;\n\tmad.wide.u32 b, %0, %6, %5;\n\t"
      "@p cp.async.cg.shared.global [%1+%9], [a], 16, %7;\n\t"
      "@p cp.async.cg.shared.global [%2+%9], [b], 16, %8;\n\t}" ::"r"(from), "r"(dst0), "r"(dst1), "l"(base0), "r"(stride0),
      "l"(base1), "r"(stride1), "r"(bytes0), "r"(bytes1), "n"(OFF)
      : "memory");
}

}  // namespace ssc
