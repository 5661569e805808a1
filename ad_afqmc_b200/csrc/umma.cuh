// Blackwell (sm_100a) primitives: mbarriers with bounded waits, TMA tiled
// loads, TMEM allocation/loads and tcgen05.mma descriptors.
//
// Every wait on an mbarrier polls a bounded number of times; on timeout the
// caller receives false, records an error flag and unwinds (no trap, no
// endless spin).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace afq {

// ---------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t su32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile(
      "{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(su32(bar))
      : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(
          su32(bar)),
      "r"(bytes)
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(su32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: ~1e8 polls (each try_wait already suspends for a while).
constexpr uint32_t kMaxPolls = 1u << 27;

// The first poll stands apart from the loop: a wait on a barrier that is
// already complete then costs 41 cycles instead of 264 (one thread, per K block
// of the GEMMs' issue loop).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          uint32_t max_polls = kMaxPolls) {
  if (mbar_try_wait(bar, parity)) return true;
#pragma unroll 1
  for (uint32_t i = 1; i < max_polls; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// The waits of the GEMM kernels, called by whole warps.  A wait that runs out sets the
// error flag and the CTA's abort word; from then on every wait of the CTA that is
// not complete at once gives up too.
//  * mbar_wait_or_abort returns whether the barrier completed, the same in every lane (a
//    lane may see it complete while its neighbour polls on), so that the branch on it is
//    uniform.  The producers test it for every stage and stop at the first failure: a
//    barrier may not be armed again before its phase is over, nor a stage filled while
//    it is read.  The MMA warps test it once per accumulator.
//  * mbar_wait_run_on returns nothing.  The MMA warps use it per K block: an MMA on a stage that
//    was not filled harms nothing, and the test there cost the exchange 10 % and
//    a step 1 % (N = 200 and 300); the epilogue and FP64 consumer warps use it because
//    they meet at named barriers: they run on to their end over data that nobody uses.
// A role that issues ends with ring_drain, so that nothing lands in shared memory or
// TMEM that the CTA no longer owns.
static __device__ __noinline__ bool mbar_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort, int* err,
                                                   uint32_t max_polls) {
  for (uint32_t i = 0; i < max_polls; ++i) {
    if ((i & 1023) == 0 && *abort) return false;
    if (mbar_try_wait(bar, parity)) return true;
  }
  atomicExch(err, 1);
  *abort = 1;
  return false;
}
__device__ __forceinline__ bool mbar_wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort, int* err,
                                                   uint32_t max_polls = kMaxPolls) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) ok = mbar_wait_slow(bar, parity, abort, err, max_polls);
  return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void mbar_wait_run_on(uint64_t* bar, uint32_t parity, volatile int* abort, int* err) {
  if (!mbar_try_wait(bar, parity)) mbar_wait_slow(bar, parity, abort, err, kMaxPolls);
  __syncwarp();
}

// true in one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.u32 %0, 1, 0, P;\n}" : "=r"(p));
  return p != 0;
}

// A role's place in a ring of shared-memory stages.
struct Ring {
  uint64_t *full, *empty;  // per stage: filled, read
  int stages, stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance() {
    if (++stage == stages) {
      stage = 0;
      phase ^= 1;
    }
  }
};

// The producer's n next stages: one lane calls issue(stage, i) once the stage has been
// read.  False, with nothing more issued, once a wait fails.
template <class Issue>
__device__ __forceinline__ bool ring_fill(Ring& r, int n, volatile int* abort, int* err, Issue&& issue,
                                          uint32_t max_polls = kMaxPolls) {
  for (int i = 0; i < n; ++i) {
    if (!mbar_wait_or_abort(&r.empty[r.stage], r.phase ^ 1, abort, err, max_polls)) return false;
    if (elect_one()) issue(r.stage, i);
    __syncwarp();
    r.advance();
  }
  return true;
}

// The end of a role that issues: waits, whatever the abort word says, for the last round of
// `bars` (full: the producer's copies have landed; empty: the MMAs have read their
// stages).  Stages that were never used count as complete.
__device__ __forceinline__ void ring_drain(const Ring& r, uint64_t* bars) {
  Ring d = r;
  for (int s = 0; s < r.stages; ++s, d.advance()) mbar_wait(&bars[d.stage], d.phase ^ 1);
  __syncwarp();
}

// ---------------------------------------------------------------------------
// TMA (tiled, no multicast)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(su32(bar)), "r"(c0), "r"(c1)
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(su32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ---------------------------------------------------------------------------
// TMEM
// ---------------------------------------------------------------------------
// whole warp; writes the TMEM base address to *dst (shared memory)
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   su32(dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 32 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 columns of this thread's TMEM lane, load issued without waiting
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// wait for the issued TMEM loads; the destination registers pass through the
// wait so that no use of them is scheduled before it
__device__ __forceinline__ void tmem_wait_ld16x2(uint32_t (&r)[16], uint32_t (&q)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(q[0]), "+r"(q[1]),
                 "+r"(q[2]), "+r"(q[3]), "+r"(q[4]), "+r"(q[5]), "+r"(q[6]), "+r"(q[7]),
                 "+r"(q[8]), "+r"(q[9]), "+r"(q[10]), "+r"(q[11]), "+r"(q[12]), "+r"(q[13]),
                 "+r"(q[14]), "+r"(q[15])
               :
               : "memory");
}

// 16 columns of the accumulator, summing the second accumulator group (if
// any, BN columns further on) in FP32 round-to-nearest; both groups' loads
// are in flight together
__device__ __forceinline__ void acc_ld16(uint32_t taddr, int ngroups, int bn, float (&v)[16]) {
  uint32_t r[16], q[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) q[i] = 0u;
  tmem_ld16_issue(taddr, r);
  if (ngroups == 2) tmem_ld16_issue(taddr + bn, q);
  tmem_wait_ld16x2(r, q);
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
  if (ngroups == 2) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(q[i]);
  }
}

// ---------------------------------------------------------------------------
// tcgen05.mma (single CTA, A and B from shared memory)
// ---------------------------------------------------------------------------
// Instruction descriptor: dense, FP32 accumulate, A/B K-major.
// fmt: 1 = BF16 (kind::f16), 2 = TF32 (kind::tf32)
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, int fmt) {
  return (1u << 4)                      // D format F32
         | ((uint32_t)fmt << 7)         // A format
         | ((uint32_t)fmt << 10)        // B format
         | ((uint32_t)(N >> 3) << 17)   // N
         | ((uint32_t)(M >> 4) << 24);  // M
}

// Shared-memory matrix descriptor, K-major operand in the 128-byte swizzle layout written
// by TMA (rows of 128 bytes, 8-row atoms of 1024 bytes): low word the start address and the
// leading byte offset (unused, 1), both in 16 bytes; high word, the same for every operand,
// the stride byte offset 1024 / 16, the version (bit 14) and SWIZZLE_128B (2 << 29).
// 32-bit address arithmetic per MMA, which issues one MMA every ~50 cycles where
// 64-bit descriptors built from operand pointers took 66-80.
constexpr uint32_t kDescHi = (1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t saddr) { return (saddr >> 4) | (1u << 16); }
__device__ __forceinline__ void umma_bf16_lo(uint32_t dtmem, uint32_t alo, uint32_t blo,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %4, 0;\n"
      " mov.b64 da, {%1, %5};\n mov.b64 db, {%2, %5};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}" ::"r"(dtmem),
      "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
      : "memory");
}

// arrive on `bar` once all previously issued MMAs of this thread complete
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          su32(bar))
      : "memory");
}

}  // namespace afq
