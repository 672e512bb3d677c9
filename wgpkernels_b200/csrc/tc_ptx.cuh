// Inline-PTX wrappers of the sm_100a machinery the INT8 GEMM is built from: mbarriers with bounded waits, TMA tile loads (never with
// cluster multicast), tensor-memory allocation, tcgen05.mma kind::i8 with its shared-memory and instruction descriptors, tcgen05.ld / st.
#pragma once
#include "common.cuh"

namespace wq {

constexpr int kBM = 128;             // rows of a tile = tensor-memory lanes
constexpr int kStageK = 128;         // bytes (= INT8 elements) of K per stage: one 128-byte swizzle row, one scale block
constexpr int kMmaK = 32;            // K of one tcgen05.mma kind::i8
constexpr int kTmemColumns = 512;    // all of an SM's tensor memory (one CTA per SM)

WQ_DEVICE uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// The warp's number as a value the compiler knows to be the same in all lanes, and one lane of a converged warp (the same one every time).  A role
// that issues TMA or tensor-core instructions runs its loop with the whole warp and only the issue under elect_one(): its loop variables and
// descriptors then live in uniform registers, from which these instructions take their operands.  In a loop that lane 0 runs alone every
// operand is moved there first, at each instruction, on issue slots that the drain warps want.  Measured, loops of lane 0 -> this form (GEMM alone):
// exact+g 32768 x 5120 x 5120 2007 -> 1678 us, block 1393 -> 1126 (128-channel tiles), row 557 -> 550.
WQ_DEVICE int uniform_warp() { return __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0); }
WQ_DEVICE bool elect_one() {
    uint32_t elected;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(elected));
    return elected != 0;
}

WQ_DEVICE void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
WQ_DEVICE void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
WQ_DEVICE void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// One potentially blocking test of the phase: the hardware may suspend the thread for up to `kSuspendNs` (it resumes as soon as the
// phase completes), so a waiting role does not spend its scheduler's issue slots on polling.
constexpr uint32_t kSuspendNs = 4000;
WQ_DEVICE bool mbar_test(uint32_t bar, uint32_t parity);
WQ_DEVICE bool mbar_try_wait(uint32_t bar, uint32_t parity) {
#ifdef WQ_WAIT_SPIN
    return mbar_test(bar, parity);
#endif
    uint32_t done;
#ifdef WQ_WAIT_NOHINT
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
#endif
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(kSuspendNs)
        : "memory");
    return done != 0;
}
// Non-blocking test of the phase: the cheap first look (the phase has usually completed by the time a role asks).
WQ_DEVICE bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Waits for the phase of `parity`, for roughly `limit` clocks at most; false when the CTA is aborting or the wait ran out (then `code`
// is recorded in `status` and the abort flag raised).  The common case costs one try_wait (which parks the thread in hardware) and a
// branch; the clock and the abort flag are only looked at every 32 unsuccessful tries.
WQ_DEVICE bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code, int* status, long long limit) {
    long long start = 0;
    for (uint32_t spin = 1;; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 31u) == 0u) {
            if (*abort_flag) return false;
            const long long now = clock64();
            if (spin == 32u) start = now;
            if (now - start > limit) {
                *abort_flag = code;
                atomicCAS(status, 0, code);
                return false;
            }
        }
    }
}

// A warp leaves a role as one.  Lanes that decided for themselves could part on an abort: one leaves for the CTA's last barrier, the others wait
// for it wherever the warp meets next, for ever.  And every lane has looked at a phase before the warp acts on it: what is issued lets the
// barrier go on, and a lane that looked a whole phase later would take its parity for one that has yet to complete.  So a role votes on a
// wait (or, where only one lane waits, on what came of it),
WQ_DEVICE bool whole_warp(bool ok) { return __all_sync(0xffffffffu, ok); }
// or, where the vote costs too much (the MMA issuers: `exact` on 64 x 5120 x 5120 20.7 -> 21.8 us), the warp meets with __syncwarp() behind the
// waits of every step, and a lane that gave up keeps coming to the meetings of the steps that are left.
WQ_DEVICE void keep_meeting(int steps) {
#pragma unroll 1
    for (; steps > 0; --steps) __syncwarp();
}

// An aborting producer: waits for the last copies it issued into each of its stages, so that shared memory is not given back under them.
// Bit s of `fills`: parity of the number of fills issued into stage s; the last one completes the phase of the opposite parity (on a barrier
// without a fill that phase counts as completed).  At most kLandLimit clocks (a millisecond, against the microseconds of a copy) a stage.
constexpr long long kLandLimit = 2000000;
WQ_DEVICE void await_issued_fills(uint32_t bar_full, int stages, uint32_t fills) {
    for (int s = 0; s < stages; ++s) {
        const long long start = clock64();
        while (!mbar_try_wait(bar_full + 8 * s, ((fills >> s) & 1u) ^ 1u) && clock64() - start < kLandLimit) {}
    }
}

WQ_DEVICE void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map),
                 "r"(bar), "r"(x), "r"(y)
                 : "memory");
}
// ---- CTA pairs (clusters of two): one MMA works on both CTAs' tensor memory and shared memory (cta_group::2) -------------------------
WQ_DEVICE uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
WQ_DEVICE uint32_t cluster_size() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return n;
}
// the address of this CTA's shared-memory location `address` in CTA `rank` of the cluster
WQ_DEVICE uint32_t in_cta(uint32_t address, uint32_t rank) {
    uint32_t mapped;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(mapped) : "r"(address), "r"(rank));
    return mapped;
}
WQ_DEVICE void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrival on a barrier of another CTA of the cluster
WQ_DEVICE void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// a tile into this CTA's shared memory, its bytes counted on a barrier of either CTA of the pair (no multicast)
WQ_DEVICE void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(map), "r"(cluster_bar), "r"(x), "r"(y)
                 : "memory");
}
WQ_DEVICE void prefetch_tensormap(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }

WQ_DEVICE void tmem_alloc(uint32_t slot_in_smem, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_in_smem), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
WQ_DEVICE void tmem_dealloc(uint32_t address, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
WQ_DEVICE void tmem_alloc_pair(uint32_t slot_in_smem, uint32_t columns) {  // by one warp of each CTA of the pair
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_in_smem), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
WQ_DEVICE void tmem_dealloc_pair(uint32_t address, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
WQ_DEVICE void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
WQ_DEVICE void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// The mbarrier is arrived on once every tcgen05 operation this thread issued before has completed.
WQ_DEVICE void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// The same for the MMAs of a pair: the barrier at this offset of BOTH CTAs is arrived on.
WQ_DEVICE void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(uint16_t(3))
                 : "memory");
}
// One MMA of a pair: A = 128 rows of each CTA, B = N / 2 rows of each CTA, D = 128 lanes x N columns in each CTA's tensor memory.
WQ_DEVICE void mma_i8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// D (tensor memory, 128 lanes x N columns of INT32) = or += A (128 x 32 INT8, smem) * B (N x 32 INT8, smem)^T
WQ_DEVICE void mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Consecutive columns of this thread's lane (a warp reads the 32 lanes of its quarter of tensor memory).
#define WQ_R4(a, i) "=r"(a[i]), "=r"(a[i + 1]), "=r"(a[i + 2]), "=r"(a[i + 3])
WQ_DEVICE void tmem_load_32(uint32_t taddr, int* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : WQ_R4(v, 0), WQ_R4(v, 4), WQ_R4(v, 8), WQ_R4(v, 12), WQ_R4(v, 16), WQ_R4(v, 20), WQ_R4(v, 24), WQ_R4(v, 28)
        : "r"(taddr)
        : "memory");
}
WQ_DEVICE void tmem_load_16(uint32_t taddr, int* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : WQ_R4(v, 0), WQ_R4(v, 4), WQ_R4(v, 8), WQ_R4(v, 12)
                 : "r"(taddr)
                 : "memory");
}
WQ_DEVICE void tmem_load_8(uint32_t taddr, int* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : WQ_R4(v, 0), WQ_R4(v, 4) : "r"(taddr) : "memory");
}
#undef WQ_R4
// Completes the loads issued before it.  The wait has no operands that say so: whatever reads the registers has to come after
// tmem_loaded(registers) as well, or the compiler may convert a value before the wait that makes it valid (it did, with the last columns of a
// chunk, where registers were short; whether that shows depends on how long the load happens to take).
WQ_DEVICE void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
#define WQ_RW4(a, i) "+r"(a[i]), "+r"(a[i + 1]), "+r"(a[i + 2]), "+r"(a[i + 3])
template <int N> WQ_DEVICE void tmem_loaded(int (&v)[N]) {
    static_assert(N == 1 || N == 8 || N == 16 || N == 32, "the registers of one load");
    if constexpr (N == 8) asm volatile("" : WQ_RW4(v, 0), WQ_RW4(v, 4)::"memory");
    if constexpr (N == 16) asm volatile("" : WQ_RW4(v, 0), WQ_RW4(v, 4), WQ_RW4(v, 8), WQ_RW4(v, 12)::"memory");
    if constexpr (N == 32)
        asm volatile("" : WQ_RW4(v, 0), WQ_RW4(v, 4), WQ_RW4(v, 8), WQ_RW4(v, 12), WQ_RW4(v, 16), WQ_RW4(v, 20), WQ_RW4(v, 24), WQ_RW4(v, 28)::"memory");
}
#undef WQ_RW4

// Shared-memory operand descriptor: K-major rows of 128 bytes, 128-byte swizzle, 8-row groups 1024 bytes apart.
WQ_DEVICE uint64_t smem_descriptor(uint32_t address) {
    uint64_t d = (address & 0x3ffffu) >> 4;       // start address, 16-byte units
    d |= uint64_t(1) << 16;                       // leading byte offset (unused for swizzled K-major layouts)
    d |= uint64_t(1024 >> 4) << 32;               // stride byte offset between 8-row groups
    d |= uint64_t(1) << 46;                       // descriptor version of sm_100
    d |= uint64_t(2) << 61;                       // 128-byte swizzle
    return d;
}
// Instruction descriptor: INT32 accumulator, signed INT8 A and B, both K-major, M = m (256 for a pair of CTAs), N = n.
__host__ __device__ constexpr uint32_t instruction_descriptor(int n, int m = kBM) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

}  // namespace wq
