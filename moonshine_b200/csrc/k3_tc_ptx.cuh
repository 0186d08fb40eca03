// Inline-PTX wrappers for the Blackwell (sm_100a) pieces the grouped GEMM uses:
// mbarriers, TMA tiled loads (no cluster forms), tensor memory allocation,
// tcgen05 MMA / commit / load, and the proxy fences between them.
#pragma once

#include "k3_common.cuh"

namespace k3::tc {

K3_DEVINL uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// ---------------------------------------------------------------- one thread of a warp
// TMA, MMA and commit instructions take their operands from uniform registers.  A branch on
// lane == 0 does not tell the compiler that one thread runs it; elect.sync does, in a warp whose
// index is the same in all lanes for the compiler too (warp_index).  Measured, one thread issuing
// back to back, lane == 0 / elected: block-scaled MMA of N = 16 31 / 23 ns, N = 64 33 / 28, N = 128 39 / 36;
// TMA box of 64 x 32 bf16 32 to 62 / 19 to 43 (by boxes per stage).  Branches on run-time
// values between the instructions cost as much again (N = 128 57 ns), so issue loops are straight-line.
K3_DEVINL uint32_t warp_index() { return __shfl_sync(0xffffffffu, threadIdx.x / kWarp, 0); }

// true in one lane of a converged warp, the same lane each time
K3_DEVINL bool elect_one() {
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    return elected != 0u;
}

// ------------------------------------------------------------------ mbarrier
K3_DEVINL void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

K3_DEVINL void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

K3_DEVINL void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

K3_DEVINL bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// has the phase of this parity completed? (does not wait)
K3_DEVINL bool mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: gives up two seconds after it started (wall clock of the
// device) or as soon as another thread of the CTA gave up (abort_flag in shared
// memory).  Returns false on give-up.
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

K3_DEVINL unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

K3_DEVINL bool mbar_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag,
                         unsigned long long limit_ns = kWaitLimitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_timer_ns();
    for (uint32_t spin = 1;; spin++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 63u) == 0u) {
            if (*abort_flag != 0u) return false;
            if (global_timer_ns() - t0 > limit_ns) break;
        }
    }
    *abort_flag = 1u;
    return false;
}

K3_DEVINL void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// generic-proxy writes to shared memory -> visible to the async proxy (MMA, TMA)
K3_DEVINL void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------- TMA
K3_DEVINL void prefetch_tensormap(const void *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// 2-D tiled load global -> shared of this CTA, completion on an mbarrier.
K3_DEVINL void tma_load_2d(void *dst, const void *map, uint64_t *bar, int32_t x, int32_t y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// L2 policy for data that is read once (a weight stream): its lines are the first to be
// replaced, so the stream does not push out what other kernels left in L2 - in particular
// not lines that would have to be written back first.
K3_DEVINL uint64_t l2_policy_evict_first() {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    return policy;
}

// tma_load_2d with an L2 cache policy
K3_DEVINL void tma_load_2d_hint(void *dst, const void *map, uint64_t *bar, int32_t x, int32_t y, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
        "[%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(policy)
        : "memory");
}

// 2-D tiled prefetch global -> L2 only (no shared-memory destination, no barrier).
K3_DEVINL void tma_prefetch_2d(const void *map, int32_t x, int32_t y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y)
                 : "memory");
}

// ------------------------------------------------------------- asynchronous copies
// kBytes (8 or 16) global -> shared memory of one thread, both aligned to them
template <uint32_t kBytes>
K3_DEVINL void cp_async(void *dst, const void *src) {
    if constexpr (kBytes == 16u) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    } else {
        static_assert(kBytes == 8u, "8 or 16 bytes");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
    }
}
// one arrival of this thread on `bar` (counted in its initial value) when its copies so far are done
K3_DEVINL void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
K3_DEVINL void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// -------------------------------------------------------------- tensor memory
K3_DEVINL void tmem_alloc(uint32_t *dst_smem, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(dst_smem)),
                 "r"(columns)
                 : "memory");
}

K3_DEVINL void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

K3_DEVINL void tmem_dealloc(uint32_t taddr, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns)
                 : "memory");
}

K3_DEVINL void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

K3_DEVINL void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc], kind::f16 (bf16 inputs, fp32 accumulate)
K3_DEVINL void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// mbarrier arrives once every MMA issued so far by this thread has completed
K3_DEVINL void mma_commit(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// 32 lanes x 32 consecutive fp32 columns: thread i of the warp receives lane
// (base lane + i), registers r[0..31] = columns c..c+31.
K3_DEVINL void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

K3_DEVINL void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------- descriptors
// Shared-memory matrix descriptor of a K-major bf16 tile stored as 8-row x
// 128-byte atoms with the 128-byte swizzle (what a TMA load with
// CU_TENSOR_MAP_SWIZZLE_128B of a {64 elements, rows} box writes):
//   bits [0,14)  start address >> 4        bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4   bits [46,48) descriptor version (1)
//   bits [61,64) layout: 2 = 128-byte swizzle
// Stride between consecutive 8-row atoms is 1024 bytes; the leading offset is
// not used by swizzled K-major layouts.
K3_DEVINL uint64_t make_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor, kind::f16: D fp32, A and B bf16, both K-major.
//   bits [4,6) D format (1 = f32)   bits [7,10) A format (1 = bf16)
//   bits [10,13) B format           bit 15 / 16 A / B major (0 = K)
//   bits [17,23) N >> 3             bits [24,29) M >> 4
K3_DEVINL constexpr uint32_t make_idesc_bf16(uint32_t m, uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

}  // namespace k3::tc
