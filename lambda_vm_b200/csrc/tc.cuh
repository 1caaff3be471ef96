// Asynchronous copies, and the tcgen05, TMEM and mbarrier primitives of the
// kernels that run byte products (kind::i8, u8 x u8 -> s32) on the tensor cores.
#pragma once
#include <stdint.h>

#include "wait.cuh"

namespace sg {
namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One bounded look at the barrier's phase: the thread sleeps until it
// completes, or for the hinted time (ns).
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(100000u)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t clock_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// The last wait of a CTA that leaves after a timeout: its products may still
// read shared memory and write TMEM, so they get two seconds more before both
// are given back.
static __device__ __noinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
    const uint32_t go_on = 0;
    bounded_wait([=] { return mbar_try(bar, parity); }, clock_ns, &go_on, WAIT_LIMIT_NS);
}
static __device__ __noinline__ void mbar_wait_slow(uint32_t bar, uint32_t parity, volatile uint32_t* abort, unsigned* err) {
    if (bounded_wait([=] { return mbar_try(bar, parity); }, clock_ns, abort, WAIT_LIMIT_NS)) return;
    *abort = 1;
    *(volatile unsigned*)err = 1;
}
// Wait for the barrier's phase, two seconds at most; on a timeout the CTA's
// abort word is set (every later wait then returns after one look and the CTA
// leaves the kernel at its next tile) and so is the context's error word.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort, unsigned* err) {
    if (!mbar_try(bar, parity)) mbar_wait_slow(bar, parity, abort, err);
}

// K-major operand without swizzle: 8 x 16-byte core matrices of 128 contiguous
// bytes; lbo: bytes between the two 16-byte K slices, sbo: between 8-row groups.
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}
// u8 x u8 -> s32, M = 128, N columns
__host__ __device__ constexpr uint32_t mma_idesc(uint32_t n) { return (2u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

// D (128 x n s32 at TMEM column d) (+)= A (128 rows) x B (n rows)^T over 32 K
// bytes; accumulate 0 starts a sum. The completion of all products issued by
// this thread arrives on `bar` after mma_commit.
__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t da, uint64_t db, uint32_t n, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(da), "l"(db), "r"(mma_idesc(n)), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 8 columns of this warp's 32 rows, complete on return.
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(addr)
        : "memory");
}

// One thread of a warp (the branch it guards is warp-uniform, so the
// descriptors stay in uniform registers).
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}

// 8 bytes from global to shared memory without registers; zeros when !valid.
__device__ __forceinline__ void copy_async8(uint32_t dst, const uint64_t* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Arrive on the barrier when this thread's copies so far have landed.
__device__ __forceinline__ void copy_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint64_t x, uint64_t y) {
    asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(addr), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t addr, uint64_t x) {
    asm volatile("st.shared.u64 [%0], %1;" ::"r"(addr), "l"(x) : "memory");
}

}  // namespace tc
}  // namespace sg
