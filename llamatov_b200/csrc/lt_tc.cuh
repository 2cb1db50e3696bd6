// Plumbing of the tensor-core kernels (tcgen05 + tensor memory + TMA): mbarriers with bounded waits, tiled loads,
// shared-memory operand descriptors, tensor-memory loads, the tensor-map encoder.
#pragma once
#include <cuda.h>

#include "lt_common.cuh"
#include "lt_wait.cuh"

namespace lt {
namespace tc {

constexpr long long WAIT_LIMIT = 3000000000LL;  // SM clocks (> 1 s) before a wait gives up

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait.  *abort_flag (shared) is set by the first wait of the CTA that runs out of time;
// from then on every wait returns immediately so that all roles run to the end of their loops.
template <int SLEEP_NS = 0>
__device__ __forceinline__ void mbar_wait(unsigned long long* bar, unsigned parity, volatile int* abort_flag,
                                          int* status) {
    if (mbar_try_wait(bar, parity)) return;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (SLEEP_NS > 0) __nanosleep(SLEEP_NS);
        if (*abort_flag) return;
        if (clock64() - t0 > WAIT_LIMIT) {
            *abort_flag = 1;
            atomicOr(status, LT_STATUS_WAIT_TIMEOUT);
            return;
        }
    }
}

// The same by shared address.  A wait whose barrier has completed still takes 90 clocks, so a role asks (bar_test) one step
// ahead and hands the answer to the wait, which then costs a branch.
__device__ __forceinline__ bool bar_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// suspended for up to a millisecond at a time: warps that poll take issue slots from the warps that work
__device__ __forceinline__ bool bar_sleep(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bar_wait(bool done, unsigned bar, unsigned parity, volatile int* abort_flag, int* status) {
    if (done) return;
    bounded_wait([&] { return bar_sleep(bar, parity); }, [] { return (long long)clock64(); }, WAIT_LIMIT, abort_flag, [&] {
        *abort_flag = 1;
        atomicOr(status, LT_STATUS_WAIT_TIMEOUT);
    });
}
// The wait of a whole warp for a place that it fills by bulk copies: false once a wait of the CTA has run out of time and the place is
// not free.  No copy is begun then, since what is in flight has to land before the CTA leaves.  (The flag is looked at where the
// place is not free at once: at every step it cost 28672 x 4096 x 32 3 %.)
__device__ __forceinline__ bool acquire(unsigned bar, unsigned parity, volatile int* abort_flag, int* status) {
    if (__all_sync(0xffffffffu, bar_test(bar, parity))) return true;
    bar_wait(false, bar, parity, abort_flag, status);
    return !__any_sync(0xffffffffu, *abort_flag != 0);
}

// One thread of a converged warp.  Roles whose single thread issues copies or MMAs run their loops as a warp and pick the
// thread at the instruction: counters and descriptors then stay in uniform registers, which those instructions read.
__device__ __forceinline__ bool elect_one() {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}
__device__ __forceinline__ void bar_arrive_if(bool yes, unsigned bar) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %0, 0;\n\t"
        "@p mbarrier.arrive.shared::cta.b64 _, [%1];\n\t}" ::"r"((unsigned)yes),
        "r"(bar)
        : "memory");
}
__device__ __forceinline__ void bar_arrive(unsigned bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void bar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_commit(unsigned bar) {   // arrives when the MMAs this thread has issued are complete
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// D[tmem] = A[smem] * B[smem], int8 x int8 -> int32, overwriting D
__device__ __forceinline__ void mma_i8(unsigned d_tmem, unsigned long long adesc, unsigned long long bdesc,
                                       unsigned idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc)
        : "memory");
}

// K-major shared-memory operand descriptor.  Rows are `row_bytes` apart inside an 8-row swizzle
// atom, atoms follow each other every 8*row_bytes (the stride byte offset); the leading byte
// offset is unused for swizzled K-major operands whose K extent fits the swizzle width.
template <int CB>
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr) {
    constexpr unsigned long long layout = CB == 4 ? 2ull : (CB == 2 ? 4ull : 6ull);  // 128B / 64B / 32B swizzle
    constexpr unsigned long long sbo = (8ull * CB * 32ull) >> 4;
    return (unsigned long long)((addr >> 4) & 0x3FFFu) | (1ull << 16) | (sbo << 32) | (1ull << 46) | (layout << 61);
}

template <int CW>
__device__ __forceinline__ void tmem_ld(unsigned taddr, int (&v)[CW]);
template <>
__device__ __forceinline__ void tmem_ld<4>(unsigned taddr, int (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(taddr));
}
template <>
__device__ __forceinline__ void tmem_ld<8>(unsigned taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
template <>
__device__ __forceinline__ void tmem_ld<16>(unsigned taddr, int (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
// Completes the TMEM loads of this thread.  The loaded registers are passed through the
// statement (eight at a time) so that no use of them can be scheduled above the wait.
__device__ __forceinline__ void reg_fence4(int* v) {
    asm volatile("" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3])::"memory");
}

// ---------------------------------------------------------------------------- host side

typedef CUresult (*encode_fn_t)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline encode_fn_t encode_fn() {
    static encode_fn_t fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = (encode_fn_t)p;
    }
    return fn;
}

}  // namespace tc
}  // namespace lt
