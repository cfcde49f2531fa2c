// TMA and mbarrier primitives of the time-step kernels (sm_100a): bounded waits, box
// loads into shared memory and prefetches into L2. No cluster multicast is used.
#pragma once
#include <cuda.h>

#include <stdint.h>

namespace ifosb {

__device__ __forceinline__ uint32_t su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Bounded wait: gives up after `limit_ns` of wall time (1 s unless a test lowers
// it; a TMA box lands in microseconds).
__device__ __forceinline__ bool mbar_wait(uint64_t *b, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try(b, parity)) return true;
    const uint64_t t0 = gtimer();
    while (!mbar_try(b, parity))
        if (gtimer() - t0 > limit_ns) return false;
    return true;
}
constexpr uint64_t WAIT_LIMIT_NS = 1000000000ull;
__device__ __forceinline__ void tma_load5(void *dst, const CUtensorMap *m, int c0, int c1, int c2, int c3, int c4,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(su32(dst)),
        "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(su32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load4(void *dst, const CUtensorMap *m, int c0, int c1, int c2, int c3, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(su32(dst)),
        "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(su32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load3(void *dst, const CUtensorMap *m, int c0, int c1, int c2, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(su32(dst)),
        "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(su32(bar))
        : "memory");
}

// L2 prefetch of a box (no shared memory, no completion): warms L2 for a later load.
__device__ __forceinline__ void tma_prefetch5(const CUtensorMap *m, int c0, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.prefetch.tensor.5d.L2.global.tile [%0, {%1, %2, %3, %4, %5}];" ::"l"(m), "r"(c0), "r"(c1),
                 "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
}
__device__ __forceinline__ void tma_prefetch3(const CUtensorMap *m, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(m), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void tma_prefetch4(const CUtensorMap *m, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(m), "r"(c0), "r"(c1), "r"(c2),
                 "r"(c3)
                 : "memory");
}

// Tensor-map coordinates of a cell: z index k+7, row i+1, plane j+2.
__device__ __forceinline__ int zc(int k) { return k + 7; }
__device__ __forceinline__ int xc(int i) { return i + 1; }
__device__ __forceinline__ int yc_(int j) { return j + 2; }

// Programmatic dependent launch: a kernel of the time loop may let its successor's CTAs
// take their places before it ends (all of its own have called pdl_release or ended),
// and waits itself, before it touches anything the loop writes, until its predecessor
// has finished and its writes are visible. Without the launch attribute both are no-ops.
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Failure-path test knobs: the mbarrier wait limit, and the box of a chunk from which
// on a CTA issues no more loads (-1 = never); the waits for boxes never issued run out.
struct WaitCtl {
    uint64_t limit_ns;
    int stop_it;
};

}  // namespace ifosb
