// Device helpers shared by the kernels that multiply packed INT4 rows on the tensor cores without
// dequantizing them (the one-token decode kernel and the 2..16-row block kernels): bulk copies into
// a warp's shared-memory slot with completion on the warp's mbarrier, and the slots' layout.
#pragma once

#include "ff_gemv_device.cuh"
#include "ff_internal.cuh"
#include "ff_tc_device.cuh"

namespace ff {

constexpr uint32_t kCopySpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- bulk copies into a warp's slot, completion on the warp's mbarrier -------------------------

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// 16-byte aligned source and destination, size a multiple of 16.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Called by the whole warp when it has used its slot's contents, before the next copies into the
// slot are requested.  The values read from the slot have been consumed by then (the arithmetic
// depends on them), so the reads are complete; the warp barrier orders every lane's reads before
// the requesting lane's next copy — the consumer-release / producer-acquire hand-off of a copy
// pipeline, with the warp barrier in place of the "empty" mbarrier.  (A proxy fence here would also
// wait for the warp's outstanding L2 prefetches.)
__device__ __forceinline__ void slot_release() { __syncwarp(); }
// Bounded wait for the warp's copies; flips the parity.  On running out the error flag is raised
// and the warp carries on (its rows are then wrong, the launch still ends).
static __device__ __noinline__ bool slot_wait_slow(uint32_t bar, uint32_t parity) {
    bool done = false;
    for (uint32_t i = 0; i < kCopySpinLimit && !done; ++i) done = mbar_try_wait(bar, parity);
    return done;
}
// (The first poll stands alone: a poll inside the bounded loop measured about 200 cycles on a
// barrier that was already complete, a stand-alone one 7.)
__device__ __forceinline__ void slot_wait(uint32_t bar, uint32_t &parity, uint32_t *errorFlag) {
    bool done = mbar_try_wait(bar, parity);
    if (!done) done = slot_wait_slow(bar, parity);
    if (!done && (threadIdx.x & 31) == 0) atomicExch(errorFlag, 10u);
    parity ^= 1u;
    __syncwarp();
}

__device__ __forceinline__ void named_barrier(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__host__ __device__ inline uint32_t pad16u(uint32_t bytes) { return (bytes + 15u) & ~15u; }
// Row-piece stride in a slot: at least `bytes`, a multiple of 16, and 32 or 96 modulo 128 so that
// the four tile rows a half-warp reads with 64-bit loads fall into different bank octets.
__host__ __device__ inline uint32_t piece_stride(uint32_t bytes) {
    uint32_t s = pad16u(bytes);
    while ((s & 127u) != 32u && (s & 127u) != 96u) s += 16u;
    return s;
}
}  // namespace ff
