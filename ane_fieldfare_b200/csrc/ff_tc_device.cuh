// Device wrappers shared by the tensor-core GEMMs (INT4 and INT8 weights): bounded mbarrier waits, TMA
// loads, tcgen05 loads, stores, MMAs and commits, for one CTA and for a pair; and the driver's tensor
// map encoder.
#pragma once

#include "ff_internal.cuh"

namespace ff {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- tcgen05 / TMA / mbarrier wrappers ------------------------------------------------------

constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// How a wait orders what follows it: kLocal, acquire at CTA scope, where threads or copies of this CTA signal the
// barrier; kPair, relaxed at cluster scope, where the other CTA of a pair or the MMAs of both do: what they hand over
// is tensor memory, which the tcgen05 fences on either side order, or stages that completed MMAs have read.  (An
// acquire at cluster scope in one warp's loop costs the whole CTA 4 to 10 % of a GEMM.)
enum class Order { kLocal, kPair };
#define FF_MBAR_POLL(instruction)                             \
    asm volatile(                                             \
        "{\n"                                                 \
        ".reg .pred p;\n" instruction " p, [%1], %2;\n"       \
        "selp.u32 %0, 1, 0, p;\n"                             \
        "}\n"                                                 \
        : "=r"(ok)                                            \
        : "r"(bar), "r"(parity)                               \
        : "memory")
template <Order kOrder = Order::kLocal>
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if (kOrder == Order::kLocal) FF_MBAR_POLL("mbarrier.try_wait.parity.shared::cta.b64");
    else FF_MBAR_POLL("mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64");
    return ok != 0;
}
// one look, without the suspension that a try_wait may take
template <Order kOrder = Order::kLocal>
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    if (kOrder == Order::kLocal) FF_MBAR_POLL("mbarrier.test_wait.parity.shared::cta.b64");
    else FF_MBAR_POLL("mbarrier.test_wait.parity.relaxed.cluster.shared::cta.b64");
    return ok != 0;
}
#undef FF_MBAR_POLL
// Bounded wait.  Returns false when the limit ran out or another thread of the CTA gave up; the
// caller leaves its loop.  `abortFlag` lives in shared memory.  kSleep: pause between polls, for
// the warps whose polling would otherwise take issue slots from the dequantizing warps.
// The first poll stands alone in front of the loop: measured on the device, a wait that finds its
// barrier already complete costs 7 cycles this way and about 200 when the poll sits inside the
// bounded loop.
template <bool kSleep, Order kOrder>
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile uint32_t *abortFlag) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_wait<kOrder>(bar, parity)) return true;
        if (kSleep) __nanosleep(40);
        if ((i & 255u) == 255u && *abortFlag) return false;
    }
    *abortFlag = 1u;
    return false;
}
template <Order kOrder = Order::kLocal>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t *abortFlag) {
    return mbar_try_wait<kOrder>(bar, parity) || mbar_wait_slow<false, kOrder>(bar, parity, abortFlag);
}
template <Order kOrder = Order::kLocal>
__device__ __forceinline__ bool mbar_wait_idle(uint32_t bar, uint32_t parity, volatile uint32_t *abortFlag) {
    return mbar_try_wait<kOrder>(bar, parity) || mbar_wait_slow<true, kOrder>(bar, parity, abortFlag);
}

// Box of a map at (x, y[, z]) into shared memory (128-byte aligned); x times the element's size a multiple of 16.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                            int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 32 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tc_load_32cols(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 16 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tc_load_16cols(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// 16 lanes x 32 fp32 columns: r[4 j + i] is lane l / 4 (i < 2) or l / 4 + 8, column 8 j + 2 (l % 4) + i % 2,
// for the warp's lane l.
__device__ __forceinline__ void tc_load_16x32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major bf16 tile stored with the 128-byte swizzle:
// rows are 128 bytes apart, groups of eight rows 1024 bytes apart (stride byte offset), the
// leading byte offset is unused for swizzled K-major tiles (set to 1), descriptor version 1,
// layout type 2 (128-byte swizzle).  The tile base must be 1024-byte aligned; `byteOffset`
// advances along K inside the swizzle atom (32 bytes per K=16 slice).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smemAddr) {
    uint64_t desc = (uint64_t)((smemAddr & 0x3FFFFu) >> 4);
    desc |= (uint64_t)1 << 16;
    desc |= (uint64_t)(1024 >> 4) << 32;
    desc |= (uint64_t)1 << 46;
    desc |= (uint64_t)2 << 61;
    return desc;
}
// Instruction descriptor: fp32 accumulate, bf16 A and B, both K-major, M = 256 (128 rows in
// either CTA of the pair), N = `n` (a multiple of 32 up to 256, half of it in either CTA).
__device__ __forceinline__ uint32_t umma_idesc_bf16_m256(uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((256u >> 4) << 24);
}
// D[tmem] (+)= A[tmem] * B[smem] over the CTA pair: in either CTA, A is 128 lanes x 16 bf16
// (eight 32-bit columns per lane), B half of the N rows, D 128 lanes x N columns.
__device__ __forceinline__ void tc_mma_bf16_a_tmem(uint32_t tmemD, uint32_t tmemA, uint64_t descB,
                                                   uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmemD),
        "r"(tmemA), "l"(descB), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void tc_store_32cols(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
        "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
        "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// ---- two CTAs of a cluster working as one tensor-core unit (cta_group::2) ----
__device__ __forceinline__ uint32_t cluster_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the shared::cluster address of `addr` (a shared-memory address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
    return out;
}
// Arrives on a barrier that may live in the other CTA of the pair (`clusterAddr` from map_to_cta), for a hand-over of
// tensor memory: relaxed, since the tcgen05 fences in front of it and behind the wait order the accesses.  (A
// cluster-scope release holds the warp until everything it has in flight is acknowledged, over a thousand cycles here.)
__device__ __forceinline__ void mbar_arrive_pair(uint32_t clusterAddr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(clusterAddr) : "memory");
}
// A copy into this CTA's shared memory whose completion is counted on a barrier of either CTA of the pair (`clusterBar`).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t clusterBar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(clusterBar)
        : "memory");
}
// A wait of a whole converged warp whose lanes then act as one: either all of them go on or none.
template <bool kSleep, Order kOrder>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t *abortFlag) {
    if (__all_sync(0xFFFFFFFFu, mbar_try_wait<kOrder>(bar, parity))) return true;
    return __all_sync(0xFFFFFFFFu, mbar_wait_slow<kSleep, kOrder>(bar, parity, abortFlag));
}
// one lane of the converged warp (the form in which the compiler knows that a single lane is active)
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xFFFFFFFF;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(one));
    return one != 0;
}
// the warp's index, known to be the same in all its lanes
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0); }
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrives once on the barrier at this shared-memory offset in both CTAs when the MMAs issued so far are done
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"((uint16_t)3)
        : "memory");
}

// ---- host: tensor map encoder ----

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled(const char **error) {
    // looked up once (thread-safe initialisation of a function-local static)
    static const EncodeTiledFn fn = [] {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t st = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q);
        if (st != cudaSuccess || q != cudaDriverEntryPointSuccess) sym = nullptr;
        return reinterpret_cast<EncodeTiledFn>(sym);
    }();
    if (!fn) fail(error, "cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

// A map of `rank` dimensions without element strides; parts of a box past the tensor read as zero.
inline bool encode_map(CUtensorMap *map, CUtensorMapDataType type, uint32_t rank, const void *base, const cuuint64_t *dims,
                       const cuuint64_t *strides, const cuuint32_t *box, CUtensorMapSwizzle swizzle, const char *what, const char **error) {
    const EncodeTiledFn fn = encode_tiled(error);
    if (!fn) return false;
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult rc = fn(map, type, rank, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return fail(error, std::string("cuTensorMapEncodeTiled(") + what + ") failed: " + std::to_string((int)rc));
    return true;
}

}  // namespace ff
