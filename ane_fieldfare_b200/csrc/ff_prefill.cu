// Prefill path of the INT4 MoE block: router for many rows, device-side permute (counting sort by
// expert), and the grouped INT4 -> bf16 GEMMs on the 5th-generation tensor cores.
//
// GEMM scheme.  Two CTAs of a cluster work as one tensor-core unit (cta_group::2, M = 256).  A unit of work
// is (row tile of up to 128 or 192 expert-sorted rows, two neighbouring tiles of 128 weight rows, one in either
// CTA: 64 gate + 64 up rows of the same features, or 128 down rows).  The dequantized weights are the MMA's A
// operand in tensor memory, the rows (tokens) its B operand in shared memory, half of the tile in either CTA.
// The contraction goes in steps of 64 (one quantization group), handed over two at a time.  Per CTA:
//   * warp 0 copies the token half tiles of a pair of steps (128-byte swizzle), completing on the leader's step
//     barrier; warp 26 copies packed codes, four steps of 128 weight rows at a time;
//   * sixteen warps in four groups, a group every fourth pair, turn codes into bf16 pairs (one fused multiply-add
//     with the group's scale and bias, a single rounding of q*scale+bias) and store them to tensor memory;
//   * warp 1 of the leader issues a pair's eight tcgen05.mma (K=16 each) into one of two accumulators of 128 or 192
//     columns, and one tcgen05.commit that frees the pair's stages in both CTAs;
//   * eight warps in two sets drain the finished accumulator (GeGLU to bf16 activations, or bf16 partial rows
//     scattered to (token, rank)) while the next unit's MMAs fill the other one.
// Within every aligned run of eight contraction elements the order is 0,4,1,5,2,6,3,7 in BOTH
// operands (a masked word yields codes j and j+4 side by side), which leaves every dot product
// unchanged; the activation buffers this file writes use that order.
//
// What bounds it: few rows an expert, the instructions of the dequantizing warps (a step is 160 instructions of each
// of its four warps, 72 of them the conversion itself) and the issuing warp's 430 cycles beside the MMAs of a
// hand-over; many, the tensor core, then the power limit.  With a hand-over every step, a group every fourth one: 77
// rows 252 us for two layers, 4096 rows 678 us; in pairs with a group's addresses running along 218 and 653; a group
// per pair, its slots fixed 203 and 634; tiles of 128 rows with eight weight stages 193 at 77 rows.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets the context's error flag and
// the whole CTA leaves its loops, frees its TMEM and returns.
//
// Reference kernels this file stands in for (paths inside the reference project):
//   Sources/ANEFieldfareHotpath/Metal/Prefill/prefill.metal:447-542 (router block),
//   :609-779 (routed experts as tiled matrix multiplies),
//   Sources/ANEFieldfareHotpath/Metal/TensorCore/tensorops.metal:14-298 (dense INT4 GEMM),
//   Sources/ANEFieldfareHotpath/Kernels/Prefill/MoE/PrefillMoEGrouping.swift:49-110 (the sort).
#include <algorithm>
#include <cstring>

#include "ff_gemv_device.cuh"
#include "ff_internal.cuh"
#include "ff_tc_device.cuh"

namespace ff {

// ---- router for many rows ------------------------------------------------------------------

// For every expert the logit is formed in the order the decode router uses (lane l chains fmaf
// over [256 i + 8 l, +8) for i ascending, butterfly 16..1, then the logit bias), so logits and
// indices are bitwise those of the single-row kernel.  Then the warp-wide top-K.
//
// A warp owns kTok tokens and walks the experts eight at a time with a register tile of
// kTok x 8 running sums.  The tokens' inputs sit in shared memory as bf16 for the whole kernel;
// the router rows stream through a small ring, one [8 experts x 256 inputs] block per copy (a
// tiled bulk tensor copy issued by a producer warp, completion on an mbarrier), in exactly the
// order the chains consume them: block i of a slice holds, for lane l, its eight elements of
// step i.  Per block a lane turns the 8 x 8 router values and its kTok x 8 inputs into fp32 once
// and issues 8 x kTok x 8 fmaf, element by element over all chains, so consecutive fmaf are
// independent.  A CTA takes 32 tokens (4096 tokens = 128 CTAs, one wave); shared memory holds
// their inputs whatever the split into warps, and the split that measured best is sixteen warps of
// two tokens (four warps per scheduler hide the shared-memory and conversion latencies): 164 us
// for 4096 tokens, against 182 us with eight warps of four, 214 us with four warps of eight, and
// 197 us for the previous kernel (whole eight-expert slices in shared memory, four tokens per
// warp, four warps per SM in two waves, packed FMAs fed by three integer-pipe cycles of conversions
// each).  In-kernel cycle counts: the chains 135 us of which 10 % waiting for blocks, top-K 15 us.
constexpr int kRouterTokensPerCta = 32;  // computing warps x tokens per warp (one more warp issues the copies)
constexpr int kRouterExperts = 8;   // experts per slice = rows of a streamed block
constexpr int kRouterBlockK = 256;  // inputs per streamed block: one step of every lane's chain
constexpr int kRouterRing = 8;      // blocks in flight
constexpr uint32_t kRouterBlockBytes = kRouterExperts * kRouterBlockK * 2;

static __device__ __noinline__ bool rt_wait_slow(uint32_t bar, uint32_t parity) {
    bool done = false;
    for (uint32_t spin = 0; spin < (1u << 22) && !done; ++spin) done = mbar_try_wait(bar, parity);
    return done;
}
// bounded; the first poll stands alone (inside the bounded loop it costs about 200 cycles even
// when the barrier is complete)
__device__ __forceinline__ bool rt_wait(uint32_t bar, uint32_t parity) {
    return mbar_try_wait(bar, parity) || rt_wait_slow(bar, parity);
}

// A multiple of 16, so that the next warp's rows are aligned: the logits of an even number of rows take an even number of
// experts' room.  (The sum rounded up instead: 17 rows of 2816 inputs and 128 experts 143.5 us, so 140.0.)
__host__ __device__ inline size_t router_warp_bytes(int tokens, int D, int E) {
    return (size_t)tokens * D * 2 + (size_t)tokens * (E + (E & 1)) * 4;
}

template <int kTok>
__global__ void __launch_bounds__((kRouterTokensPerCta / kTok + 1) * 32)
k_router_rows(const __grid_constant__ CUtensorMap mapW, const uint16_t *scale, const float *bias,
              const uint16_t *gain, const uint16_t *x, uint32_t xStride, int T, int E, int D, int K,
              uint32_t *ids, uint16_t *weights, float *logitsOut, uint32_t *errorFlag) {
    constexpr int kRouterWarps = kRouterTokensPerCta / kTok;
    static_assert(kTok % 2 == 0, "see router_warp_bytes");
    extern __shared__ __align__(128) uint8_t rsmRaw[];
    __shared__ __align__(8) uint64_t ringBar[2 * kRouterRing];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // ring of router blocks, then per computing warp: kTok input rows as bf16 and kTok x E logits
    const size_t perWarp = router_warp_bytes(kTok, D, E);
    const uint32_t ringAddr = (uint32_t)__cvta_generic_to_shared(rsmRaw);
    const uint32_t barBase = (uint32_t)__cvta_generic_to_shared(&ringBar[0]);
    auto barFull = [&](int s) { return barBase + 8u * (uint32_t)s; };
    auto barEmpty = [&](int s) { return barBase + 8u * (uint32_t)(kRouterRing + s); };
    const int nSlices = (E + kRouterExperts - 1) / kRouterExperts;
    const int nBlocks = (D + kRouterBlockK - 1) / kRouterBlockK;
    if (threadIdx.x == 0) {
        for (int st = 0; st < kRouterRing; ++st) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(barFull(st)) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(barEmpty(st)), "r"(kRouterWarps) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == kRouterWarps) {
        // ---- producer: every block of every slice, in consumption order ----
        if (lane == 0) {
            uint32_t st = 0, phase = 0;
            bool ok = true;
            for (int sl = 0; sl < nSlices && ok; ++sl)
                for (int i = 0; i < nBlocks; ++i) {
                    if (!rt_wait(barEmpty(st), phase ^ 1u)) {
                        atomicExch(errorFlag, 11u);
                        ok = false;
                        break;
                    }
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barFull(st)),
                                 "r"(kRouterBlockBytes)
                                 : "memory");
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                        " [%0], [%1, {%2, %3}], [%4];" ::"r"(ringAddr + st * kRouterBlockBytes),
                        "l"(reinterpret_cast<uint64_t>(&mapW)), "r"(i * kRouterBlockK), "r"(sl * kRouterExperts),
                        "r"(barFull(st))
                        : "memory");
                    if (++st == kRouterRing) {
                        st = 0;
                        phase ^= 1u;
                    }
                }
        }
        return;
    }

    uint8_t *warpBase = rsmRaw + (size_t)kRouterRing * kRouterBlockBytes + warp * perWarp;
    uint16_t *xs = reinterpret_cast<uint16_t *>(warpBase);
    float *lg = reinterpret_cast<float *>(warpBase + (size_t)kTok * D * 2);
    const int t0 = (blockIdx.x * kRouterWarps + warp) * kTok;
    const int nTok = max(0, min(kTok, T - t0));
    for (int tt = 0; tt < kTok; ++tt) {
        const uint16_t *xr = x + (size_t)min(t0 + min(tt, max(nTok, 1) - 1), T - 1) * xStride;
        for (int i = lane * 8; i < D; i += 256)
            *reinterpret_cast<uint4 *>(xs + (size_t)tt * D + i) = *reinterpret_cast<const uint4 *>(xr + i);
    }
    __syncwarp();

    uint32_t st = 0, phase = 0;
    bool ok = true;
    for (int sl = 0; sl < nSlices && ok; ++sl) {
        float acc[kTok][kRouterExperts];
#pragma unroll
        for (int t = 0; t < kTok; ++t)
#pragma unroll
            for (int e = 0; e < kRouterExperts; ++e) acc[t][e] = 0.0f;
        for (int i = 0; i < nBlocks; ++i) {
            if (!rt_wait(barFull(st), phase)) {
                if (lane == 0) atomicExch(errorFlag, 11u);
                ok = false;
                break;
            }
            const int base = i * kRouterBlockK + 8 * lane;
            if (base < D) {
                float xv[kTok][8];
                uint4 sv = make_uint4(0, 0, 0, 0);
                if (scale) sv = *reinterpret_cast<const uint4 *>(scale + base);
                const uint32_t ss[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
                for (int t = 0; t < kTok; ++t) {
                    const uint4 raw = *reinterpret_cast<const uint4 *>(xs + (size_t)t * D + base);
                    const uint32_t xr[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        float a0 = __uint_as_float(xr[k] << 16), a1 = __uint_as_float(xr[k] & 0xFFFF0000u);
                        if (scale) {
                            a0 = a0 * __uint_as_float(ss[k] << 16);
                            a1 = a1 * __uint_as_float(ss[k] & 0xFFFF0000u);
                        }
                        xv[t][2 * k] = a0;
                        xv[t][2 * k + 1] = a1;
                    }
                }
                const uint8_t *blockPtr = rsmRaw + (size_t)st * kRouterBlockBytes;
                float wv[kRouterExperts][8];
#pragma unroll
                for (int e = 0; e < kRouterExperts; ++e) {
                    const uint4 raw = *reinterpret_cast<const uint4 *>(blockPtr + (size_t)e * (kRouterBlockK * 2) + lane * 16);
                    const uint32_t ww[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        wv[e][2 * k] = __uint_as_float(ww[k] << 16);
                        wv[e][2 * k + 1] = __uint_as_float(ww[k] & 0xFFFF0000u);
                    }
                }
                // element by element, all (token, expert) chains side by side: consecutive fmaf are
                // independent, every chain still takes its eight elements in ascending order
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int e = 0; e < kRouterExperts; ++e)
#pragma unroll
                        for (int t = 0; t < kTok; ++t) acc[t][e] = fmaf(wv[e][k], xv[t][k], acc[t][e]);
            }
            // this warp is done with the block
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(barEmpty(st)) : "memory");
            if (++st == kRouterRing) {
                st = 0;
                phase ^= 1u;
            }
        }
        if (!ok) break;
#pragma unroll
        for (int t = 0; t < kTok; ++t)
#pragma unroll
            for (int e = 0; e < kRouterExperts; ++e) {
                float v = acc[t][e];
#pragma unroll
                for (int offset = 16; offset >= 1; offset >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, offset);
                const int ex = sl * kRouterExperts + e;
                if (lane == 0 && ex < E) lg[t * E + ex] = bias ? v + bias[ex] : v;
            }
    }
    __syncwarp();
    for (int tt = 0; tt < nTok; ++tt) {
        const int t = t0 + tt;
        if (logitsOut)
            for (int e = lane; e < E; e += 32) logitsOut[(size_t)t * E + e] = lg[tt * E + e];
        warp_topk(lg + tt * E, E, K, gain, ids + (size_t)t * K, weights + (size_t)t * K);
    }
}

static bool make_router_map(CUtensorMap *map, const void *base, uint64_t experts, uint64_t d, const char **error);

template <int kTok>
static bool launch_router_rows(FFContext *ctx, const LayerStore &L, const CUtensorMap &mapW, size_t smem,
                               const uint16_t *x, uint32_t xStride, uint32_t tokens, uint32_t *ids,
                               uint16_t *weights, float *logits, cudaStream_t stream, const char **error) {
    const int E = (int)L.routerExperts, D = (int)ctx->cfg.d;
    constexpr int kThreads = (kRouterTokensPerCta / kTok + 1) * 32;
    static KernelSmemMemo memo;
    if (!memo.prepare(k_router_rows<kTok>, ctx->device, smem, kThreads, nullptr, error)) return false;
    const uint32_t perCta = kRouterTokensPerCta;
    {
        LaunchScope scope(ctx, stream, "router_rows");
        k_router_rows<kTok><<<(tokens + perCta - 1) / perCta, kThreads, smem, stream>>>(
            mapW, L.routerScale, L.logitBias, L.gain, x, xStride, (int)tokens, E, D, (int)ctx->cfg.topK, ids,
            weights, logits, ctx->errorFlag);
    }
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

bool launch_router_prefill(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                           uint32_t tokens, uint32_t *ids, uint16_t *weights, float *logits,
                           cudaStream_t stream, const char **error) {
    const int E = (int)L.routerExperts, D = (int)ctx->cfg.d;
    if (D % 8) return fail(error, "hidden size must be a multiple of 8");
    // a tiled copy descriptor over the router matrix, [8 experts x 256 inputs] boxes (built per call:
    // encoding is host arithmetic only)
    CUtensorMap mapW;
    if (!make_router_map(&mapW, L.routerW, (uint64_t)E, (uint64_t)D, error)) return false;
    constexpr int kTok = 2;
    const size_t smem = (size_t)kRouterRing * kRouterBlockBytes + (size_t)(kRouterTokensPerCta / kTok) * router_warp_bytes(kTok, D, E);
    if (smem > 226 * 1024) return fail(error, "model width too large for the router's shared memory");
    return launch_router_rows<kTok>(ctx, L, mapW, smem, x, xStride, tokens, ids, weights, logits, stream, error);
}

// ---- device-side permute -------------------------------------------------------------------

constexpr int kSortTokens = 256;  // tokens per permute block

struct RowTile {
    uint32_t rowStart;  // first row in expert-sorted order
    uint32_t rows;      // 1..kRowTile
    uint32_t expert;
    uint32_t pad;
};

// Per-warp segment histogram of a block's routes: warp w owns routes [w*seg, (w+1)*seg) of the
// block; lanes holding the same expert are grouped with match.any and the group's lowest lane adds
// the group size.  segCount is [8 warps][E] in shared memory, zeroed by the caller.
__device__ __forceinline__ void segment_histogram(const uint32_t *routes, int n, int seg, int E,
                                                  uint32_t *segCount) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int begin = warp * seg, end = min(n, begin + seg);
    for (int i0 = begin; i0 < end; i0 += 32) {
        const int i = i0 + lane;
        const bool valid = i < end;
        const uint32_t e = valid ? routes[i] : 0xFFFFFFFFu;
        const uint32_t mask = __match_any_sync(0xFFFFFFFFu, e);
        if (valid && e < (uint32_t)E && (mask & ((1u << lane) - 1u)) == 0u)
            segCount[warp * E + e] += (uint32_t)__popc(mask);
        __syncwarp();
    }
}

constexpr uint32_t kNoRow = 0xFFFFFFFFu;  // of a route to no expert

// The experts' offsets and row tiles (up to `tileRows` rows of one expert each, experts ascending) from thread
// e's number of routes to expert e (0 from E on); a CTA of at least 256 threads, of which one in a cluster writes.
// Returns the expert's offset.
// counts[0] = row tiles, counts[1] = pairs, counts[2] = experts with at least one pair.
__device__ __forceinline__ uint32_t plan_row_tiles(uint32_t total, int E, uint32_t tileRows, uint32_t *expertOffsets, RowTile *tiles,
                                                   uint32_t maxTiles, uint32_t *counts, bool writes = true) {
    __shared__ uint32_t warpSums[3][8];
    const int e = threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t myTiles = (total + tileRows - 1u) / tileRows;
    uint32_t rows = total, tileEnd = myTiles;  // inclusive sums
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, rows, o), b = __shfl_up_sync(0xFFFFFFFFu, tileEnd, o);
        if (lane >= o) {
            rows += a;
            tileEnd += b;
        }
    }
    const uint32_t active = __popc(__ballot_sync(0xFFFFFFFFu, total != 0u));
    if (lane == 31 && warp < 8) {
        warpSums[0][warp] = rows;
        warpSums[1][warp] = tileEnd;
        warpSums[2][warp] = active;
    }
    __syncthreads();
    uint32_t activeAll = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) {
            rows += warpSums[0][w];
            tileEnd += warpSums[1][w];
        }
        activeAll += warpSums[2][w];
    }
    const uint32_t start = rows - total;
    if (!writes) return start;
    if (e < E) {
        expertOffsets[e] = start;
        for (uint32_t i = 0, tix = tileEnd - myTiles; i < total; i += tileRows, ++tix)
            if (tix < maxTiles) tiles[tix] = RowTile{start + i, min(tileRows, total - i), (uint32_t)e, 0u};
    }
    if (e == 255) {
        expertOffsets[E] = rows;
        counts[0] = min(tileEnd, maxTiles);
        counts[1] = rows;
        counts[2] = activeAll;
        counts[3] = 0;
    }
    return start;
}

// Pass 1: per block of 256 tokens, how many routes name each expert.
__global__ void __launch_bounds__(256)
k_route_count(const uint32_t *ids, int T, int K, int E, uint32_t *blockCounts) {
    pdl_enter();
    extern __shared__ uint32_t sRoutes[];
    __shared__ uint32_t segCount[8 * kMaxExperts];
    const int t0 = blockIdx.x * kSortTokens;
    const int n = min(kSortTokens, T - t0) * K;
    for (int i = threadIdx.x; i < n; i += blockDim.x) sRoutes[i] = ids[(size_t)t0 * K + i];
    for (int i = threadIdx.x; i < 8 * E; i += blockDim.x) segCount[i] = 0;
    __syncthreads();
    segment_histogram(sRoutes, n, (n + 7) / 8, E, segCount);
    __syncthreads();
    const int e = threadIdx.x;
    if (e < E) {
        uint32_t c = 0;
        for (int w = 0; w < 8; ++w) c += segCount[w * E + e];
        blockCounts[(size_t)blockIdx.x * E + e] = c;
    }
}

// Pass 2 (one block): exclusive prefix of every expert's counts over the blocks, then the plan.
__global__ void __launch_bounds__(256)
k_route_scan(uint32_t *blockCounts, int blocks, int E, uint32_t tileRows, uint32_t *expertOffsets, RowTile *tiles,
             uint32_t maxTiles, uint32_t *counts) {
    pdl_enter();
    uint32_t total = 0;
    const int e = threadIdx.x;
    if (e < E) {
        // eight blocks' counts are fetched together (independent loads), then turned into prefixes
        uint32_t run = 0;
        for (int b0 = 0; b0 < blocks; b0 += 8) {
            uint32_t c[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) c[i] = b0 + i < blocks ? blockCounts[(size_t)(b0 + i) * E + e] : 0u;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (b0 + i < blocks) {
                    blockCounts[(size_t)(b0 + i) * E + e] = run;
                    run += c[i];
                }
        }
        total = run;
    }
    plan_row_tiles(total, E, tileRows, expertOffsets, tiles, maxTiles, counts);
}

// Every route's position in (expert, token, rank) order; writes the sorted pair list.
// Position = expert offset + routes to the expert in earlier blocks + in earlier warp segments of
// this block + earlier in this warp's segment (earlier 32-route batches, then lower lanes).
// `base`: of expert threadIdx.x, the first two terms.
__device__ __forceinline__ void place_routes(const uint32_t *sRoutes, uint32_t *segCount, int n, int seg, uint32_t base,
                                             int t0, int K, int E, FFTokenExpertPair *sorted,
                                             uint32_t *rowOfRoute) {
    const int e = threadIdx.x;
    if (e < E) {
        // turn the segment counts into each segment's first position for this expert
        uint32_t run = base;
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = segCount[w * E + e];
            segCount[w * E + e] = run;
            run += c;
        }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int begin = warp * seg, end = min(n, begin + seg);
    for (int i0 = begin; i0 < end; i0 += 32) {
        const int i = i0 + lane;
        const bool valid = i < end;
        const uint32_t ex = valid ? sRoutes[i] : 0xFFFFFFFFu;
        const uint32_t mask = __match_any_sync(0xFFFFFFFFu, ex);
        const bool live = valid && ex < (uint32_t)E;
        uint32_t pos = 0;
        if (live) pos = segCount[warp * E + ex] + (uint32_t)__popc(mask & ((1u << lane) - 1u));
        __syncwarp();
        if (live && (mask & ((1u << lane) - 1u)) == 0u) segCount[warp * E + ex] += (uint32_t)__popc(mask);
        __syncwarp();
        if (live) {
            const uint32_t token = (uint32_t)(t0 + i / K), rank = (uint32_t)(i % K);
            sorted[pos] = FFTokenExpertPair{token, ex, rank, 0u};
        }
        if (rowOfRoute && valid) rowOfRoute[(size_t)t0 * K + i] = live ? pos : kNoRow;
    }
}

// Pass 3.
__global__ void __launch_bounds__(256)
k_route_scatter(const uint32_t *ids, int T, int K, int E,
                const uint32_t *blockCounts, const uint32_t *expertOffsets,
                FFTokenExpertPair *sorted, uint32_t *rowOfRoute) {
    pdl_enter();
    extern __shared__ uint32_t sRoutes[];
    __shared__ uint32_t segCount[8 * kMaxExperts];
    const int t0 = blockIdx.x * kSortTokens;
    const int n = min(kSortTokens, T - t0) * K;
    for (int i = threadIdx.x; i < n; i += blockDim.x) sRoutes[i] = ids[(size_t)t0 * K + i];
    for (int i = threadIdx.x; i < 8 * E; i += blockDim.x) segCount[i] = 0;
    __syncthreads();
    const int seg = (n + 7) / 8;
    segment_histogram(sRoutes, n, seg, E, segCount);
    __syncthreads();
    const int e = threadIdx.x;
    place_routes(sRoutes, segCount, n, seg, e < E ? expertOffsets[e] + blockCounts[(size_t)blockIdx.x * E + e] : 0u, t0, K, E,
                 sorted, rowOfRoute);
}

// All three passes in one launch of a cluster of eight CTAs for up to kClusterRoutes routes: every CTA counts its
// share, a warp its part of that with the routes and their matches in registers, the CTAs read one another's counts
// from shared memory, plan alike, and place.  Bound by its latencies, then by eight SMs' matches and scattered stores.
// us in a graph, Zipf routes, 128 experts, one launch / three: 77 rows 3.7 / -, 257 4.3 / 15.1, 613 5.1 / 15.3, 1500
// 7.9 / 15.5, 4096 15.4 / 16.9, 6000 21.2 / 17.4 (for fewer routes a row see sort_in_one_launch).  (CTAs of 1024 threads, or
// sixteen of them, are faster by themselves, 10.9 us at 4096 rows, but wait longer for SMs beside the shared FFN: a layer of
// 300 rows 308 us for 298.)
constexpr int kSortCtas = 8, kSortThreads = 512, kSortRounds = 8;  // rounds of 32 routes of a warp
constexpr int kClusterRoutes = kSortCtas * kSortThreads * kSortRounds;
__global__ void __cluster_dims__(kSortCtas, 1, 1) __launch_bounds__(kSortThreads, 1)
k_route_sort(const uint32_t *ids, int T, int K, int E, uint32_t tileRows, uint32_t *expertOffsets, RowTile *tiles, uint32_t maxTiles,
             uint32_t *counts, FFTokenExpertPair *sorted, uint32_t *rowOfRoute) {
    pdl_enter();
    __shared__ uint32_t segCount[(kSortThreads / 32) * kMaxExperts];  // a warp's routes to every expert, then its next place
    __shared__ uint32_t ctaCount[kMaxExperts], sBase[kMaxExperts];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = threadIdx.x;
    const uint32_t cta = cluster_cta_rank();
    const int perCta = (T + kSortCtas - 1) / kSortCtas * K, first = min((int)cta * perCta, T * K), n = min(perCta, T * K - first);
    const int seg = (n + kSortThreads / 32 - 1) / (kSortThreads / 32), begin = warp * seg, end = min(n, begin + seg);
    uint32_t *mine = segCount + warp * E;
    uint32_t id[kSortRounds], peers[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const int i = begin + 32 * r + lane;
        id[r] = i < end ? ids[first + i] : 0xFFFFFFFFu;
    }
    for (int x = lane; x < E; x += 32) mine[x] = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        if (begin + 32 * r >= end) break;
        peers[r] = __match_any_sync(0xFFFFFFFFu, id[r]);
        if (id[r] < (uint32_t)E && (peers[r] & ((1u << lane) - 1u)) == 0u) mine[id[r]] += (uint32_t)__popc(peers[r]);
        __syncwarp();
    }
    __syncthreads();
    if (e < E) {
        uint32_t run = 0;
#pragma unroll 8
        for (int w = 0; w < kSortThreads / 32; ++w) {
            const uint32_t c = segCount[w * E + e];
            segCount[w * E + e] = run;
            run += c;
        }
        ctaCount[e] = run;
    }
    cluster_sync_all();
    uint32_t total = 0, earlier = 0;
    if (e < E) {
        uint32_t c[kSortCtas];
        const uint32_t addr = smem_u32(ctaCount + e);
#pragma unroll
        for (uint32_t i = 0; i < kSortCtas; ++i) asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(c[i]) : "r"(map_to_cta(addr, i)));
#pragma unroll
        for (uint32_t i = 0; i < kSortCtas; ++i) {
            total += c[i];
            if (i < cta) earlier += c[i];
        }
    }
    const uint32_t start = plan_row_tiles(total, E, tileRows, expertOffsets, tiles, maxTiles, counts, cta == 0u);
    if (e < E) sBase[e] = start + earlier;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        if (begin + 32 * r >= end) break;
        const int i = first + begin + 32 * r + lane;
        const bool valid = begin + 32 * r + lane < end, live = valid && id[r] < (uint32_t)E;
        const uint32_t lower = peers[r] & ((1u << lane) - 1u);
        uint32_t pos = 0;
        if (live) pos = sBase[id[r]] + mine[id[r]] + (uint32_t)__popc(lower);
        __syncwarp();
        if (live && lower == 0u) mine[id[r]] += (uint32_t)__popc(peers[r]);
        __syncwarp();
        if (live) sorted[pos] = FFTokenExpertPair{(uint32_t)(i / K), id[r], (uint32_t)(i % K), 0u};
        if (rowOfRoute && valid) rowOfRoute[i] = live ? pos : kNoRow;
    }
    cluster_sync_all();  // no CTA leaves while another may read its counts
}

// Row tiles of a dense problem: T rows of one "expert" (the shared FFN).
__global__ void k_dense_tiles(int T, int tileRows, RowTile *tiles, uint32_t *counts) {
    pdl_enter();
    const int n = (T + tileRows - 1) / tileRows;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        tiles[i] = RowTile{(uint32_t)(i * tileRows), (uint32_t)min(tileRows, T - i * tileRows), 0u, 0u};
    if (threadIdx.x == 0) {
        counts[0] = (uint32_t)n;
        counts[1] = (uint32_t)T;
        counts[2] = 1;
        counts[3] = 0;
    }
}

// Copies rows of x into the GEMM's activation buffer, reordering every aligned run of eight
// elements to 0,4,1,5,2,6,3,7: row t to row t (K = 0), or to the rows of its K routes.  One thread per
// 16 bytes read; bound by the writes.  (Going through the sorted rows instead reads every token K times, from
// memory where the rows exceed the L2: the block of 32768 tokens and eight routes took 160 us more.)
__global__ void __launch_bounds__(256)
k_gather_rows(const uint16_t *x, uint32_t xStride, uint32_t rows, const uint32_t *rowOfRoute, int K, int D, uint16_t *out) {
    pdl_enter();
    const int chunksPerRow = D / 8;
    const size_t total = (size_t)rows * chunksPerRow;
    const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t step = gridDim.x * blockDim.x, stepRows = step / chunksPerRow;
    const int stepChunks = (int)(step - stepRows * chunksPerRow);
    uint32_t r = (uint32_t)(first / chunksPerRow);
    int c = (int)(first - (size_t)r * chunksPerRow);
    for (size_t i = first; i < total; i += step, r += stepRows, c += stepChunks) {
        if (c >= chunksPerRow) {
            c -= chunksPerRow;
            ++r;
        }
        const uint4 v = *reinterpret_cast<const uint4 *>(x + (size_t)r * xStride + c * 8);
        // halves h0..h7 -> h0,h4,h1,h5,h2,h6,h3,h7
        uint4 o;
        o.x = __byte_perm(v.x, v.z, 0x5410);
        o.y = __byte_perm(v.x, v.z, 0x7632);
        o.z = __byte_perm(v.y, v.w, 0x5410);
        o.w = __byte_perm(v.y, v.w, 0x7632);
        if (K == 0) {
            *reinterpret_cast<uint4 *>(out + (size_t)r * D + c * 8) = o;
        } else {
            const uint32_t *routes = rowOfRoute + (size_t)r * K;
#pragma unroll 8
            for (int k = 0; k < K; ++k) {
                const uint32_t row = __ldg(routes + k);
                if (row != kNoRow) *reinterpret_cast<uint4 *>(out + (size_t)row * D + c * 8) = o;
            }
        }
    }
}

// ---- grouped INT4 GEMM ---------------------------------------------------------------------

constexpr int kWeightRows = 128;  // weight rows of a unit = TMEM lanes of its accumulator
constexpr int kTileK = 64;        // one quantization group per step
constexpr int kTokStages = 4;     // token half tiles of two steps (TMA destinations)
constexpr int kQuad = 4;          // steps whose packed codes come as one copy (128 bytes of a weight row)
constexpr int kMaxPackStages = 6; // quads of packed codes in flight: as many as shared memory holds
constexpr int kGroups = 4;        // dequantizing groups: one for each slot of the step ring
constexpr int kDequantWarps = 16; // four groups of four warps; a group covers the 128 TMEM lanes
constexpr int kEpilogueSets = 2;  // of four warps each, taking turns at 32-token chunks
// warp 0 token copies, warp 1 MMA, warps 2-17 dequantize, warps 18-25 epilogue (TMEM lane quarter =
// warp & 3), warp 26 code copies
constexpr int kFirstEpilogueWarp = 2 + kDequantWarps;
constexpr int kCodeWarp = kFirstEpilogueWarp + 4 * kEpilogueSets;
constexpr int kGemmThreads = (kCodeWarp + 1) * 32;
constexpr int kEpilogueThreads = 128 * kEpilogueSets;
constexpr uint32_t kTokSmallRows = 32;                            // of those, copied for a small tile
constexpr uint32_t kPackTileBytes = kWeightRows * kTileK / 2 * kQuad;  // 16384: two [64 rows x 128 bytes] boxes
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kStagePitchGateUp = 64 * 2 + 16;               // bytes per token row of the output tile
constexpr uint32_t kStagePitchDown = 128 * 2 + 16;
constexpr uint32_t kStageBytesGateUp = 32u * kStagePitchGateUp;   // one 32-token output tile
constexpr uint32_t kStageBytesDown = 32u * kStagePitchDown;
// per set two output tiles; down: two row tables, too
constexpr uint32_t kEpilogueBytesGateUp = kEpilogueSets * 2u * kStageBytesGateUp;
constexpr uint32_t kEpilogueBytesDown = kEpilogueSets * 2u * kStageBytesDown + 2u * kRowTile * 4u;
constexpr uint32_t kScaleSlotBytes = kDequantWarps * 32 * 8;      // two scale words of every dequantizing thread
__host__ __device__ constexpr uint32_t scale_buffer_bytes(uint32_t quads) { return (quads + 1u) / 2u * kScaleSlotBytes; }
// Dequantized weight tiles in tensor memory, 32 columns each behind two accumulators of `tileRows` columns.
__host__ __device__ constexpr uint32_t weight_stages(uint32_t tileRows) { return tileRows <= kRowTileSmall ? 8u : 4u; }
// A CTA's half of a step's token tile (a multiple of the 1024-byte swizzle atom).
__host__ __device__ constexpr uint32_t tok_tile_bytes(uint32_t tileRows) { return tileRows / 2u * kTileK * 2u; }
static_assert(2 * kRowTile + weight_stages(kRowTile) * 32 <= kTmemCols && 2 * kRowTileSmall + weight_stages(kRowTileSmall) * 32 <= kTmemCols, "tensor memory layout");
static_assert(kRowTile % 32 == 0 && (int)kRowTile <= kEpilogueThreads && kRowTileSmall % 32 == 0, "row tile");
static_assert((int)weight_stages(kRowTileSmall) <= 2 * kTokStages && 2 * kTokStages % weight_stages(kRowTile) == 0, "rings");
static_assert(kTokStages == kGroups && kQuad == 4, "a group owns a slot; two pairs a quad");

enum GemmMode : int { kModeGateUp = 0, kModeDown = 1 };

struct GemmArgs {
    const uint32_t *scaleWords;  // scale | bias words of expert 0 (see pack_scales), of its down rows for the down GEMM
    uint64_t scaleStride;        // words between experts
    uint32_t tileRows, packStages;
    uint32_t scaleBuffers;     // see GemmRings
    uint32_t K;                // contraction length (multiple of 64)
    uint32_t N;                // outputs per row: F (gate/up) or D (down)
    uint32_t nTiles;           // weight-row tiles: ceil(N/64) for gate/up, ceil(N/128) for down
    const RowTile *tiles;
    const uint32_t *counts;    // counts[0] = row tiles
    uint16_t *out;             // gate/up: activations [row][N]; down: output rows [*][N]
    const FFTokenExpertPair *pairs;  // down: row -> (token, rank); null: row -> row
    uint32_t topK;
    uint32_t roundGateUp;      // gate/up: round both to bf16 before the activation
    uint32_t *errorFlag;
};

// element at position p of a run of eight in the order 0,4,1,5,2,6,3,7
__device__ __forceinline__ uint32_t interleaved_element(uint32_t p) { return (p >> 1) | ((p & 1u) << 2); }
// eight columns each of four 8 x 8 bf16 blocks, transposed: lane l gives the address of row l & 7 of block l >> 3
__device__ __forceinline__ void store_blocks_transposed(uint32_t addr, const uint32_t (&p)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(p[0]), "r"(p[1]), "r"(p[2]),
                 "r"(p[3])
                 : "memory");
}
// two floats as bf16, the first in the low half
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// bf16 fma(q, scale, bias) of the 64 codes of eight words, as pairs (code i, code i + 4).  A nibble masked in
// place, at bits 0-3 or 4-7 of a half word, IS a bf16: the subnormal q * 2^-133 or (exponent field 0 or 1) the
// number q * 2^-129.  The FMA takes it as it stands, with the scale times 2^133 or 2^129: the same product, the
// same single rounding, 9 instructions for a word where taking the nibble to q itself needs 15.  Scales whose
// product with 2^133 is no normal bf16 (from 2^-5 on, and subnormal ones) take the longer way, a warp at a time.
__device__ __forceinline__ void dequantize_words(const uint32_t (&w)[8], uint32_t scaleBias, uint32_t (&o)[32]) {
    uint32_t s2, b2;
    asm("prmt.b32 %0, %1, %1, 0x1010;" : "=r"(s2) : "r"(scaleBias));
    asm("prmt.b32 %0, %1, %1, 0x3232;" : "=r"(b2) : "r"(scaleBias));
    const uint32_t magnitude = s2 & 0x7FFFu;
    constexpr uint32_t kMinNormal = 0x0080u, kLimit = 0x3D00u;  // 2^-126, 2^-5
    if (__all_sync(0xFFFFFFFFu, magnitude == 0u || magnitude - kMinNormal < kLimit - kMinNormal)) {
        const uint32_t sLow = magnitude ? s2 + 0x42804280u : 0u;   // exponent + 133
        const uint32_t sHigh = magnitude ? s2 + 0x40804080u : 0u;  // exponent + 129
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t upper = w[j] >> 8;
            asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[4 * j]) : "r"(w[j] & 0x000F000Fu), "r"(sLow), "r"(b2));
            asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[4 * j + 1]) : "r"(w[j] & 0x00F000F0u), "r"(sHigh), "r"(b2));
            asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[4 * j + 2]) : "r"(upper & 0x000F000Fu), "r"(sLow), "r"(b2));
            asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[4 * j + 3]) : "r"(upper & 0x00F000F0u), "r"(sHigh), "r"(b2));
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // codes i and i+4 of the word as the bf16 pair (128+q_i, 128+q_{i+4})
                const uint32_t pair = ((w[j] >> (4 * i)) & 0x000F000Fu) | 0x43004300u;
                uint32_t q2;
                asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(q2) : "r"(pair), "r"(0x43004300u));
                asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[4 * j + i]) : "r"(q2), "r"(s2), "r"(b2));
            }
        }
    }
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
k_grouped_int4_gemm(const __grid_constant__ CUtensorMap mapTok, const __grid_constant__ CUtensorMap mapTokSmall, const __grid_constant__ CUtensorMap mapW0,
                    const __grid_constant__ CUtensorMap mapW1, const GemmArgs args) {
    extern __shared__ uint8_t gemmSmemRaw[];
    __shared__ __align__(64) uint64_t barriers[2 * kTokStages + 2 * kMaxPackStages + 4 + 2 * kEpilogueSets + 1];
    __shared__ uint32_t tmemBaseSlot;
    __shared__ volatile uint32_t abortFlag;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rawBase = smem_u32(gemmSmemRaw);
    const uint32_t base = (rawBase + 1023u) & ~1023u;
    const uint32_t groupsK = args.K / kTileK, quadsK = (groupsK + kQuad - 1) / kQuad;

    // carve-up: token stages (1024-aligned), packed stages, the epilogue's buffers, scale words
    // (stage addresses are computed, not tabulated: an array indexed by the running stage would
    // live in local memory)
    const uint32_t tokBytes = tok_tile_bytes(args.tileRows), packBase = base + kTokStages * 2u * tokBytes;
    auto tokAddrOf = [&](uint32_t s) { return base + s * 2u * tokBytes; };
    auto packAddrOf = [&](uint32_t s) { return packBase + s * kPackTileBytes; };
    const uint32_t epilogueOffset = packBase + args.packStages * kPackTileBytes - rawBase;
    uint8_t *epilogueSmem = gemmSmemRaw + epilogueOffset;
    const uint32_t scaleBase = rawBase + epilogueOffset + (MODE == kModeGateUp ? kEpilogueBytesGateUp : kEpilogueBytesDown);

    const uint32_t barBase = smem_u32(barriers);
    auto barAt = [&](int i) { return barBase + 8u * (uint32_t)i; };
    auto barStep = [&](int s) { return barAt(s); };
    auto barTokEmpty = [&](int s) { return barAt(kTokStages + s); };
    auto barPackFull = [&](int s) { return barAt(2 * kTokStages + s); };
    auto barPackEmpty = [&](int s) { return barAt(2 * kTokStages + kMaxPackStages + s); };
    constexpr int kBarAcc = 2 * kTokStages + 2 * kMaxPackStages;
    auto barAccFull = [&](int s) { return barAt(kBarAcc + s); };
    auto barAccEmpty = [&](int s) { return barAt(kBarAcc + 2 + s); };
    auto barStage = [&](int set, int buffer) { return barAt(kBarAcc + 4 + 2 * set + buffer); };
    const uint32_t barRows = barAt(kBarAcc + 4 + 2 * kEpilogueSets);

    // The two CTAs of a cluster work as one unit of the tensor core: the leader (rank 0) issues
    // the MMAs for both.  What the MMA issuer waits for lives in the leader: a step's barrier counts the
    // arrivals of both CTAs' dequantizers and the bytes of both CTAs' token copies.  Barriers that the MMAs'
    // completion frees exist in either CTA and are signalled in both by one multicast commit.
    const uint32_t ctaRank = cluster_cta_rank();
    const bool leader = ctaRank == 0u;
    if (threadIdx.x == 0) {
        abortFlag = 0;
        for (int s = 0; s < kTokStages; ++s) {
            mbar_init(barStep(s), 9);      // (leader's is used) a group's four warps in either CTA, the expected bytes
            mbar_init(barTokEmpty(s), 1);  // one tcgen05.commit
        }
        for (int s = 0; s < kMaxPackStages; ++s) {
            mbar_init(barPackFull(s), 1);
            mbar_init(barPackEmpty(s), kDequantWarps / 2);  // the warps of two groups
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(barAccFull(s), 1);                     // one tcgen05.commit
            mbar_init(barAccEmpty(s), 8 * kEpilogueSets);    // (leader's is used) the epilogue warps of either CTA
        }
        for (int s = 0; s < kEpilogueSets; ++s) {
            mbar_init(barStage(s, 0), 128);  // every thread of the set
            mbar_init(barStage(s, 1), 128);
        }
        mbar_init(barRows, kEpilogueThreads);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmemBaseSlot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // the other CTA's barriers are initialised before anything arrives on them
    tc_fence_after();
    const uint32_t tmemBase = __shfl_sync(0xFFFFFFFFu, tmemBaseSlot, 0);
    pdl_enter();

    // A pair's unit: one row tile, two neighbouring weight-row tiles (this CTA takes 2 np + rank).
    // Every role reads a unit's tile one unit ahead, so that the load's latency is not in its loop.
    const uint32_t rowTiles = args.counts[0];
    const uint32_t nPairs = (args.nTiles + 1u) >> 1;
    const uint32_t units = rowTiles * nPairs;
    const uint32_t firstUnit = blockIdx.x >> 1, unitStride = gridDim.x >> 1;
    auto tileOf = [&](uint32_t u) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(args.tiles + (u < units ? u : firstUnit) / nPairs));
        return RowTile{v.x, v.y, v.z, v.w};
    };
    auto ntOf = [&](uint32_t u) { return 2u * (u % nPairs) + ctaRank; };
    // accumulator columns of a tile: its rows to the next multiple of 32, half of them in either CTA
    auto columnsOf = [&](const RowTile &tile) { return max(32u, (tile.rows + 31u) & ~31u); };
    // Tensor memory behind the two accumulators: a step's weight stage is its token stage, modulo the stages there are.
    const uint32_t wCol0 = 2u * args.tileRows, wStages = weight_stages(args.tileRows), wMask = wStages - 1u;
    // weight rows of a unit: gate rows [64 nt, +64) | up rows [64 nt, +64) for the gate/up
    // GEMM, matrix rows [128 nt, +128) for the down GEMM; loaded as two boxes of 64 rows.  In tensor
    // memory gate and up stand in turn, eight lanes each, so that the epilogue's threads find both
    // values of a feature in their own registers, and a run of eight features stands in the
    // interleaved order that the down GEMM reads.

    if (warp == 0) {
        // ---------------- token copies ----------------
        // A pair of steps is two copies, of 32 rows where the tile's half needs no more and of the whole half (64 or
        // 96) otherwise.  (16 rows at a time, as many as needed, were slower than 96 always: 353 us against 339 with 77
        // tokens.  It is the copies, not their bytes, that cost.)
        if (firstUnit < units) {
            uint32_t ts = 0, phase = 0;
            bool ok = true;
            RowTile next = tileOf(firstUnit);
            const uint32_t leaderStep = map_to_cta(barStep(0), 0u);
            for (uint32_t u = firstUnit; u < units && ok; u += unitStride) {
                const RowTile tile = next;
                next = tileOf(u + unitStride);
                const uint32_t half = columnsOf(tile) >> 1;  // this CTA's half of the tile's rows
                const int row0 = (int)(tile.rowStart + ctaRank * half);
                const CUtensorMap *map = half <= kTokSmallRows ? &mapTokSmall : &mapTok;
                const uint32_t bytes = half <= kTokSmallRows ? tok_tile_bytes(2u * kTokSmallRows) : tokBytes;
                for (uint32_t g = 0; g < kQuad * quadsK; g += 2) {
                    if (!mbar_wait_warp<true, Order::kPair>(barTokEmpty(ts), phase ^ 1u, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    if (elect_one()) {
                        const uint32_t steps = g + 1u < groupsK ? 2u : g < groupsK ? 1u : 0u;  // fewer at a row's end
                        if (leader) mbar_expect_tx(barStep(ts), 2u * steps * bytes);
                        if (steps > 0u) tma_load_2d_pair(tokAddrOf(ts), map, (int)(g * kTileK), row0, leaderStep + 8u * ts);
                        if (steps > 1u) tma_load_2d_pair(tokAddrOf(ts) + tokBytes, map, (int)((g + 1u) * kTileK), row0, leaderStep + 8u * ts);
                    }
                    ts = (ts + 1u) % kTokStages;
                    if (ts == 0) phase ^= 1u;
                }
            }
        }
    } else if (warp == kCodeWarp) {
        // ---------------- code copies: a quad of steps at a time ----------------
        if (lane == 0 && firstUnit < units) {
            uint32_t ps = 0, phase = 0;
            bool ok = true;
            RowTile next = tileOf(firstUnit);
            for (uint32_t u = firstUnit; u < units && ok; u += unitStride) {
                const RowTile tile = next;
                next = tileOf(u + unitStride);
                const uint32_t nt = ntOf(u);
                for (uint32_t q = 0; q < quadsK; ++q) {
                    if (!mbar_wait_idle(barPackEmpty(ps), phase ^ 1u, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(barPackFull(ps), kPackTileBytes);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const CUtensorMap *map = (MODE == kModeGateUp && h == 1) ? &mapW1 : &mapW0;
                        const int wRow = MODE == kModeGateUp ? (int)nt * 64 : (int)nt * 128 + h * 64;
                        tma_load_3d(packAddrOf(ps) + (uint32_t)h * (kPackTileBytes / 2), map,
                                    (int)(q * (kQuad * kTileK / 2)), wRow, (int)tile.expert, barPackFull(ps));
                    }
                    if (++ps == args.packStages) {
                        ps = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA only) ----------------
        // The whole warp runs the loop and one elected lane issues: with the loop inside a `lane == 0`
        // branch every operand goes to the uniform registers by a loop over the active lanes, and a step
        // cost this thread 820 cycles for 384 of the tensor core.
        if (leader && firstUnit < units) {
            uint32_t ts = 0, phase = 0, acc = 0, accPhase = 0;
            bool ok = true, ready = false;  // ready: seen that the next pair's weights and tokens are there
            RowTile next = tileOf(firstUnit);
            for (uint32_t u = firstUnit; u < units && ok; u += unitStride) {
                const RowTile tile = next;
                next = tileOf(u + unitStride);
                const uint32_t idesc = umma_idesc_bf16_m256(columnsOf(tile));
                if (!mbar_wait_warp<true, Order::kPair>(barAccEmpty(acc), accPhase ^ 1u, &abortFlag)) break;
                tc_fence_after();
                const uint32_t tmemD = tmemBase + acc * args.tileRows;
                for (uint32_t g = 0; g < kQuad * quadsK; g += 2) {
                    if (!__all_sync(0xFFFFFFFFu, ready) &&
                        !mbar_wait_warp<false, Order::kPair>(barStep(ts), phase, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // the next pair's barrier is looked at now and the answer used after this pair's MMAs
                    const uint32_t tn = (ts + 1u) % kTokStages;
                    if (tn == 0u) phase ^= 1u;
                    ready = mbar_test_wait<Order::kPair>(barStep(tn), phase);
                    const uint64_t descTok = umma_desc_sw128(tokAddrOf(ts));
                    const uint32_t tmemW = tmemBase + wCol0 + (2u * ts & wMask) * 32u;
                    if (elect_one()) {
                        // (the wait was for both CTAs' operands; this look acquires the token halves, whose copies
                        // complete on this CTA's barrier)
                        (void)mbar_test_wait(barStep(ts), tn == 0u ? phase ^ 1u : phase);
                        // per 16-element slice: eight columns further in TMEM, 32 bytes (>> 4 = 2) further in
                        // the token tile
                        if (g < groupsK) {
#pragma unroll
                            for (uint32_t kk = 0; kk < kTileK / 16; ++kk)
                                tc_mma_bf16_a_tmem(tmemD, tmemW + 8u * kk, descTok + 2u * kk, idesc, (g | kk) != 0u ? 1u : 0u);
                        }
                        if (g + 1u < groupsK) {
#pragma unroll
                            for (uint32_t kk = 0; kk < kTileK / 16; ++kk)
                                tc_mma_bf16_a_tmem(tmemD, tmemW + 32u + 8u * kk, descTok + (tokBytes >> 4) + 2u * kk, idesc, 1u);
                        }
                        // one signal per pair of steps: the token stage is free, and so are the weight stages that
                        // they used (the dequantizers wait on the token ring's barrier, too)
                        tc_commit_pair(barTokEmpty(ts));
                    }
                    ts = tn;
                }
                if (!ok) break;
                if (elect_one()) tc_commit_pair(barAccFull(acc));
                acc ^= 1u;
                accPhase ^= acc == 0u ? 1u : 0u;
            }
        }
    } else if (warp < kFirstEpilogueWarp) {
        // ---------------- dequantizers ----------------
        // Group `grp` (four warps, one per TMEM lane quarter) takes every fourth pair of steps, counted over all of
        // the CTA's units: pair `grp & 1` of every second quad, and slot `grp` of the step ring.  A thread turns one
        // weight row's 64 codes of a step into 32 bf16 pairs and stores them to its TMEM lane.  Four pairs are in work
        // at once, which hides a pair's latencies behind the other groups' arithmetic.
        const uint32_t grp = (uint32_t)(warp - 2) >> 2, half = grp & 1u, quadParity = grp >> 1;
        const uint32_t m = (uint32_t)(warp & 3) * 32u + (uint32_t)lane;  // TMEM lane
        // its feature within the unit (gate/up), its row in the loaded boxes
        const uint32_t feature = (m >> 4) * 8u + interleaved_element(m & 7u);
        const uint32_t boxRow = MODE == kModeGateUp ? ((m >> 3) & 1u) * 64u + feature : m;
        const uint32_t paddedK = (groupsK + 3u) & ~3u;

        // The thread's scale words of a unit (two per pair) come as asynchronous copies into a private column of
        // shared memory, one unit ahead: no global load is in flight in the steady loop (one in flight would hold up
        // the releasing arrive below for its whole latency), and none is waited for at a unit's start.
        const uint32_t myScales = scaleBase + 8u * (uint32_t)(threadIdx.x - 64);  // [buffer][every second quad][512 threads]
        auto scale_row = [&](uint32_t u, const RowTile &tile, bool &live) {
            const uint32_t nt = ntOf(u);
            const uint32_t wRow = MODE == kModeGateUp ? nt * 64u + feature : nt * 128u + m;
            live = wRow < args.N;
            const uint32_t row = MODE == kModeGateUp ? (wRow >> 3) * 16u + (wRow & 7u) + (m & 8u) : wRow;
            return args.scaleWords + (size_t)tile.expert * args.scaleStride + (size_t)(live ? row : 0u) * paddedK + 2u * half;
        };
        // quads first, first + 2, ...
        auto fetch_scales = [&](uint32_t u, const RowTile &tile, uint32_t first, uint32_t buffer) {
            bool live;
            const uint32_t *src = scale_row(u, tile, live) + first * kQuad;
            uint32_t dst = myScales + buffer * scale_buffer_bytes(quadsK);
            for (uint32_t q = first; q < quadsK; q += 2, dst += kScaleSlotBytes, src += 2 * kQuad)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(live ? 8u : 0u) : "memory");
        };
        auto scales_arrived = [] { asm volatile("cp.async.wait_all;" ::: "memory"); };
        // What the loop needs stands in registers; the slots of the group are always the same.
        const uint32_t rowOffset = boxRow * 128u, flip = boxRow & 7u;
        uint32_t codes[4];  // its 64 bytes of a quad's row: 16-byte chunks with the 128-byte swizzle
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) codes[c] = packBase + rowOffset + (((4u * half + c) ^ flip) << 4);
        const uint32_t stepBar = map_to_cta(barStep((int)grp), 0u);
        const uint32_t tmemW = tmemBase + wCol0 + (2u * grp & wMask) * 32u + (((uint32_t)(warp & 3) * 32u) << 16);
        // The weight stages were last read by the MMAs `wStages` steps back: their completion is that pair's signal
        // on the token ring.  (A first pair waits for the parity of a phase before the barrier's first: not at all.)
        const uint32_t freeBar = barTokEmpty((int)(wStages == 8u ? grp : grp ^ 2u));
        uint32_t freePhase = wStages == 8u || grp < 2u ? 1u : 0u;
        uint32_t ps = quadParity, pPhase = 0;
        uint32_t quad0 = 0;  // quads of the CTA's earlier units
        bool ok = firstUnit < units;
        RowTile tile{}, next{};
        if (ok) {
            next = tileOf(firstUnit);
            if (args.scaleBuffers) fetch_scales(firstUnit, next, quadParity, 0);
        }
        uint32_t unitNo = 0;
        for (uint32_t u = firstUnit; u < units && ok; u += unitStride, ++unitNo, quad0 += quadsK) {
            tile = next;
            next = tileOf(u + unitStride);
            const uint32_t first = (quad0 ^ quadParity) & 1u;
            const uint32_t buffer = args.scaleBuffers == 2 ? unitNo & 1u : 0u;
            if (args.scaleBuffers == 2) {
                scales_arrived();
                if (u + unitStride < units) fetch_scales(u + unitStride, next, (quad0 + quadsK ^ quadParity) & 1u, buffer ^ 1u);
            } else if (args.scaleBuffers == 1) {
                if (unitNo) fetch_scales(u, tile, first, 0);
                scales_arrived();
            }
            uint32_t scaleAddr = myScales + buffer * scale_buffer_bytes(quadsK);
            // (A row's last quad may have fewer than four steps: the rest is converted like any other, from codes
            // that read as zero, and no MMA uses it.)
            for (uint32_t q = first; q < quadsK; q += 2, scaleAddr += kScaleSlotBytes) {
                if (!mbar_wait_warp<false, Order::kLocal>(barPackFull((int)ps), pPhase, &abortFlag)) {
                    ok = false;
                    break;
                }
                uint32_t sb[2];
                if (args.scaleBuffers) {
                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(sb[0]), "=r"(sb[1]) : "r"(scaleAddr));
                } else {
                    bool live;
                    const uint32_t *src = scale_row(u, tile, live) + q * kQuad;
                    sb[0] = live ? __ldg(src) : 0u;
                    sb[1] = live ? __ldg(src + 1) : 0u;
                }
                uint32_t w[2][8], o[32];
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(w[c >> 1][4 * (c & 1)]), "=r"(w[c >> 1][4 * (c & 1) + 1]), "=r"(w[c >> 1][4 * (c & 1) + 2]),
                                   "=r"(w[c >> 1][4 * (c & 1) + 3])
                                 : "r"(codes[c] + ps * kPackTileBytes));
                dequantize_words(w[0], sb[0], o);
                // the codes are in registers: their tile may be copied over
                __syncwarp();
                if (lane == 0) mbar_arrive(barPackEmpty((int)ps));
                ps += 2u;
                if (ps >= args.packStages) {
                    ps -= args.packStages;
                    pPhase ^= 1u;
                }
                // (waited for only here: the conversion above runs under the MMAs that read the stages before)
                if (!mbar_wait_warp<false, Order::kPair>(freeBar, freePhase, &abortFlag)) {
                    ok = false;
                    break;
                }
                freePhase ^= 1u;
                tc_fence_after();
                tc_store_32cols(tmemW, o);
                dequantize_words(w[1], sb[1], o);
                tc_store_32cols(tmemW + 32u, o);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_pair(stepBar);
            }
        }
        scales_arrived();  // nothing of this thread's is in flight when shared memory is released
    } else {
        // ---------------- epilogue: TMEM -> registers -> shared -> global ----------------
        // Two sets of four warps take 32-token chunks (accumulator columns) in turn.  A warp reads its
        // quarter's lanes as 16 x 8 blocks: a thread holds rows r and r + 8 (gate and up of one feature,
        // or two outputs), r = lane / 4, of two neighbouring tokens.  Transposing 8 x 8 stores put the
        // bf16 results into a [token][output] tile in shared memory, which the set then writes out a
        // token row at a time, 16 bytes per thread.  (Two tiles in turn: one is rewritten two chunks
        // later, after every thread has passed the barrier in between.)
        const uint32_t set = (uint32_t)(warp - kFirstEpilogueWarp) >> 2;
        const uint32_t quarter = (uint32_t)(warp & 3);
        const uint32_t te = (uint32_t)threadIdx.x - kFirstEpilogueWarp * 32u;  // 0..255
        const uint32_t t = te & 127u;                                          // within the set
        constexpr uint32_t kPitch = MODE == kModeGateUp ? kStagePitchGateUp : kStagePitchDown;
        constexpr uint32_t kStageBytes = 32u * kPitch;
        uint8_t *stageBuf = epilogueSmem + set * 2u * kStageBytes;
        uint32_t *rowTable = reinterpret_cast<uint32_t *>(epilogueSmem + kEpilogueSets * 2u * kStageBytesDown);  // down only
        uint32_t acc = 0, accPhase = 0, chunk = 0, unitNo = 0;
        bool ok = true;
        // where a row of a unit goes (down), looked up one unit ahead
        auto row_target = [&](const RowTile &tile, uint32_t r) {
            uint32_t outRow = tile.rowStart + min(r, tile.rows - 1u);
            if (args.pairs) {
                const uint4 p = __ldg(reinterpret_cast<const uint4 *>(args.pairs + outRow));
                outRow = p.x * args.topK + p.z;  // token, expert, rank, -
            }
            return outRow;
        };
        RowTile tile{}, next{};
        uint32_t nextTarget = 0;
        if (firstUnit < units) {
            next = tileOf(firstUnit);
            if (MODE == kModeDown) nextTarget = row_target(next, te);
        }
        for (uint32_t u = firstUnit; u < units && ok; u += unitStride, ++unitNo) {
            tile = next;
            next = tileOf(u + unitStride);
            const uint32_t nt = ntOf(u);
            uint32_t *rowOf = rowTable + (unitNo & 1u) * kRowTile;
            if (MODE == kModeDown) {
                if (te < kRowTile) rowOf[te] = nextTarget;
                mbar_arrive(barRows);
                nextTarget = row_target(next, te);
            }
            if (!mbar_wait_idle<Order::kPair>(barAccFull(acc), accPhase, &abortFlag)) break;
            if (MODE == kModeDown && !mbar_wait(barRows, unitNo & 1u, &abortFlag)) break;
            tc_fence_after();
            const uint32_t taddr = tmemBase + acc * args.tileRows + ((quarter * 32u) << 16);
#pragma unroll 1
            for (uint32_t c0 = 32u * set; c0 < tile.rows; c0 += 32u * kEpilogueSets, ++chunk) {
                const uint32_t buffer = chunk & 1u;
                uint8_t *stage = stageBuf + buffer * kStageBytes;
                const uint32_t tokenRow = smem_u32(stage) + (uint32_t)lane * kPitch;  // of token `lane`
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    uint32_t v[16];
                    tc_load_16x32(taddr + ((16u * h) << 16) + c0, v);
                    tc_wait_ld();
                    uint32_t p[4];
                    if (MODE == kModeGateUp) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            float act[2];
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                float g = __uint_as_float(v[4 * j + i]), up = __uint_as_float(v[4 * j + 2 + i]);
                                if (args.roundGateUp) {
                                    g = bf16_round(g);
                                    up = bf16_round(up);
                                }
                                act[i] = gelu_tanh_fast(g) * up;
                            }
                            p[j] = bf16_pair(act[0], act[1]);
                        }
                        store_blocks_transposed(tokenRow + (2u * quarter + h) * 16u, p);
                    } else {
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                p[j] = bf16_pair(__uint_as_float(v[4 * j + 2 * r]), __uint_as_float(v[4 * j + 2 * r + 1]));
                            store_blocks_transposed(tokenRow + (4u * quarter + 2u * h + r) * 16u, p);
                        }
                    }
                }
                mbar_arrive(barStage(set, buffer));
                if (!mbar_wait(barStage(set, buffer), (chunk >> 1) & 1u, &abortFlag)) {
                    ok = false;
                    break;
                }
                // a token row of the tile is 128 (gate/up) or 256 bytes: eight or sixteen threads
                constexpr uint32_t kPieces = MODE == kModeGateUp ? 8 : 16, kTokensPerPass = 128 / kPieces;
                const uint32_t piece = t % kPieces, tok0 = t / kPieces;
                const uint32_t col0 = nt * (8u * kPieces) + piece * 8u;
#pragma unroll
                for (uint32_t tok = tok0; tok < 32u + tok0; tok += kTokensPerPass) {
                    if (c0 + tok < tile.rows && col0 < args.N) {
                        const uint4 val = *reinterpret_cast<const uint4 *>(stage + tok * kPitch + piece * 16u);
                        const uint32_t row = MODE == kModeGateUp ? tile.rowStart + c0 + tok : rowOf[c0 + tok];
                        *reinterpret_cast<uint4 *>(args.out + (size_t)row * args.N + col0) = val;
                    }
                }
            }
            if (!ok) break;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_pair(map_to_cta(barAccEmpty(acc), 0u));
            if (++acc == 2) {
                acc = 0;
                accPhase ^= 1u;
            }
        }
    }

    // teardown: every thread arrives here, also after a wait that ran out
    __syncwarp();
    if (abortFlag) {
        // give copies still in flight time to land before shared memory is released
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
        if (threadIdx.x == 0) atomicExch(args.errorFlag, 1u + (uint32_t)MODE);
    }
    tc_fence_before();
    __syncthreads();
    // neither CTA leaves (or frees its tensor memory) while the other may still arrive on its
    // barriers or have MMAs reading its shared memory
    cluster_sync_all();
    tc_fence_after();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmemBase),
                     "r"(kTmemCols)
                     : "memory");
    }
}

// ---- host side -----------------------------------------------------------------------------

// bf16 activations [rows][k] (row pitch `strideElems`), box 64 x `boxRows` (the half of a row tile that
// one CTA of a pair holds), 128-byte swizzle.
static bool make_activation_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t k,
                                uint64_t strideElems, uint32_t boxRows, const char **error) {
    cuuint64_t dims[2] = {k, rows};
    cuuint64_t strides[1] = {strideElems * 2};
    cuuint32_t box[2] = {(cuuint32_t)kTileK, boxRows};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "activations", error);
}

// router matrix bf16 [experts][d]: boxes of 256 inputs x 8 experts, no swizzle; parts of a box past
// the matrix read as zero.
static bool make_router_map(CUtensorMap *map, const void *base, uint64_t experts, uint64_t d, const char **error) {
    if ((reinterpret_cast<uintptr_t>(base) & 15u) || (d * 2) % 16) return fail(error, "router rows must be 16-byte aligned");
    cuuint64_t dims[2] = {d, experts};
    cuuint64_t strides[1] = {d * 2};
    cuuint32_t box[2] = {(cuuint32_t)kRouterBlockK, (cuuint32_t)kRouterExperts};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, "router", error);
}

// Packed codes of one matrix across all experts seen as 64-bit words [experts][rows][rowBytes/8],
// box `boxBytes` x `boxRows` x 1 without swizzle: a tile of whole row pieces in one copy, rows
// `boxBytes` apart in shared memory.  Out-of-range parts of a box read as zero.
bool make_row_box_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t rowBytes, uint64_t experts,
                      uint64_t expertStride, uint32_t boxBytes, uint32_t boxRows, const char **error) {
    if (rowBytes % 16 || boxBytes % 16 || boxBytes / 8 > 256 || boxRows > 256 || expertStride % 16)
        return fail(error, "row box does not fit a tensor map");
    cuuint64_t dims[3] = {rowBytes / 8, rows, experts};
    cuuint64_t strides[2] = {rowBytes, expertStride ? expertStride : rows * rowBytes};
    cuuint32_t box[3] = {boxBytes / 8, boxRows, 1};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, "row boxes", error);
}

// Packed codes of one matrix across all experts: bytes [experts][rows][cols/2], box 64 rows x 128 bytes (four
// steps; parts past a row read as zero), 128-byte swizzle so that a warp's 128-bit reads of 32 rows meet no
// bank twice.  (Boxes of one step's 32 bytes kept the copying thread busy for 600 cycles a step.)
static bool make_weight_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols,
                            uint64_t experts, uint64_t expertStride, const char **error) {
    cuuint64_t dims[3] = {cols / 2, rows, experts};
    cuuint64_t strides[2] = {cols / 2, expertStride};
    cuuint32_t box[3] = {(cuuint32_t)(kQuad * kTileK / 2), 64, 1};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "weights", error);
}

bool prefill_prepare_layer(FFContext *ctx, LayerStore &L, const char **error) {
    if (L.mapsReady) return true;
    const FFConfig &c = ctx->cfg;
    if (L.experts) {
        const uint32_t *o = &L.off.gateWOff;
        for (int m = 0; m < 3; ++m) {
            const uint64_t rows = m == 2 ? c.d : c.f, cols = m == 2 ? c.f : c.d;
            if (!make_weight_map(&L.routedMap[m], L.experts + o[3 * m], rows, cols, L.expertCount,
                                 L.stride, error))
                return false;
        }
    }
    if (L.shared) {
        const uint32_t *o = &L.sharedOff.gateWOff;
        uint64_t payload = 0;
        packed_offsets(c.d, c.sharedF, &payload);
        for (int m = 0; m < 3; ++m) {
            const uint64_t rows = m == 2 ? c.d : c.sharedF, cols = m == 2 ? c.sharedF : c.d;
            if (!make_weight_map(&L.sharedMap[m], L.shared + o[3 * m], rows, cols, 1,
                                 (payload + 15) & ~15ull, error))
                return false;
        }
    }
    L.mapsReady = true;
    return true;
}

// Slots that the code ring needs at least.  A group takes every second quad, so in a ring of odd length it skips every second
// phase of a slot, and its parity says nothing about the phase it skips.  What orders that phase is the pair that the group
// stored last: it waited for the MMAs `weightStages / 2` pairs further back, so quads up to 2 + weightStages / 4 back have
// landed.  (Three slots with eight weight stages were one short: a conversion could start on the slot's former codes.)
__host__ __device__ constexpr uint32_t min_pack_stages(uint32_t weightStages) { return 2u + weightStages / 4u; }

// Sizes of a GEMM's rings for a contraction of K.
struct GemmRings {
    uint32_t packStages;    // quads of packed codes
    uint32_t scaleBuffers;  // units whose scale words are held: 2 (one ahead), 1 (the unit's own) or 0 (read step by step)
    size_t smem;
};
static GemmRings gemm_rings(int mode, uint32_t K, uint32_t tileRows) {
    const uint32_t quads = (K / kTileK + kQuad - 1) / kQuad;
    GemmRings r{min_pack_stages(weight_stages(tileRows)), 2, 0};
    const auto bytes = [&] {
        return 1024 + (size_t)kTokStages * 2 * tok_tile_bytes(tileRows) + (size_t)r.packStages * kPackTileBytes +
               (mode == kModeGateUp ? kEpilogueBytesGateUp : kEpilogueBytesDown) + (size_t)r.scaleBuffers * scale_buffer_bytes(quads);
    };
    while (r.scaleBuffers && bytes() > 226 * 1024) --r.scaleBuffers;
    while (r.packStages < (uint32_t)kMaxPackStages && bytes() + kPackTileBytes <= 226 * 1024) ++r.packStages;
    r.smem = bytes();
    return r;
}

// Rows of a routed GEMM's tiles.  Tiles of 128 rows leave tensor memory for eight weight stages instead of four, and a
// step of few columns then costs what its conversion does; tiles of 192 convert an expert's weights fewer times.
// Whole layer of d 2816, f 704, shared 2112, us with 128 / 192: 77 rows (5 an expert) 146 / 155, 613 (38) 203 / 209,
// 1400 (87) 291 / 298, 1500 (94) 313 / 313, 2000 (125) 373 / 357, 4096 648 / 634.
static uint32_t routed_tile_rows(uint32_t pairs, uint32_t experts) { return pairs <= 96u * experts ? kRowTileSmall : kRowTile; }

// Of the shared FFN's two GEMMs: where whole waves of a step take less time; a step of 192 rows takes 1.36 times one of 128
// (their columns 1.5).  And tiles of 128 rows while gate/up has at most two waves of them, unless those of 192 save both
// GEMMs a wave: the second is mostly the last row tile's units, which have few columns.  us with 128 / 192 (d x f, waves of
// gate/up and down): 2816 x 2112, 77 rows (1, 1 / 1, 1) 23.7 / 25.8, 613 (2, 1 / 1, 1) 34.1 / 38.4, 1500 50.6 / 55.3, 3000 97.9 / 89.9,
// 4096 124.5 / 130.2; 4096 x 2048, 613 rows (2, 2 / 1, 1) 50.9 / 42.1; 6144 x 1024, 1500 rows (2, 4 / 1, 3) 64.8 / 54.8; 5120 x 1536, 3000
// rows (4, 7 / 3, 5) 118.4 / 125.3; 2816 x 6144, 300 rows 46.5 / 53.9, 1000 101.0 / 85.8, 4096 (21, 5 / 15, 4) 326.9 / 342.6.
static uint32_t dense_tile_rows(uint32_t smCount, uint32_t d, uint32_t f, uint32_t tokens) {
    const uint32_t clusters = std::max(1u, smCount / 2u);
    const auto waves = [&](uint32_t rows, uint32_t nTiles) {
        return ((uint64_t)((tokens + rows - 1u) / rows) * ((nTiles + 1u) / 2u) + clusters - 1u) / clusters;
    };
    const uint32_t gateUp = (f + 63u) / 64u, down = (d + 127u) / 128u;
    const uint64_t gSmall = waves(kRowTileSmall, gateUp), dSmall = waves(kRowTileSmall, down);
    const uint64_t gLarge = waves(kRowTile, gateUp), dLarge = waves(kRowTile, down);
    if (gSmall <= 2u && (gLarge == gSmall || dLarge == dSmall)) return kRowTileSmall;
    return (gSmall * d + dSmall * f) * 100u <= (gLarge * d + dLarge * f) * 136u ? kRowTileSmall : kRowTile;
}

// `rows` activation rows of args.K elements at `x`
template <int MODE>
static bool launch_gemm(FFContext *ctx, const uint16_t *x, uint64_t rows, const CUtensorMap &mapW0,
                        const CUtensorMap &mapW1, GemmArgs args, uint32_t maxUnits,
                        cudaStream_t stream, const char **error) {
    CUtensorMap mapA, mapASmall;
    if (!make_activation_map(&mapA, x, rows, args.K, args.K, args.tileRows / 2, error) ||
        !make_activation_map(&mapASmall, x, rows, args.K, args.K, kTokSmallRows, error))
        return false;
    auto kernel = k_grouped_int4_gemm<MODE>;
    const GemmRings rings = gemm_rings(MODE, args.K, args.tileRows);
    args.packStages = rings.packStages;
    args.scaleBuffers = rings.scaleBuffers;
    const size_t smem = rings.smem;
    static KernelSmemMemo memo;
    if (!memo.prepare(kernel, ctx->device, smem, kGemmThreads, nullptr, error)) return false;
    // clusters of two CTAs; a cluster takes (row tile, pair of weight-row tiles) units
    const uint32_t pairUnits = (maxUnits + 1) / 2 + 1;
    const uint32_t grid = 2u * std::max(1u, std::min<uint32_t>((uint32_t)ctx->smCount / 2u, pairUnits));
    {
        LaunchScope scope(ctx, stream, MODE == kModeGateUp ? "int4_gemm_gate_up_act" : "int4_gemm_down");
        FF_CUDA_OK(launch_pdl(kernel, grid, kGemmThreads, smem, stream,
                              mapA, mapASmall, mapW0, mapW1, args),
                   error);
    }
    return true;
}

static bool check_gemm_shapes(const FFConfig &c, uint32_t f, const char **error) {
    if (c.d % 64 || f % 64) return fail(error, "GEMM path needs widths that are multiples of 64");
    return true;
}

// Whether k_route_sort takes less time than the three launches: it grows with the routes (3.1 us and 0.4 for every 1024),
// they with the routes of a block of 256 rows.  us in a graph, 128 experts, one launch / three: one route a row 8192 routes 6.5 /
// 7.3, 16384 9.6 / 8.8, 32768 16.0 / 12.2; two a row 8192 6.4 / 8.4, 16384 9.6 / 9.0, 32768 16.1 / 10.9; four a row 16384 9.6 /
// 11.2, 24576 12.9 / 11.7; eight a row 32768 16.3 / 18.0.
static bool sort_in_one_launch(uint32_t tokens, uint32_t topK) {
    return tokens * topK <= 8192u + 3072u * topK && (tokens + kSortCtas - 1) / kSortCtas * topK <= (uint32_t)(kClusterRoutes / kSortCtas);
}

// Sorts the routes (stable, by expert) and plans the row tiles.
static bool sort_routes(FFContext *ctx, const uint32_t *ids, uint32_t tokens, int E, uint32_t tileRows, uint32_t *offsets, RowTile *tiles,
                              FFTokenExpertPair *sorted, uint32_t *rowOfRoute, cudaStream_t stream, const char **error) {
    const int T = (int)tokens, K = (int)ctx->cfg.topK;
    const uint32_t blocks = (tokens + kSortTokens - 1) / kSortTokens;
    const size_t sortSmem = (size_t)kSortTokens * K * sizeof(uint32_t);
    const uint32_t maxTiles = ctx->maxUnits / 2;  // first half of the tile buffer
    if (sort_in_one_launch(tokens, ctx->cfg.topK)) {
        LaunchScope scope(ctx, stream, "route_sort");
        FF_CUDA_OK(launch_pdl(k_route_sort, kSortCtas, kSortThreads, 0, stream, ids, T, K, E, tileRows, offsets, tiles, maxTiles, ctx->unitCount, sorted,
                              rowOfRoute),
                   error);
        return true;
    }
    {
        LaunchScope scope(ctx, stream, "route_count");
        FF_CUDA_OK(launch_pdl(k_route_count, blocks, 256, sortSmem, stream, ids, T, K, E, ctx->blockCounts), error);
    }
    {
        LaunchScope scope(ctx, stream, "route_scan");
        FF_CUDA_OK(launch_pdl(k_route_scan, 1, 256, 0, stream, ctx->blockCounts, (int)blocks, E, tileRows, offsets, tiles, maxTiles, ctx->unitCount),
                   error);
    }
    LaunchScope scope(ctx, stream, "route_scatter");
    FF_CUDA_OK(launch_pdl(k_route_scatter, blocks, 256, sortSmem, stream, ids, T, K, E, ctx->blockCounts, offsets, sorted,
                          rowOfRoute),
               error);
    return true;
}

bool launch_prefill_routed(FFContext *ctx, LayerStore &L, const uint16_t *x, uint32_t xStride,
                           uint32_t tokens, const uint32_t *ids, uint16_t *partials,
                           cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (tokens == 0) return true;
    if (!ctx->xSorted) return fail(error, "context was created with maxTokens <= 16: no prefill scratch");
    if (!L.experts) return fail(error, "layer has no resident experts");
    if (!check_gemm_shapes(c, c.f, error) || !prefill_prepare_layer(ctx, L, error)) return false;
    const int K = (int)c.topK, E = (int)L.expertCount;
    RowTile *tiles = reinterpret_cast<RowTile *>(ctx->units);
    const uint32_t tileRows = routed_tile_rows(tokens * c.topK, (uint32_t)E);
    if (!sort_routes(ctx, ids, tokens, E, tileRows, ctx->expertOffsets, tiles, ctx->sortedPairs, ctx->rowOfRoute, stream, error)) return false;
    const uint32_t pairs = tokens * c.topK;
    {
        LaunchScope scope(ctx, stream, "gather_rows");
        FF_CUDA_OK(launch_pdl(k_gather_rows, ctx->smCount * 8, 256, 0, stream,
                              x, xStride, tokens, ctx->rowOfRoute, K, (int)c.d, ctx->xSorted),
                   error);
    }

    const uint32_t tileBound = pairs / tileRows + (uint32_t)E;
    const uint64_t rows = (uint64_t)pairs + 256;
    GemmArgs a{};
    a.tileRows = tileRows;
    a.scaleWords = L.routedScales;
    a.scaleStride = scale_words(c.d, c.f);
    a.K = c.d;
    a.N = c.f;
    a.nTiles = (c.f + 63) / 64;
    a.tiles = tiles;
    a.counts = ctx->unitCount;
    a.out = ctx->acts;
    a.pairs = nullptr;
    a.topK = c.topK;
    a.roundGateUp = 0;
    a.errorFlag = ctx->errorFlag;
    if (!launch_gemm<kModeGateUp>(ctx, ctx->xSorted, rows, L.routedMap[0], L.routedMap[1], a, tileBound * a.nTiles,
                                  stream, error))
        return false;

    GemmArgs b = a;
    b.scaleWords = L.routedScales + scale_words_gate_up(c.d, c.f);
    b.K = c.f;
    b.N = c.d;
    b.nTiles = (c.d + 127) / 128;
    b.out = partials;
    b.pairs = ctx->sortedPairs;
    return launch_gemm<kModeDown>(ctx, ctx->acts, rows, L.routedMap[2], L.routedMap[2], b, tileBound * b.nTiles,
                                  stream, error);
}

// The stable counting sort of routes by a group id, on its own: `groupIds` [tokens][K] on the device
// (ids >= groups are dropped), `sortedPairs` receives (token, group, rank, 0) in (group, token,
// rank) order, `offsets` [groups + 1] the first row of every group.  Uses the context's permute
// scratch.
bool launch_route_sort(FFContext *ctx, const uint32_t *groupIds, uint32_t tokens, uint32_t groups,
                       FFTokenExpertPair *sortedPairs, uint32_t *offsets, cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (tokens == 0) return true;
    if (!ctx->xSorted) return fail(error, "context was created with maxTokens <= 16: no prefill scratch");
    if (groups == 0 || groups > c.experts) return fail(error, "group count must be 1..experts of the context");
    if (tokens > c.maxTokens) return fail(error, "rows exceed the context's maxTokens");
    return sort_routes(ctx, groupIds, tokens, (int)groups, kRowTile, offsets, reinterpret_cast<RowTile *>(ctx->units), sortedPairs, nullptr, stream,
                       error);
}

bool launch_prefill_shared(FFContext *ctx, LayerStore &L, const uint16_t *x, uint32_t xStride,
                           uint32_t tokens, uint16_t *y, cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (tokens == 0) return true;
    if (!ctx->xShared) return fail(error, "context was created with maxTokens <= 16: no prefill scratch");
    if (!L.shared) return fail(error, "layer has no resident shared FFN");
    if (!check_gemm_shapes(c, c.sharedF, error) || !prefill_prepare_layer(ctx, L, error)) return false;
    // dense problem: its row tiles live behind the routed ones in the units buffer
    RowTile *tiles = reinterpret_cast<RowTile *>(ctx->units) + ctx->maxUnits / 2;
    uint32_t *counts = ctx->unitCount + 4;
    const uint32_t tileRows = dense_tile_rows((uint32_t)ctx->smCount, c.d, c.sharedF, tokens);
    {
        LaunchScope scope(ctx, stream, "dense_tiles");
        FF_CUDA_OK(launch_pdl(k_dense_tiles, 1, 256, 0, stream,
                              (int)tokens, (int)tileRows, tiles, counts),
                   error);
    }
    {
        LaunchScope scope(ctx, stream, "gather_rows");
        FF_CUDA_OK(launch_pdl(k_gather_rows, ctx->smCount * 8, 256, 0, stream,
                              x, xStride, tokens, nullptr, 0, (int)c.d, ctx->xShared),
                   error);
    }
    const uint32_t rowTiles = (tokens + tileRows - 1) / tileRows;
    const uint64_t rows = (uint64_t)tokens + 256;
    GemmArgs a{};
    a.tileRows = tileRows;
    a.scaleWords = L.sharedScales;
    a.K = c.d;
    a.N = c.sharedF;
    a.nTiles = (c.sharedF + 63) / 64;
    a.tiles = tiles;
    a.counts = counts;
    a.out = ctx->sharedActs;
    a.topK = c.topK;
    a.roundGateUp = 1;
    a.errorFlag = ctx->errorFlag;
    if (!launch_gemm<kModeGateUp>(ctx, ctx->xShared, rows, L.sharedMap[0], L.sharedMap[1], a, rowTiles * a.nTiles, stream,
                                  error))
        return false;
    GemmArgs b = a;
    b.scaleWords = L.sharedScales + scale_words_gate_up(c.d, c.sharedF);
    b.K = c.sharedF;
    b.N = c.d;
    b.nTiles = (c.d + 127) / 128;
    b.out = y;
    b.pairs = nullptr;
    return launch_gemm<kModeDown>(ctx, ctx->sharedActs, rows, L.sharedMap[2], L.sharedMap[2], b, rowTiles * b.nTiles,
                                  stream, error);
}

}  // namespace ff

// For the host-side tests, not part of the interface: packed-code stages, weight stages, scale buffers and shared memory
// of the GEMM over K (mode 0 gate/up, 1 down) with tiles of `tileRows` rows.
extern "C" void ff_prefill_gemm_rings(uint32_t mode, uint32_t K, uint32_t tileRows, uint32_t *sizes) {
    const ff::GemmRings r = ff::gemm_rings((int)mode, K, tileRows);
    sizes[0] = r.packStages;
    sizes[1] = ff::weight_stages(tileRows);
    sizes[2] = r.scaleBuffers;
    sizes[3] = (uint32_t)r.smem;
}
// ... and the rows of the shared FFN's tiles.
extern "C" uint32_t ff_prefill_dense_tile_rows(uint32_t smCount, uint32_t d, uint32_t f, uint32_t tokens) {
    return ff::dense_tile_rows(smCount, d, f, tokens);
}

extern "C" bool ff_last_prefill_routes(FFContext *ctx, FFTokenExpertPair *sortedPairs,
                                       uint32_t *offsets, const char **error) {
    using namespace ff;
    if (error) *error = nullptr;
    if (!ctx || !sortedPairs || !offsets) return fail(error, "null argument");
    if (!ctx->sortedPairs) return fail(error, "context has no prefill scratch");
    FF_CUDA_OK(cudaSetDevice(ctx->device), error);
    FF_CUDA_OK(cudaDeviceSynchronize(), error);
    uint32_t counts[4] = {0, 0, 0, 0};
    FF_CUDA_OK(cudaMemcpy(counts, ctx->unitCount, sizeof(counts), cudaMemcpyDeviceToHost), error);
    FF_CUDA_OK(cudaMemcpy(sortedPairs, ctx->sortedPairs, (size_t)counts[1] * sizeof(FFTokenExpertPair),
                          cudaMemcpyDeviceToHost),
               error);
    FF_CUDA_OK(cudaMemcpy(offsets, ctx->expertOffsets, (size_t)(ctx->cfg.experts + 1) * sizeof(uint32_t),
                          cudaMemcpyDeviceToHost),
               error);
    return true;
}
