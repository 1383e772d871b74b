// Router of a prefill chunk (more rows than a decode/verify block) when only the routes are asked for: few pairs of row and
// expert have every logit formed in one launch (k_router_tile), more as follows.
//
// The contract is bitwise: logits are sums in a fixed fp32 order (bf16 router: lane l chains fmaf over
// [256 i + 8 l, +8); INT8 router: over elements 64 g + 2 l, + 1; xor butterfly; then the logit bias),
// and the K largest are taken, ties to the lower id.  Forming all of them in that order costs 2 D E
// serial fp32 operations a row (160 us for 4096 rows of 2816 x 128; the INT8 order 480 us), although
// only about nine of 128 matter.  So:
//   1. k_router_approx: all logits on the tensor cores (bf16 products, fp32 sums in any order);
//   2. k_router_select: a warp per row bounds how far each exact logit can be from its approximation,
//      keeps every expert that can be among the K largest, forms those logits in the contract's order
//      and ranks them.
// The bound holds for any data: with unspecified rounding at single precision or better, a sum of n
// products is within n 2^-23 sum|w x| of its value (the fixed-order sum likewise, with its own n), a
// folded weight bf16(w * scale) within 2^-9 |w scale|, and sum|w x| <= |w| |x| in 2-norms.  The norms are
// formed where squares neither vanish nor overflow.  What underflows, flushed to zero or not, adds at most
// 2^-126 per operation and operand (RouterBound::floor, and a part of perNorm); rows so large that a term
// or a partial sum could overflow in some order (RouterBound::limit), or that hold a NaN or an infinity, keep
// every expert, so at worst every logit is formed exactly.
//
// Rows of 2816 inputs, 128 experts: 4096 rows 160 us with every logit in that order, 16 + 42 us now; INT8, 2000
// rows 264 us, 13 + 50 us now.  Bound by the latency and the L2 traffic of the exact logits (nine or ten
// router rows per token).
#include <algorithm>

#include "ff_gemv_device.cuh"
#include "ff_internal.cuh"
#include "ff_tc_device.cuh"

namespace ff {
namespace {

// ---- 1. approximate logits -----------------------------------------------------------------------

constexpr int kApproxStages = 3;
constexpr uint32_t kExpertTile = 128, kApproxK = 64;
constexpr uint32_t kExpertBytes = kExpertTile * kApproxK * 2;
constexpr uint32_t kMaxSplits = 8;   // parts of the contraction, summed by the selecting kernel
constexpr int kApproxThreads = 192;  // warp 0 copies, warp 1 MMAs, warps 2-5 write out

__device__ __forceinline__ void mma_bf16_ss(uint32_t tmemD, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmemD),
        "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void commit_one(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// CTA (token tile, expert tile, split): parts[split][token][expert] = sum over the split's inputs.
// Experts are the MMA's rows (TMEM lanes), tokens its columns.
__global__ void __launch_bounds__(kApproxThreads)
k_router_approx(const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapX, uint32_t tileTokens,
                uint32_t tokens, uint32_t E, uint32_t steps, uint32_t splits, float *parts, uint32_t *errorFlag) {
    extern __shared__ uint8_t smemRaw[];
    __shared__ uint64_t barriers[2 * kApproxStages + 1];
    __shared__ uint32_t tmemBaseSlot;
    __shared__ volatile uint32_t abortFlag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smemRaw) + 1023u) & ~1023u;
    const uint32_t stageBytes = kExpertBytes + tileTokens * kApproxK * 2;
    const uint32_t barBase = smem_u32(barriers);
    auto barFull = [&](uint32_t s) { return barBase + 8u * s; };
    auto barEmpty = [&](uint32_t s) { return barBase + 8u * (kApproxStages + s); };
    const uint32_t barDone = barBase + 16u * kApproxStages;
    const uint32_t perSplit = (steps + splits - 1) / splits;
    const uint32_t g0 = blockIdx.z * perSplit, g1 = min(steps, g0 + perSplit);
    const uint32_t token0 = blockIdx.x * tileTokens, expert0 = blockIdx.y * kExpertTile;
    if (threadIdx.x == 0) {
        abortFlag = 0;
        for (uint32_t s = 0; s < kApproxStages; ++s) {
            mbar_init(barFull(s), 1);
            mbar_init(barEmpty(s), 1);
        }
        mbar_init(barDone, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemBaseSlot)),
                     "r"(kExpertTile)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmemBase = tmemBaseSlot;
    pdl_enter();
    if (warp == 0) {
        if (lane == 0) {
            uint32_t st = 0, phase = 0;
            for (uint32_t g = g0; g < g1; ++g) {
                if (!mbar_wait(barEmpty(st), phase ^ 1u, &abortFlag)) break;
                mbar_expect_tx(barFull(st), stageBytes);
                tma_load_2d(base + st * stageBytes, &mapW, (int)(g * kApproxK), (int)expert0, barFull(st));
                tma_load_2d(base + st * stageBytes + kExpertBytes, &mapX, (int)(g * kApproxK), (int)token0, barFull(st));
                if (++st == kApproxStages) {
                    st = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((tileTokens >> 3) << 17) | ((kExpertTile >> 4) << 24);
            uint32_t st = 0, phase = 0;
            bool ok = true;
            for (uint32_t g = g0; g < g1; ++g) {
                if (!mbar_wait(barFull(st), phase, &abortFlag)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t a = umma_desc_sw128(base + st * stageBytes), b = umma_desc_sw128(base + st * stageBytes + kExpertBytes);
#pragma unroll
                for (uint32_t kk = 0; kk < kApproxK / 16; ++kk)
                    mma_bf16_ss(tmemBase, a + 2u * kk, b + 2u * kk, idesc, (g > g0 || kk) ? 1u : 0u);
                commit_one(barEmpty(st));
                if (++st == kApproxStages) {
                    st = 0;
                    phase ^= 1u;
                }
            }
            if (ok) commit_one(barDone);
        }
    } else if (mbar_wait_idle(barDone, 0, &abortFlag)) {
        tc_fence_after();
        const uint32_t quarter = (uint32_t)(warp & 3), e = expert0 + quarter * 32u + (uint32_t)lane;
        float *out = parts + ((size_t)blockIdx.z * tokens + token0) * E;
        for (uint32_t c0 = 0; c0 < tileTokens && token0 + c0 < tokens; c0 += 32) {
            uint32_t v[32];
            tc_load_32cols(tmemBase + ((quarter * 32u) << 16) + c0, v);
            tc_wait_ld();
#pragma unroll
            for (uint32_t j = 0; j < 32; ++j)
                if (e < E && token0 + c0 + j < tokens) out[(size_t)(c0 + j) * E + e] = __uint_as_float(v[j]);
        }
    }
    __syncwarp();
    if (abortFlag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);  // copies in flight land before shared memory is released
        if (threadIdx.x == 0) atomicExch(errorFlag, 11u);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(kExpertTile) : "memory");
}

// ---- 2. exact logits of the experts that can matter, and the top K --------------------------------

// Warps of a CTA; `warpsPerRow` (1, 2, 4 or 8) of them share a row.
constexpr int kSelectWarps = 8;

// Butterfly 16, 8, 4, 2, 1 over N values per lane at once: every level halves the values a lane carries
// (a lane keeps the ones of its side), the additions are those of N separate butterflies.  Returns the
// sum of value index `which` (the same for all lanes that differ only in the low bits).
template <int N>
__device__ __forceinline__ float butterfly(float (&v)[N], int lane, int &which) {
    int offset = 16;
    which = 0;
#pragma unroll
    for (int n = N; n > 1; n >>= 1, offset >>= 1) {
        const bool upper = lane & offset;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            if (i < n / 2) {
                const float give = upper ? v[i] : v[i + n / 2], keep = upper ? v[i + n / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, give, offset);
            }
        }
        which = which * 2 + (upper ? 1 : 0);
    }
    float s = v[0];
    for (; offset >= 1; offset >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, offset);
    return s;
}

// Group i of eight in an INT8 router row: lane codes q (two per group), aux = scale | bias << 16 per group.
// acc = fma(s, fma(q1, x1, q0 x0), acc); acc = fma(b, x0 + x1, acc): the reference kernel's order
// (Metal/MoE/moe.metal:65-103) made definite.
__device__ __forceinline__ float int8_group(const uint4 &q, const uint4 (&aux)[2], int i, float x0, float x1, float xsum, float acc) {
    const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
    const uint32_t aw[8] = {aux[0].x, aux[0].y, aux[0].z, aux[0].w, aux[1].x, aux[1].y, aux[1].z, aux[1].w};
    const uint32_t two = (i & 1) ? qw[i >> 1] >> 16 : qw[i >> 1];
    const float q0 = (float)(two & 0xFFu), q1 = (float)((two >> 8) & 0xFFu);
    acc = fmaf(__uint_as_float(aw[i] << 16), fmaf(q1, x1, q0 * x0), acc);
    return fmaf(__uint_as_float(aw[i] & 0xFFFF0000u), xsum, acc);
}

struct SelectArgs {
    const uint16_t *W;               // bf16 router [E][D]
    const uint4 *Q;                  // INT8 router in lane order (see k_router_int8_lanes)
    const uint32_t *qAux;
    const uint16_t *scale, *gain;    // per input, per expert; or null
    const float *bias;               // logit bias or null
    const RouterBound *bounds;       // [E]
    const uint16_t *x;
    uint32_t xStride, splits, warpsPerRow;
    int T, E, D, K;
    const float *parts;              // [splits][T][E]
    uint32_t *ids;
    uint16_t *weights;
};

// Exact logits (before the bias) of N experts for the bf16 row staged at `xs`, into out[0..N).
template <int N>
__device__ __forceinline__ void exact_bf16(const SelectArgs &a, const uint4 *xs, const uint16_t *experts, float *out, int lane) {
    const uint4 *W = reinterpret_cast<const uint4 *>(a.W);
    const int chunks = a.D >> 3;
    float acc[N];
    uint32_t row[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        acc[n] = 0.0f;
        row[n] = (uint32_t)experts[n] * (uint32_t)chunks;
    }
#pragma unroll(N > 4 ? 1 : 2)
    for (int c = lane; c < chunks; c += 32) {
        uint4 wv[N];
#pragma unroll
        for (int n = 0; n < N; ++n) wv[n] = __ldg(W + row[n] + c);
        const uint4 xv = xs[c];
        float xe[8] = {__uint_as_float(xv.x << 16), __uint_as_float(xv.x & 0xFFFF0000u), __uint_as_float(xv.y << 16),
                       __uint_as_float(xv.y & 0xFFFF0000u), __uint_as_float(xv.z << 16), __uint_as_float(xv.z & 0xFFFF0000u),
                       __uint_as_float(xv.w << 16), __uint_as_float(xv.w & 0xFFFF0000u)};
        if (a.scale) {
            const uint4 sv = __ldg(reinterpret_cast<const uint4 *>(a.scale) + c);
            const uint32_t ss[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                xe[2 * k] = xe[2 * k] * __uint_as_float(ss[k] << 16);
                xe[2 * k + 1] = xe[2 * k + 1] * __uint_as_float(ss[k] & 0xFFFF0000u);
            }
        }
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const uint32_t ww[4] = {wv[n].x, wv[n].y, wv[n].z, wv[n].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc[n] = fmaf(__uint_as_float(ww[k] << 16), xe[2 * k], acc[n]);
                acc[n] = fmaf(__uint_as_float(ww[k] & 0xFFFF0000u), xe[2 * k + 1], acc[n]);
            }
        }
    }
    int which;
    const float v = butterfly<N>(acc, lane, which);
    if ((lane & (32 / N - 1)) == 0) out[which] = v;
}

__device__ __forceinline__ void exact_pair_int8(const SelectArgs &a, const float2 *xs, uint32_t e0, uint32_t e1, float *out, int lane) {
    const int groups = a.D >> 6, runs = (groups + 7) >> 3;
    const uint4 *q0 = a.Q + (size_t)e0 * runs * 32 + lane, *q1 = a.Q + (size_t)e1 * runs * 32 + lane;
    const uint4 *b0 = reinterpret_cast<const uint4 *>(a.qAux + (size_t)e0 * runs * 8), *b1 = reinterpret_cast<const uint4 *>(a.qAux + (size_t)e1 * runs * 8);
    float acc[2] = {0.0f, 0.0f};
    for (int r = 0; r < runs; ++r) {
        const uint4 qa = __ldg(q0 + r * 32), qb = __ldg(q1 + r * 32);
        const uint4 sa[2] = {__ldg(b0 + 2 * r), __ldg(b0 + 2 * r + 1)}, sb[2] = {__ldg(b1 + 2 * r), __ldg(b1 + 2 * r + 1)};
        const int n = min(8, groups - 8 * r);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (i < n) {
                const float2 xv = xs[(8 * r + i) * 32 + lane];
                const float sum = xv.x + xv.y;
                acc[0] = int8_group(qa, sa, i, xv.x, xv.y, sum, acc[0]);
                acc[1] = int8_group(qb, sb, i, xv.x, xv.y, sum, acc[1]);
            }
        }
    }
    int which;
    const float v = butterfly<2>(acc, lane, which);
    if ((lane & 15) == 0) out[which] = v;
}

// `warpsPerRow` warps per row: all stage the row (bf16; INT8: fp32 times the per-input scale, which
// keeps that work out of the pairs' loops), the first one picks the experts to form exactly, all form
// them a few at a time, the first one ranks them.
template <bool INT8>
__global__ void __launch_bounds__(kSelectWarps * 32, INT8 ? 4 : 3)
k_router_select(const SelectArgs a) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t selectSmem[];
    constexpr int kMaxRows = INT8 ? kSelectWarps / 2 : kSelectWarps;
    __shared__ uint16_t sExpert[kMaxRows][kMaxExperts + 8];
    __shared__ float sLogit[kMaxRows][kMaxExperts + 8];
    __shared__ float sTopScore[kMaxRows][8];
    __shared__ uint32_t sTopId[kMaxRows][8];
    __shared__ int sKept[kMaxRows];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp / (int)a.warpsPerRow, sub = warp - slot * (int)a.warpsPerRow;
    const int t = (int)blockIdx.x * (kSelectWarps / (int)a.warpsPerRow) + slot;
    const bool live = t < a.T;
    const int E = a.E, K = a.K;
    uint8_t *xs = selectSmem + (size_t)slot * a.D * (INT8 ? 4 : 2);
    const uint16_t *xr = a.x + (size_t)(live ? t : 0) * a.xStride;
    float approx[8];
    if (live && sub == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = j * 32 + lane;
            approx[j] = 0.0f;
            if (e < E)
                for (uint32_t p = 0; p < a.splits; ++p) approx[j] += __ldg(a.parts + ((size_t)p * a.T + t) * E + e);
        }
    }
    if (live) {
        for (int c = sub * 32 + lane; c < (a.D >> 3); c += (int)a.warpsPerRow * 32) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(xr) + c);
            if (!INT8) {
                reinterpret_cast<uint4 *>(xs)[c] = v;
                continue;
            }
            uint4 sv = make_uint4(0, 0, 0, 0);
            if (a.scale) sv = __ldg(reinterpret_cast<const uint4 *>(a.scale) + c);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w}, f[4] = {sv.x, sv.y, sv.z, sv.w};
            float xe[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                xe[2 * k] = __uint_as_float(w[k] << 16);
                xe[2 * k + 1] = __uint_as_float(w[k] & 0xFFFF0000u);
                if (a.scale) {
                    xe[2 * k] = xe[2 * k] * __uint_as_float(f[k] << 16);
                    xe[2 * k + 1] = xe[2 * k + 1] * __uint_as_float(f[k] & 0xFFFF0000u);
                }
            }
            float4 *dst = reinterpret_cast<float4 *>(xs);
            dst[2 * c] = make_float4(xe[0], xe[1], xe[2], xe[3]);
            dst[2 * c + 1] = make_float4(xe[4], xe[5], xe[6], xe[7]);
        }
    }
    if (live && sub == 0) {
        auto square_sum = [&](float scale) {
            float sq = 0.0f;
            for (int i = lane; i < (a.D >> 3); i += 32) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(xr) + i);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float lo = __uint_as_float(w[k] << 16) * scale, hi = __uint_as_float(w[k] & 0xFFFF0000u) * scale;
                    sq = fmaf(lo, lo, sq);
                    sq = fmaf(hi, hi, sq);
                }
            }
#pragma unroll
            for (int offset = 16; offset >= 1; offset >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, offset);
            return sq;
        };
        // (below 2^-100 the squares lose digits or vanish: every |x| is below 2^-50 then, so 2^100 times the row has
        // squares from 2^-66 to 2^100)
        const float sq = square_sum(1.0f);
        const float norm = sq < 0x1p-100f ? sqrtf(square_sum(0x1p100f)) * 1.01f * 0x1p-100f : sqrtf(sq) * 1.01f;

        // the K-th largest lower bound; an expert whose upper bound reaches it can be among the K largest
        uint32_t low[8];
        float high[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = j * 32 + lane;
            low[j] = 0u;  // below every float's
            high[j] = -INFINITY;
            if (e < E) {
                const float l = a.bias ? approx[j] + a.bias[e] : approx[j];
                const RouterBound bound = a.bounds[e];
                const float eps = fmaf(bound.perNorm, norm, fmaf(fabsf(l), 2.5e-7f, bound.floor));
                const float lo = l - eps, hi = l + eps;
                const bool bounded = norm < bound.limit && lo > -INFINITY && hi < INFINITY;  // false for NaN, too
                low[j] = bounded ? ordered_key(lo) : 0u;
                // (a bias of -inf makes a logit that is never taken, whatever the sum)
                high[j] = bounded ? hi : a.bias && a.bias[e] == -INFINITY ? -INFINITY : INFINITY;
            }
        }
        uint32_t threshold = 0u, gone = 0u;
        for (int r = 0; r < K; ++r) {
            uint32_t best = 0u;
            int at = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (!((gone >> j) & 1u) && low[j] > best) {
                    best = low[j];
                    at = j;
                }
            threshold = __reduce_max_sync(0xFFFFFFFFu, best);
            if (threshold == 0u) break;
            const uint32_t holders = __ballot_sync(0xFFFFFFFFu, best == threshold);
            if (lane == __ffs(holders) - 1) gone |= 1u << at;
        }
        const float cut = threshold ? from_ordered_key(threshold) : -INFINITY;
        int kept = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const bool keep = j * 32 + lane < E && high[j] >= cut;
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, keep);
            if (keep) sExpert[slot][kept + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)(j * 32 + lane);
            kept += __popc(mask);
        }
        __syncwarp();
        if (lane < 7) sExpert[slot][kept + lane] = kept ? sExpert[slot][0] : (uint16_t)0;  // the last few are filled up
        if (lane == 0) sKept[slot] = kept;
        if (lane < 8) {
            sTopScore[slot][lane] = -INFINITY;
            sTopId[slot][lane] = 0u;
        }
    }
    if (a.warpsPerRow > 1) __syncthreads();
    else __syncwarp();  // a row is one warp's business
    const int kept = live ? sKept[slot] : 0;
    if (INT8) {
        for (int c = 2 * sub; c < kept; c += 2 * (int)a.warpsPerRow)
            exact_pair_int8(a, reinterpret_cast<const float2 *>(xs), sExpert[slot][c], sExpert[slot][c + 1], &sLogit[slot][c], lane);
    } else if (a.warpsPerRow > 2) {
        for (int c = 2 * sub; c < kept; c += 2 * (int)a.warpsPerRow)
            exact_bf16<2>(a, reinterpret_cast<const uint4 *>(xs), &sExpert[slot][c], &sLogit[slot][c], lane);
    } else {
        int c = 4 * sub;
        if (a.warpsPerRow == 1)
            for (; kept - c > 4; c += 8) exact_bf16<8>(a, reinterpret_cast<const uint4 *>(xs), &sExpert[slot][c], &sLogit[slot][c], lane);
        for (; c < kept; c += 4 * (int)a.warpsPerRow) {
            if (kept - c > 2) exact_bf16<4>(a, reinterpret_cast<const uint4 *>(xs), &sExpert[slot][c], &sLogit[slot][c], lane);
            else exact_bf16<2>(a, reinterpret_cast<const uint4 *>(xs), &sExpert[slot][c], &sLogit[slot][c], lane);
        }
    }
    if (a.warpsPerRow > 1) __syncthreads();
    else __syncwarp();
    if (!live || sub != 0) return;
    if (a.bias)
        for (int c = lane; c < kept; c += 32) sLogit[slot][c] += a.bias[sExpert[slot][c]];
    __syncwarp();
    // rank by counting (higher score, then lower id = earlier in the list); -inf and NaN are never taken
    for (int c = lane; c < kept; c += 32) {
        const float v = sLogit[slot][c];
        int rank = 0;
        for (int o = 0; o < kept; ++o) {
            const float w = sLogit[slot][o];
            rank += (w > v || (w == v && o < c)) ? 1 : 0;
        }
        if (v > -INFINITY && rank < K) {
            sTopScore[slot][rank] = v;
            sTopId[slot][rank] = sExpert[slot][c];
        }
    }
    __syncwarp();
    const float score = lane < K ? sTopScore[slot][lane] : -INFINITY;
    const float ex = lane < K ? expf(score - sTopScore[slot][0]) : 0.0f;
    float sum = 0.0f;
    for (int r = 0; r < K; ++r) sum += __shfl_sync(0xFFFFFFFFu, ex, r);
    if (lane < K) {
        const uint32_t id = sTopId[slot][lane];
        float w = ex / sum;
        if (a.gain) w = w * bf2f(a.gain[id]);
        a.ids[(size_t)t * K + lane] = id;
        a.weights[(size_t)t * K + lane] = f2bf(w);
    }
}

// ---- INT8 logits of every expert (decode and verify rows, or when the logits are asked for) --------

// One warp per expert and NT rows, the codes in lane order: a lane's codes of eight groups are one 128-bit load.
// What does not depend on the launch before (codes, scales | biases, per-input scale: the first 3072 inputs' at once) is
// requested in front of the wait for it, the rows all together behind it, so that a warp waits for memory once: one row of
// 2816 inputs and 128 experts 12.7 -> 7.2 us.  Bound by that latency, the 88 dependent multiply-adds and the ranking by the
// last CTA.
// (kLaneRuns: runs of eight groups whose operands a warp holds at a time.)
template <int NT, int kLaneRuns>
__global__ void __launch_bounds__(128)
k_router_logits_int8(const uint4 *Q, const uint32_t *aux, const uint16_t *effScale, const float *bias, const uint16_t *x,
                     uint32_t xStride, int T, int E, int D, float *logits, RouterTail tail) {
    __shared__ __align__(16) uint4 sAux[4][kLaneRuns * 2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = min((int)blockIdx.x * 4 + warp, E - 1), t0 = blockIdx.y * NT;  // (a warp past the experts repeats the last)
    const int groups = D >> 6, runs = (groups + 7) >> 3;
    const uint4 *q = Q + (size_t)e * runs * 32 + lane;
    const uint4 *sb = reinterpret_cast<const uint4 *>(aux + (size_t)e * runs * 8);
    const uint32_t *eff = reinterpret_cast<const uint32_t *>(effScale) + lane;
    uint4 qv[kLaneRuns];
    uint32_t ev[8 * kLaneRuns];
    auto fetch = [&](int r0) {
        if (lane < 2 * kLaneRuns) sAux[warp][lane] = 2 * r0 + lane < 2 * runs ? __ldg(sb + 2 * r0 + lane) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int r = 0; r < kLaneRuns; ++r) qv[r] = r0 + r < runs ? __ldg(q + (r0 + r) * 32) : make_uint4(0, 0, 0, 0);
        if (effScale) {
#pragma unroll
            for (int i = 0; i < 8 * kLaneRuns; ++i) ev[i] = __ldg(eff + min(8 * r0 + i, groups - 1) * 32);
        }
    };
    fetch(0);
    pdl_enter();
    const uint32_t *xr[NT];
    float acc[NT];
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        xr[k] = reinterpret_cast<const uint32_t *>(x + (size_t)min(t0 + k, T - 1) * xStride) + lane;
        acc[k] = 0.0f;
    }
    for (int r0 = 0; r0 < runs; r0 += kLaneRuns) {
        if (r0) {
            __syncwarp();
            fetch(r0);
        }
        uint32_t xv[NT][8 * kLaneRuns];
#pragma unroll
        for (int i = 0; i < 8 * kLaneRuns; ++i)
#pragma unroll
            for (int k = 0; k < NT; ++k) xv[k][i] = xr[k][min(8 * r0 + i, groups - 1) * 32];
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kLaneRuns; ++r) {
            const uint4 sa[2] = {sAux[warp][2 * r], sAux[warp][2 * r + 1]};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (8 * (r0 + r) + i < groups) {
#pragma unroll
                    for (int k = 0; k < NT; ++k) {
                        const uint32_t w = xv[k][8 * r + i];
                        float x0 = __uint_as_float(w << 16), x1 = __uint_as_float(w & 0xFFFF0000u);
                        if (effScale) {
                            x0 = x0 * __uint_as_float(ev[8 * r + i] << 16);
                            x1 = x1 * __uint_as_float(ev[8 * r + i] & 0xFFFF0000u);
                        }
                        acc[k] = int8_group(qv[r], sa, i, x0, x1, x0 + x1, acc[k]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        float v = acc[k];
#pragma unroll
        for (int offset = 16; offset >= 1; offset >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, offset);
        if (lane == 0 && t0 + k < T) logits[(size_t)(t0 + k) * E + e] = bias ? v + bias[e] : v;
    }
    if (tail.ids)
        for (int k = 0; k < NT && t0 + k < T; ++k)
            topk_by_last_cta(logits + (size_t)(t0 + k) * E, E, tail.K, tail.gain, tail.ids + (t0 + k) * tail.K,
                             tail.weights + (t0 + k) * tail.K, tail.counts + t0 + k, gridDim.x);
}

// ---- a short chunk: every logit in its order, and the top K, in one launch --------------------------

// CTA (expert tile, token tile): a warp per expert, its row in registers (requested in front of the wait for the launch
// before), kTileTokens rows in shared memory: bf16, or (WIDE) fp32 times the per-input scale.  The last CTA of a token
// tile ranks its rows, a warp each.  A pair of expert and row is about 280 warp instructions at 2816 inputs, which bounds
// it; the approximate logits and the selection behind them are two launches and cost less for more pairs: see
// router_tile_pays.
// Chunks of 256 inputs in registers: eleven leave 100 registers, twelve 114.  bf16, 128 experts, eleven / twelve: 2816 inputs,
// 64 rows 9.0 / 8.8, 77 11.2 / 11.3, 128 11.25 / 11.6; 3072 inputs, 64 rows 9.3 / 8.8, 128 11.8 / 11.7; 5632 inputs, 77 rows 16.5 / 17.2.
constexpr int kTileTokens = 8, kTileExperts = 8, kTileChunks = 11;
constexpr uint32_t kTileMaxRows = 160;  // (measured up to here)
static_assert((kTileMaxRows + kTileTokens - 1) / kTileTokens <= (uint32_t)kRouterCounts, "a counter for every tile of rows");
struct TileArgs {
    const uint16_t *W;           // bf16 router [E][D], or
    const uint4 *Q;              // INT8 router in lane order
    const uint32_t *qAux;
    const uint16_t *scale, *gain;
    const float *bias;
    const uint16_t *x;
    uint32_t xStride;
    int T, E, D, K;
    float *logits;               // [T][E]
    uint32_t *counts;            // CTAs of a token tile that are done, zero between launches
    uint32_t *ids;
    uint16_t *weights;
};
template <bool INT8, bool WIDE>
__global__ void __launch_bounds__(kTileExperts * 32)
k_router_tile(const TileArgs a) {
    extern __shared__ __align__(16) uint8_t selectSmem[];
    __shared__ uint32_t sLast;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = min((int)blockIdx.x * kTileExperts + warp, a.E - 1);  // (a warp past the experts repeats the last)
    const int t0 = (int)blockIdx.y * kTileTokens, tokens = min(kTileTokens, a.T - t0);
    constexpr int kRuns = 6;  // INT8: of eight groups
    const int groups = a.D >> 6, runs = (groups + 7) >> 3;
    uint4 wv[INT8 ? kRuns : kTileChunks], sb[INT8 ? 2 * kRuns : 1];
    auto fetch = [&](int first) {  // INT8: run, else chunk of 256 inputs
        if constexpr (INT8) {
#pragma unroll
            for (int r = 0; r < kRuns; ++r) {
                const bool there = first + r < runs;
                wv[r] = there ? __ldg(a.Q + ((size_t)e * runs + first + r) * 32 + lane) : make_uint4(0, 0, 0, 0);
                const uint4 *aux = reinterpret_cast<const uint4 *>(a.qAux + (size_t)e * runs * 8) + 2 * (first + r);
                sb[2 * r] = there ? __ldg(aux) : make_uint4(0, 0, 0, 0);
                sb[2 * r + 1] = there ? __ldg(aux + 1) : make_uint4(0, 0, 0, 0);
            }
        } else {
#pragma unroll
            for (int i = 0; i < kTileChunks; ++i) {
                const int base = (first + i) * 256 + 8 * lane;
                wv[i] = base < a.D ? __ldg(reinterpret_cast<const uint4 *>(a.W + (size_t)e * a.D + base)) : make_uint4(0, 0, 0, 0);
            }
        }
    };
    fetch(0);
    pdl_enter();
    const uint32_t rowBytes = (uint32_t)a.D * (WIDE ? 4u : 2u);
    {
        const int chunks = a.D >> 3;
        // a warp a row (past the rows: the last again, so that every row of the tile is defined)
        const uint4 *src = reinterpret_cast<const uint4 *>(a.x + (size_t)(t0 + min(warp, tokens - 1)) * a.xStride);
        uint8_t *dst = selectSmem + (uint32_t)warp * rowBytes;
#pragma unroll 4
        for (int c = lane; c < chunks; c += 32) {
            const uint4 v = src[c];
            if (!WIDE) {
                reinterpret_cast<uint4 *>(dst)[c] = v;
                continue;
            }
            uint4 sv = make_uint4(0, 0, 0, 0);
            if (a.scale) sv = __ldg(reinterpret_cast<const uint4 *>(a.scale) + c);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w}, f[4] = {sv.x, sv.y, sv.z, sv.w};
            float xe[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                xe[2 * k] = __uint_as_float(w[k] << 16);
                xe[2 * k + 1] = __uint_as_float(w[k] & 0xFFFF0000u);
                if (a.scale) {
                    xe[2 * k] = xe[2 * k] * __uint_as_float(f[k] << 16);
                    xe[2 * k + 1] = xe[2 * k + 1] * __uint_as_float(f[k] & 0xFFFF0000u);
                }
            }
            reinterpret_cast<float4 *>(dst)[2 * c] = make_float4(xe[0], xe[1], xe[2], xe[3]);
            reinterpret_cast<float4 *>(dst)[2 * c + 1] = make_float4(xe[4], xe[5], xe[6], xe[7]);
        }
    }
    __syncthreads();
    static_assert(kTileTokens == kTileExperts, "a warp stages a row");
    float acc[kTileTokens];
#pragma unroll
    for (int t = 0; t < kTileTokens; ++t) acc[t] = 0.0f;
    if constexpr (INT8) {
        for (int first = 0; first < runs; first += kRuns) {
            if (first) fetch(first);
#pragma unroll
            for (int r = 0; r < kRuns; ++r) {
                const uint4 aux[2] = {sb[2 * r], sb[2 * r + 1]};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int g = 8 * (first + r) + i;
                    if (g >= groups) break;
#pragma unroll
                    for (int t = 0; t < kTileTokens; ++t) {
                        const float2 x = *reinterpret_cast<const float2 *>(selectSmem + (uint32_t)t * rowBytes + (uint32_t)(g * 32 + lane) * 8u);
                        acc[t] = int8_group(wv[r], aux, i, x.x, x.y, x.x + x.y, acc[t]);
                    }
                }
            }
        }
    } else {
        const int chunks = (a.D + 255) >> 8;
        for (int first = 0; first < chunks; first += kTileChunks) {
            if (first) fetch(first);
#pragma unroll
            for (int i = 0; i < kTileChunks; ++i) {
                const int base = (first + i) * 256 + 8 * lane;
                if (base >= a.D) break;
                const uint32_t ww[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
                float w[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    w[2 * k] = __uint_as_float(ww[k] << 16);
                    w[2 * k + 1] = __uint_as_float(ww[k] & 0xFFFF0000u);
                }
#pragma unroll
                for (int t = 0; t < kTileTokens; ++t) {
                    const uint8_t *row = selectSmem + (uint32_t)t * rowBytes;
                    float x[8];
                    if (WIDE) {
                        const float4 lo = *reinterpret_cast<const float4 *>(row + (uint32_t)base * 4u), hi = *reinterpret_cast<const float4 *>(row + (uint32_t)base * 4u + 16u);
                        x[0] = lo.x, x[1] = lo.y, x[2] = lo.z, x[3] = lo.w, x[4] = hi.x, x[5] = hi.y, x[6] = hi.z, x[7] = hi.w;
                    } else {
                        const uint4 v = *reinterpret_cast<const uint4 *>(row + (uint32_t)base * 2u);
                        const uint32_t xx[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            x[2 * k] = __uint_as_float(xx[k] << 16);
                            x[2 * k + 1] = __uint_as_float(xx[k] & 0xFFFF0000u);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) acc[t] = fmaf(w[k], x[k], acc[t]);
                }
            }
        }
    }
    int which;
    const float v = butterfly<kTileTokens>(acc, lane, which);
    if ((lane & (32 / kTileTokens - 1)) == 0 && which < tokens) a.logits[(size_t)(t0 + which) * a.E + e] = a.bias ? v + a.bias[e] : v;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        sLast = atomicInc(a.counts + blockIdx.y, gridDim.x - 1u) == gridDim.x - 1u ? 1u : 0u;
    }
    __syncthreads();
    if (sLast && warp < tokens) {
        __threadfence();
        const size_t t = (size_t)(t0 + warp);
        warp_topk(a.logits + t * a.E, a.E, a.K, a.gain, a.ids + t * a.K, a.weights + t * a.K);
    }
}

// ---- at load: folded bf16 weights and the bound's coefficients --------------------------------------

// One CTA per expert.  folded = bf16(w * scale) (null: the router's own bf16 rows are multiplied).  Norms in
// double: the squares of any product of two bf16 values are normal numbers there.
__global__ void __launch_bounds__(256)
k_router_prepare(const uint16_t *W, const uint8_t *Q, const uint16_t *qScale, const uint16_t *qBias, const uint16_t *scale,
                 int D, uint16_t *folded, RouterBound *bounds) {
    __shared__ double sums[4][8];
    const int e = blockIdx.x;
    // |w scale|^2, |the terms the fixed order adds|^2, sum |w|, and the largest factor of an input in either order
    double sq = 0.0, sqTerms = 0.0, sumW = 0.0, factor = Q ? 255.0 : 1.0;
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
        const double f = scale ? (double)bf2f(scale[i]) : 1.0;
        double w, terms, plain;
        if (Q) {
            const double q = (double)Q[(size_t)e * D + i], s = (double)bf2f(qScale[(size_t)e * (D / 64) + i / 64]),
                         b = (double)bf2f(qBias[(size_t)e * (D / 64) + i / 64]);
            w = fma(q, s, b) * f;
            plain = q * fabs(s) + fabs(b);
            terms = plain * fabs(f);
            factor = fmax(factor, 255.0 * fabs(f));
        } else {
            plain = fabs((double)bf2f(W[(size_t)e * D + i]));
            w = (double)bf2f(W[(size_t)e * D + i]) * f;
            terms = fabs(w);
            factor = fmax(factor, fabs(f));
        }
        if (folded) folded[(size_t)e * D + i] = f2bf((float)w);
        sq = fma(w, w, sq);
        sqTerms = fma(terms, terms, sqTerms);
        sumW += plain + fabs(w);
    }
#pragma unroll
    for (int offset = 16; offset >= 1; offset >>= 1) {
        sq += __shfl_xor_sync(0xFFFFFFFFu, sq, offset);
        sqTerms += __shfl_xor_sync(0xFFFFFFFFu, sqTerms, offset);
        sumW += __shfl_xor_sync(0xFFFFFFFFu, sumW, offset);
        factor = fmax(factor, __shfl_xor_sync(0xFFFFFFFFu, factor, offset));
    }
    if ((threadIdx.x & 31) == 0) {
        sums[0][threadIdx.x >> 5] = sq;
        sums[1][threadIdx.x >> 5] = sqTerms;
        sums[2][threadIdx.x >> 5] = sumW;
        sums[3][threadIdx.x >> 5] = factor;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) {
            sq += sums[0][i];
            sqTerms += sums[1][i];
            sumW += sums[2][i];
            factor = fmax(factor, sums[3][i]);
        }
        const double u = 0x1p-23, tiny = 0x1p-126;
        const double chain = (double)(Q ? 4 * (D / 64) + 16 : 8 * ((D + 255) / 256) + 16);
        RouterBound b;
        // (an input of a flushed weight: tiny |x| summed over the row, at most tiny sqrt(D) |x| in the 2-norm)
        b.perNorm = (float)(1.02 * (sqrt(sq) * ((D + 16) * u + (folded ? 2.1e-3 : 0.0)) + sqrt(sqTerms) * chain * u) +
                            2.0 * tiny * sqrt((double)D));
        b.floor = (float)(tiny * (4.0 * D + 2.0 * sumW));  // products and sums; inputs and scaled inputs, times their weights
        b.limit = (float)(0x1p120 / fmax(factor, sqrt(sqTerms)));
        bounds[e] = b;
    }
}

// INT8 router rows in lane order: lanes[e][r][l] = the codes 64 g + 2 l, + 1 of the eight groups g = 8 r..,
// aux[e][g] = scale | bias << 16; groups past the row are zero.
__global__ void __launch_bounds__(256)
k_router_int8_lanes(const uint8_t *Q, const uint16_t *qScale, const uint16_t *qBias, int D, uint16_t *lanes, uint32_t *aux) {
    const int e = blockIdx.x, groups = D >> 6, padded = ((groups + 7) >> 3) << 3;
    for (int i = threadIdx.x; i < padded * 32; i += blockDim.x) {
        const int r = i >> 8, l = (i >> 3) & 31, g = 8 * r + (i & 7);
        lanes[(size_t)e * padded * 32 + i] =
            g < groups ? *reinterpret_cast<const uint16_t *>(Q + (size_t)e * D + g * 64 + 2 * l) : (uint16_t)0;
    }
    for (int g = threadIdx.x; g < padded; g += blockDim.x)
        aux[(size_t)e * padded + g] =
            g < groups ? (uint32_t)qScale[(size_t)e * groups + g] | ((uint32_t)qBias[(size_t)e * groups + g] << 16) : 0u;
}

bool router_map(CUtensorMap *map, const uint16_t *base, uint64_t rows, uint64_t d, uint64_t stride, uint32_t boxRows,
                const char **error) {
    const cuuint64_t dims[2] = {d, rows}, strides[1] = {stride * 2};
    const cuuint32_t box[2] = {kApproxK, boxRows};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "router", error);
}

}  // namespace

// Rows of partial logits a context of `maxTokens` can need: splits are used only while the token
// tiles leave SMs idle.
size_t router_parts_rows(size_t maxTokens, int smCount) {
    return std::min<size_t>(maxTokens * kMaxSplits, std::max<size_t>(maxTokens, (size_t)smCount * 128));
}

bool router_prepare(FFContext *ctx, LayerStore &L, const char **error) {
    const int E = (int)L.routerExperts, D = (int)ctx->cfg.d;
    if (L.routerQ || L.routerScale)
        FF_CUDA_OK(cudaMalloc(reinterpret_cast<void **>(&L.routerFolded), (size_t)E * D * 2), error);
    FF_CUDA_OK(cudaMalloc(reinterpret_cast<void **>(&L.routerBounds), (size_t)E * sizeof(RouterBound)), error);
    if (L.routerQ) {
        const size_t padded = ((size_t)(D / 64) + 7) / 8 * 8;
        FF_CUDA_OK(cudaMalloc(reinterpret_cast<void **>(&L.routerLanes), (size_t)E * padded * 64), error);
        FF_CUDA_OK(cudaMalloc(reinterpret_cast<void **>(&L.routerAux), (size_t)E * padded * 4), error);
        k_router_int8_lanes<<<E, 256>>>(L.routerQ, L.routerQScale, L.routerQBias, D, L.routerLanes, L.routerAux);
    }
    k_router_prepare<<<E, 256>>>(L.routerW, L.routerQ, L.routerQScale, L.routerQBias, L.routerScale, D, L.routerFolded,
                                  L.routerBounds);
    FF_CUDA_OK(cudaGetLastError(), error);
    FF_CUDA_OK(cudaStreamSynchronize(nullptr), error);
    return true;
}

static bool launch_router_tile(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens, uint32_t *ids,
                               uint16_t *weights, cudaStream_t stream, const char **error) {
    TileArgs a{};
    a.W = L.routerW;
    a.Q = reinterpret_cast<const uint4 *>(L.routerLanes);
    a.qAux = L.routerAux;
    a.scale = L.routerScale;
    a.gain = L.gain;
    a.bias = L.logitBias;
    a.x = x;
    a.xStride = xStride;
    a.T = (int)tokens;
    a.E = (int)L.routerExperts;
    a.D = (int)ctx->cfg.d;
    a.K = (int)ctx->cfg.topK;
    a.logits = ctx->routerParts;
    a.counts = ctx->routerCounts;
    a.ids = ids;
    a.weights = weights;
    const int form = L.routerQ ? 2 : L.routerScale ? 1 : 0;
    auto kernel = form == 2 ? k_router_tile<true, true> : form == 1 ? k_router_tile<false, true> : k_router_tile<false, false>;
    const size_t smem = (size_t)kTileTokens * a.D * (form ? 4 : 2);
    static KernelSmemMemo memo[3];
    if (!memo[form].prepare(kernel, ctx->device, smem, kTileExperts * 32, nullptr, error)) return false;
    LaunchScope scope(ctx, stream, "router_tile");
    FF_CUDA_OK(launch_pdl(kernel, dim3((a.E + kTileExperts - 1) / kTileExperts, (tokens + kTileTokens - 1) / kTileTokens), kTileExperts * 32, smem,
                          stream, a),
               error);
    return true;
}

// Whether k_router_tile takes less time than the two launches: these hardly grow with the rows, it by its CTAs an SM and
// their inputs.  us in a graph on 148 SMs, this / those:
//   bf16, 2816 inputs, CTAs an SM 1 (17 rows, 128 experts) 9.3 / 13.9, 2 (77 rows) 11.3 / 16.4, 3 (160 rows) 15.1 / 18.0, 4
//     (128 rows, 256 experts) 19.0 / 20.3, 5 (160 rows) 24.5 / 20.4; 4096 inputs 3 18.3 / 18.9, 4 23.4 / 21.5; 6144 inputs 2 17.4 /
//     19.9, 3 24.8 / 22.1;
//   INT8, 2816 inputs, 2 15.1 / 22.6, 3 21.5 / 23.2, 4 26.8 / 25.0; one CTA's fp32 rows an SM, so that the second runs behind the
//     first: 4096 inputs 1 14.1 / 21.7, 2 24.7 / 25.6 (codes from memory 38.9 / 35.8);
//   bf16 with a per-input scale, whose rows are widened for every expert tile: 1024 inputs 2 11.0 / 14.6, 3 16.8 / 14.8; 2816
//     inputs 1 13.7 / 16.4 (fewer than 64 experts, where the two launches are shorter, 12.4 / 11.9), 2 20.3 / 19.3, 3 35.5 / 19.5;
//     4096 inputs 1 17.6 / 17.1.
static bool router_tile_pays(const FFContext *ctx, const LayerStore &L, uint32_t tokens) {
    const uint32_t D = ctx->cfg.d, E = L.routerExperts, sms = (uint32_t)ctx->smCount;
    const size_t smem = (size_t)kTileTokens * D * (L.routerQ || L.routerScale ? 4 : 2), smBytes = 220 * 1024;
    if (tokens > kTileMaxRows || smem > 200 * 1024) return false;
    const uint32_t ctas = (E + kTileExperts - 1) / kTileExperts * ((tokens + kTileTokens - 1) / kTileTokens);
    const uint32_t perSm = (ctas + sms - 1) / sms;
    if (L.routerQ) return perSm * D <= 9216u && (perSm == 1u || 2 * smem <= smBytes);
    if (L.routerScale) return perSm * D <= (E < 64u ? 2048u : 3000u);
    return perSm * D <= 12288u;
}

bool launch_router_select(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                          uint32_t *ids, uint16_t *weights, cudaStream_t stream, const char **error) {
    const uint32_t E = L.routerExperts, D = ctx->cfg.d, K = ctx->cfg.topK;
    if (router_tile_pays(ctx, L, tokens))
        return launch_router_tile(ctx, L, x, xStride, tokens, ids, weights, stream, error);
    // Token tile: as large as the rows allow (the router's 720 KB are read once per tile and split);
    // the contraction is split while tiles x splits stay within one CTA per SM.
    const uint32_t tileTokens = std::min(128u, (tokens + 31u) & ~31u);
    const uint32_t tiles = (tokens + tileTokens - 1) / tileTokens, expertTiles = (E + kExpertTile - 1) / kExpertTile;
    const uint32_t steps = D / kApproxK;
    uint32_t splits = std::max(1u, std::min({kMaxSplits, (uint32_t)ctx->smCount / std::max(1u, tiles * expertTiles), steps}));
    splits = (steps + (steps + splits - 1) / splits - 1) / ((steps + splits - 1) / splits);  // no empty split
    CUtensorMap mapW, mapX;
    if (!router_map(&mapW, L.routerFolded ? L.routerFolded : L.routerW, E, D, D, kExpertTile, error) ||
        !router_map(&mapX, x, tokens, D, xStride, tileTokens, error))
        return false;
    const size_t smem = 1024 + (size_t)kApproxStages * (kExpertBytes + tileTokens * kApproxK * 2);
    static KernelSmemMemo memo, memoSelect[2];
    if (!memo.prepare(k_router_approx, ctx->device, 1024 + (size_t)kApproxStages * 2 * kExpertBytes, kApproxThreads, nullptr, error))
        return false;
    {
        LaunchScope scope(ctx, stream, "router_approx");
        FF_CUDA_OK(launch_pdl(k_router_approx, dim3(tiles, expertTiles, splits), kApproxThreads, smem, stream,
                              mapW, mapX, tileTokens, tokens, E, steps,
                                                                                         splits, ctx->routerParts, ctx->errorFlag),
                   error);
    }
    SelectArgs a{};
    a.W = L.routerW;
    a.Q = reinterpret_cast<const uint4 *>(L.routerLanes);
    a.qAux = L.routerAux;
    a.scale = L.routerScale;
    a.gain = L.gain;
    a.bias = L.logitBias;
    a.bounds = L.routerBounds;
    a.x = x;
    a.xStride = xStride;
    a.splits = splits;
    a.T = (int)tokens;
    a.E = (int)E;
    a.D = (int)D;
    a.K = (int)K;
    a.parts = ctx->routerParts;
    a.ids = ids;
    a.weights = weights;
    // As many warps a row as keep the rows in one wave (the launch bounds give 24 warps an SM, 32 for INT8), INT8 two
    // at least.  bf16, us of this kernel with 8 / 4 / 2 / 1 warps: 77 rows 14.8 / 18.9 / 20.9 / 21.0, 512 rows 23.0 / 18.9 /
    // 19.0 / 23.0, 1500 rows 39.4 / 31.1 / 23.1 / 25.1, 2048 rows 49.5 / 39.3 / 33.2 / 27.1; INT8 with 8 / 4 / 2: 512 rows
    // 25.0 / 26.0 / 35.4, 1024 rows 37.3 / 33.2 / 39.4, 2048 rows 57.9 / 51.8 / 49.7.
    const uint32_t resident = (uint32_t)ctx->smCount * (L.routerQ ? 32u : 24u);
    a.warpsPerRow = kSelectWarps;
    while (a.warpsPerRow > (L.routerQ ? 2u : 1u) && (uint64_t)tokens * a.warpsPerRow > resident) a.warpsPerRow /= 2;
    const uint32_t perCta = kSelectWarps / a.warpsPerRow;
    const size_t rowBytes = (size_t)D * (L.routerQ ? 4 : 2);
    auto kernel = L.routerQ ? k_router_select<true> : k_router_select<false>;
    if (!memoSelect[L.routerQ ? 1 : 0].prepare(kernel, ctx->device, kSelectWarps * (size_t)D * 2, kSelectWarps * 32, nullptr, error))
        return false;
    {
        LaunchScope scope(ctx, stream, "router_select");
        FF_CUDA_OK(launch_pdl(kernel, (tokens + perCta - 1) / perCta, kSelectWarps * 32, perCta * rowBytes, stream,
                              a),
                   error);
    }
    return true;
}

bool launch_router_logits_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                               float *logits, const RouterTail &tail, cudaStream_t stream, const char **error) {
    const int E = (int)L.routerExperts, D = (int)ctx->cfg.d;
    if (xStride % 2 || ((uintptr_t)x & 3)) return fail(error, "input rows must be 4-byte aligned");
    const uint4 *lanes = reinterpret_cast<const uint4 *>(L.routerLanes);
    {
        LaunchScope scope(ctx, stream, "router_logits_int8");
        // A turn of a warp's loop loads all its places, so what it holds follows the row's runs of eight groups.
        // A block: a warp per expert and row, for the latency, with up to six runs in flight (three CTAs an SM): four where that
        // makes the row's turns even (1088 to 2048 and 3136 to 4096 inputs), two where the row has no more or where the CTAs would
        // be more than six an SM.  us in a graph, six / four / two: 512 inputs, 128 experts, one row 6.0 / 5.6 / 5.3, 16 rows 9.6 / 6.9 /
        // 6.4; 2816 inputs, 128 experts, one row 5.8 / 6.6 / 6.7, 16 rows 9.5 / 10.0 / 11.5; 4096 inputs, 128 experts, one row 7.8 / 6.8 /
        // 7.7, 16 rows 15.1 / 10.6 / 13.6, 256 experts, 13 rows 20.2 / 16.0 / 15.5, 16 rows 24.5 / 17.7 / 17.9.
        // More rows: two rows and few registers a warp, and two runs where their number is even; else three where it divides
        // or the CTAs are few, else one.  three / two / one, 128 experts: 1536 inputs, 17 rows 6.6 / 7.3 / -, 160 rows 18.9 / 21.5 / -;
        // 2304 inputs, 160 rows - / 29.5 / 27.5; 2816 inputs, 160 rows 31.1 / 31.4 / 32.0; 4096 inputs, 160 rows 43.5 / 41.4 / 41.9.
        const dim3 grid((E + 3) / 4, tokens <= (uint32_t)kMaxGemvRows ? tokens : (tokens + 1) / 2);
        const uint32_t ctas = grid.x * grid.y, sms = (uint32_t)ctx->smCount;
        const uint32_t runs = ((uint32_t)D / 64u + 7u) / 8u, turns = (runs + 5u) / 6u, inTurn = (runs + turns - 1u) / turns;
        auto kernel = k_router_logits_int8<1, 6>;
        if (tokens <= (uint32_t)kMaxGemvRows) {
            if (inTurn <= 2u || ctas > 6u * sms) kernel = k_router_logits_int8<1, 2>;
            else if (inTurn <= 4u) kernel = k_router_logits_int8<1, 4>;
        } else if (runs % 2u == 0u) {
            kernel = k_router_logits_int8<2, 2>;
        } else {
            kernel = runs % 3u == 0u || (runs > 3u && ctas <= 3u * sms) ? k_router_logits_int8<2, 3> : k_router_logits_int8<2, 1>;
        }
        FF_CUDA_OK(launch_pdl(kernel, grid, 128, 0, stream, lanes, L.routerAux, L.routerScale, L.logitBias, x, xStride, (int)tokens, E, D,
                              logits, tail),
                   error);
    }
    return true;
}

}  // namespace ff
