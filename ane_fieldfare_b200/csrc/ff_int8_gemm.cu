// INT8 affine shared FFN for more rows than a decode/verify block, on the 5th-generation tensor cores.
//
// A weight is w = q s + b (q 0..255; s, b bf16, one pair per row and 64 inputs).  Rounding w to bf16
// would lose most of q's bits, and a tensor-core sum over the whole contraction is less exact than the
// fp32 sums the operator promises (its 376 truncated additions moved 12 % of the outputs to the
// neighbouring bf16 value), so the contraction stays in groups: q is exact in bf16 and is multiplied
// as it is, a step of 64 inputs is one accumulation of four MMAs in tensor memory, and sixteen warps
// fetch every step's sums and add them up in registers as acc = fma(s, sum, acc), rounded to nearest.
// The bias part, sum_g b_g X_g with X_g the sum of the token over group g, is a few more steps of the
// same kind: A = the row's biases, B = X_g as three bf16 pieces (their sum is X_g to fp32's 24 bits),
// scale 1.
//
// Two CTAs of a cluster work as one tensor-core unit (cta_group::2, M = 256: either CTA 128 weight
// rows, half of the token tile).  Per CTA: warp 0 TMA producer, warp 1 MMA issuer (leader only),
// warps 2-9 turn codes into bf16 pairs in tensor memory (two groups of four warps, alternate steps),
// warps 10-25 drain, four for every 32 tokens of the tile: a thread owns one weight row and 32 tokens.  Tensor memory: three accumulators of
// 128 columns, four operand stages of 32.
//
// What bounds it: the draining warps.  A step is 2700 warp instructions of a CTA (128 tokens; 512 of them the
// multiply-adds), and each warp goes through a step's wait, loads and arrival one after another, 800 to 900 cycles
// for the tensor core's 256.  2000 rows of 2816 x 2112: gate/up and down 153 us; with eight draining warps of 64
// tokens, which did not fit their registers, 191 us.  Small tiles leave draining warps without tokens: with these waiting and
// arriving at every step, 17 rows 39.9 us, 300 rows 44.7, and 36.1 and 42.2 without them.  Measured and not kept: loads of 32 columns (181 us: nothing
// overlaps them), eight warps with 152 registers by setmaxnreg and a load always in flight (199 us), packed
// multiply-adds (the compiler moves as many registers as they save), one dequantizing group (171 us).
//
// Error against 64 bits: the tensor core truncates where it aligns a group's products, so a token with one
// value of 2^16 times the rest whose weight q s + b is zero comes out 3.4e-3 off (fp32 FMAs 2.1e-3, the
// block kernel 2.2e-3), at 2^12 1.76e-3 against 1.67e-3 without it (the outputs' bf16 rounding).
//
// Reference kernels this file stands in for (paths inside the reference project):
//   Sources/ANEFieldfareHotpath/Metal/Quant/dequant_int8.metal:41-138,
//   Sources/ANEFieldfareHotpath/Kernels/MoE/SharedExpertInt8.swift:7-29.
#include <algorithm>

#include "ff_gemv_device.cuh"
#include "ff_internal.cuh"
#include "ff_tc_device.cuh"

namespace ff {
namespace {

constexpr int kStages = 8;          // token and packed-code tiles in flight
constexpr int kDequantGroups = 2;   // of four warps each
constexpr int kOperandStages = 4;   // weight operands in tensor memory, 32 columns each
constexpr int kAccs = 3;            // accumulators in tensor memory
constexpr uint32_t kMaxRows = 128;  // tokens of a tile = accumulator columns
constexpr uint32_t kStepK = 64;
constexpr uint32_t kTokBytes = kMaxRows / 2 * kStepK * 2;  // a CTA's half of a token tile
constexpr uint32_t kCodeBytes = 128 * kStepK;
constexpr uint32_t kOperandCol = kAccs * kMaxRows;
constexpr int kDrainSets = 4;       // of four warps each: a set drains kSetTokens of the tile's tokens
constexpr int kDrainThreads = 128 * kDrainSets;
constexpr uint32_t kSetTokens = kMaxRows / kDrainSets;
constexpr int kThreads = (2 + 4 * kDequantGroups) * 32 + kDrainThreads;
constexpr int kBarriers = 4 * kStages + 2 * kAccs + kDrainSets + 1;
constexpr uint32_t kPassTokens = 16;             // tokens of a set that become outputs at a time
constexpr uint32_t kXchgBytes = 128u * 8u * 4u;  // half of them, of every row, from gate to up or back
constexpr uint32_t kTilePitchGateUp = 64 * 2 + 16, kTilePitchDown = 128 * 2 + 16;
static_assert(kOperandCol + kOperandStages * 32 <= 512, "tensor memory layout");
static_assert(kSetTokens == 32, "tiles are multiples of a set's tokens");
static_assert(kStages % kOperandStages == 0 && kOperandStages % kDequantGroups == 0, "rings");

enum Mode : int { kGateUp = 0, kDown = 1 };

struct Int8GemmArgs {
    const uint16_t *scale[2], *bias[2];  // of matrix 0 / 1: [rows][K / 64]
    uint32_t K, N;                       // contraction, outputs per token
    uint32_t nTiles;                     // weight-row tiles: N/64 for gate/up, N/128 (rounded up) for down
    uint32_t tokens, tileRows, rowTiles;
    uint16_t *out;                       // [tokens][N]
    uint16_t *sums;                      // gate/up: group sums of the output rows, sums_pitch(N) apart
    uint32_t *errorFlag;
};

// Group sums of a row of K values: per 64 groups three runs of 64 bf16 pieces (high, middle, low).
__host__ __device__ inline uint32_t sum_blocks(uint32_t K) { return (K / kStepK + 63u) / 64u; }
__host__ __device__ inline uint32_t sums_pitch(uint32_t K) { return 192u * sum_blocks(K); }

__device__ __forceinline__ void store_group_sum(uint16_t *sumsRow, uint32_t group, float v) {
    uint16_t *dst = sumsRow + (group >> 6) * 192u + (group & 63u);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint16_t piece = f2bf(v);
        dst[64 * i] = piece;
        v -= bf2f(piece);
    }
}
__device__ __forceinline__ float sum8(const uint4 &v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) s += __uint_as_float(w[i] << 16) + __uint_as_float(w[i] & 0xFFFF0000u);
    return s;
}

// Group sums of x's rows; eight neighbouring threads hold one group.  Memory bound (x once).
__global__ void __launch_bounds__(256)
k_group_sums(const uint16_t *x, uint32_t xStride, uint32_t rows, uint32_t D, uint16_t *sums) {
    pdl_enter();
    const uint32_t chunks = D / 8, pitch = sums_pitch(D);
    const size_t total = (size_t)rows * chunks;
    // (total, the block and the grid stride are multiples of eight: a group's threads stay together)
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(i / chunks), c = (uint32_t)(i - (size_t)r * chunks);
        const uint32_t peers = 0xFFu << (threadIdx.x & 24);
        float s = sum8(*reinterpret_cast<const uint4 *>(x + (size_t)r * xStride + c * 8));
        s += __shfl_xor_sync(peers, s, 1);
        s += __shfl_xor_sync(peers, s, 2);
        s += __shfl_xor_sync(peers, s, 4);
        if ((c & 7u) == 0) store_group_sum(sums + (size_t)r * pitch, c >> 3, s);
    }
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
k_int8_gemm(const __grid_constant__ CUtensorMap mapTok, const __grid_constant__ CUtensorMap mapSums,
            const __grid_constant__ CUtensorMap mapW0, const __grid_constant__ CUtensorMap mapW1,
            const Int8GemmArgs args) {
    extern __shared__ uint8_t smemRaw[];
    __shared__ uint64_t barriers[kBarriers];
    __shared__ uint32_t tmemBaseSlot;
    __shared__ volatile uint32_t abortFlag;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rawBase = smem_u32(smemRaw), base = (rawBase + 1023u) & ~1023u;
    const uint32_t groupsK = args.K / kStepK, steps = groupsK + 3u * sum_blocks(args.K);
    // Draining sets whose tokens a tile has; the rest of the sixteen warps would only wait and arrive, which small tiles paid
    // for at every step.
    const uint32_t drainSets = args.tileRows / kSetTokens, drainThreads = 128u * drainSets;

    // carve-up: token tiles, code tiles, two buffers of scales, exchange rows (gate/up), output tiles
    auto tokAddr = [&](uint32_t s) { return base + s * kTokBytes; };
    auto codeAddr = [&](uint32_t s) { return base + kStages * kTokBytes + s * kCodeBytes; };
    uint8_t *rest = smemRaw + (base - rawBase) + kStages * (kTokBytes + kCodeBytes);
    uint16_t *scaleBuf = reinterpret_cast<uint16_t *>(rest);  // [2][128][groupsK]
    uint8_t *epilogue = rest + 2u * 128u * groupsK * 2u;

    const uint32_t barBase = smem_u32(barriers);
    auto barAt = [&](uint32_t i) { return barBase + 8u * i; };
    auto barStep = [&](uint32_t s) { return barAt(s); };
    auto barTokEmpty = [&](uint32_t s) { return barAt(kStages + s); };
    auto barCodeFull = [&](uint32_t s) { return barAt(2 * kStages + s); };
    auto barCodeEmpty = [&](uint32_t s) { return barAt(3 * kStages + s); };
    auto barAccFull = [&](uint32_t s) { return barAt(4 * kStages + s); };
    auto barAccEmpty = [&](uint32_t s) { return barAt(4 * kStages + kAccs + s); };
    auto barSet = [&](uint32_t h) { return barAt(4 * kStages + 2 * kAccs + h); };
    const uint32_t barScales = barAt(4 * kStages + 2 * kAccs + kDrainSets);

    // What the MMA issuer waits for lives in the leader: a step's barrier counts the arrivals of both CTAs'
    // dequantizers and the bytes of both CTAs' token copies.  Barriers that the MMAs' completion frees exist
    // in either CTA (one multicast commit).
    const uint32_t ctaRank = cluster_cta_rank();
    const bool leader = ctaRank == 0u;
    if (threadIdx.x == 0) {
        abortFlag = 0;
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(barStep(s), 9);  // (leader's is used) a group's four warps in either CTA, the expected bytes
            mbar_init(barTokEmpty(s), 1);
            mbar_init(barCodeFull(s), 1);
            mbar_init(barCodeEmpty(s), 4);
        }
        for (uint32_t s = 0; s < kAccs; ++s) {
            mbar_init(barAccFull(s), 1);
            mbar_init(barAccEmpty(s), 2 * drainThreads / 32);
        }
        for (uint32_t s = 0; s < kDrainSets; ++s) mbar_init(barSet(s), 128);
        mbar_init(barScales, drainThreads);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemBaseSlot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmemBase = __shfl_sync(0xFFFFFFFFu, tmemBaseSlot, 0);
    pdl_enter();

    // A pair's unit: one token tile, two neighbouring weight-row tiles (this CTA takes 2 np + rank).
    const uint32_t nPairs = (args.nTiles + 1u) >> 1, units = args.rowTiles * nPairs;
    const uint32_t firstUnit = blockIdx.x >> 1, unitStride = gridDim.x >> 1;
    auto ntOf = [&](uint32_t u) { return 2u * (u % nPairs) + ctaRank; };
    auto tokenOf = [&](uint32_t u) { return u / nPairs * args.tileRows; };
    auto rowsOf = [&](uint32_t u) { return min(args.tileRows, args.tokens - tokenOf(u)); };
    auto columnsOf = [&](uint32_t u) { return (rowsOf(u) + 31u) & ~31u; };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        {
            uint32_t st = 0, phase = 0;
            bool ok = true;
            const uint32_t leaderStep = map_to_cta(barStep(0), 0u);
            for (uint32_t u = firstUnit; u < units && ok; u += unitStride) {
                const uint32_t nt = ntOf(u);
                const int row0 = (int)(tokenOf(u) + ctaRank * (columnsOf(u) >> 1));
                for (uint32_t g = 0; g < steps; ++g) {
                    if (!mbar_wait_warp<true, Order::kLocal>(barCodeEmpty(st), phase ^ 1u, &abortFlag) ||
                        !mbar_wait_warp<true, Order::kPair>(barTokEmpty(st), phase ^ 1u, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    if (elect_one()) {
                        if (g < groupsK) {
                            mbar_expect_tx(barCodeFull(st), kCodeBytes);
#pragma unroll
                            for (int q = 0; q < 2; ++q)
                                tma_load_3d(codeAddr(st) + (uint32_t)q * (kCodeBytes / 2), MODE == kGateUp && q == 1 ? &mapW1 : &mapW0,
                                            (int)(g * kStepK), (int)(MODE == kGateUp ? nt * 64u : nt * 128u + (uint32_t)q * 64u), 0,
                                            barCodeFull(st));
                        } else {
                            mbar_arrive(barCodeFull(st));  // a bias step reads no codes
                        }
                        if (leader) mbar_expect_tx(barStep(st), 2u * kTokBytes);
                        const uint32_t bar = leaderStep + 8u * st;
                        if (g < groupsK) tma_load_2d_pair(tokAddr(st), &mapTok, (int)(g * kStepK), row0, bar);
                        else tma_load_2d_pair(tokAddr(st), &mapSums, (int)((g - groupsK) * kStepK), row0, bar);
                    }
                    if (++st == kStages) {
                        st = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (leader CTA only) ----------------
        // (the whole warp runs the loop and one elected lane issues: inside a `lane == 0` branch every
        // operand would go to the uniform registers by a loop over the active lanes)
        if (leader) {
            uint32_t st = 0, phase = 0, op = 0, accPhases = 0;  // a bit for each accumulator; a unit starts with the first
            bool ok = true;
            for (uint32_t u = firstUnit; u < units && ok; u += unitStride) {
                uint32_t acc = 0;
                const uint32_t idesc = umma_idesc_bf16_m256(columnsOf(u));
                for (uint32_t g = 0; g < steps; ++g) {
                    if (!mbar_wait_warp<false, Order::kPair>(barStep(st), phase, &abortFlag) ||
                        !mbar_wait_warp<false, Order::kPair>(barAccEmpty(acc), (accPhases >> acc & 1u) ^ 1u, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t descTok = umma_desc_sw128(tokAddr(st));
                    const uint32_t tmemW = tmemBase + kOperandCol + op * 32u, tmemD = tmemBase + acc * kMaxRows;
                    if (elect_one()) {
                        // (the wait was for both CTAs' operands; this look acquires the token halves, whose copies
                        // complete on this CTA's barrier)
                        (void)mbar_test_wait(barStep(st), phase);
#pragma unroll
                        for (uint32_t kk = 0; kk < kStepK / 16; ++kk)
                            tc_mma_bf16_a_tmem(tmemD, tmemW + 8u * kk, descTok + 2u * kk, idesc, kk ? 1u : 0u);
                        tc_commit_pair(barTokEmpty(st));  // the token stage and the operand stage are free
                        tc_commit_pair(barAccFull(acc));
                    }
                    if (++st == kStages) {
                        st = 0;
                        phase ^= 1u;
                    }
                    op = (op + 1u) % kOperandStages;
                    accPhases ^= 1u << acc;
                    if (++acc == kAccs) acc = 0;
                }
            }
        }
    } else if (warp < 2 + 4 * kDequantGroups) {
        // ---------------- codes -> bf16 operand in tensor memory ----------------
        // Group `grp` takes every second step; a thread turns one weight row's 64 codes into 32 pairs.
        const uint32_t grp = (uint32_t)(warp - 2) >> 2;
        const uint32_t m = (uint32_t)(warp & 3) * 32u + (uint32_t)lane;  // weight row of the unit = TMEM lane
        const uint32_t tmemLane = tmemBase + kOperandCol + (((uint32_t)(warp & 3) * 32u) << 16);
        const uint16_t *biases = (MODE == kGateUp && m >= 64u) ? args.bias[1] : args.bias[0];
        uint32_t st = grp, phase = 0, op = grp, stepNo = grp;
        uint32_t g = grp;
        for (uint32_t u = firstUnit; u < units;) {
            if (g >= steps) {
                g -= steps;
                u += unitStride;
                continue;
            }
            // the operand stage was last read four steps back: that step's signal on the token ring
            const uint32_t back = (st + kStages - kOperandStages) % kStages;
            if (!mbar_wait(barCodeFull(st), phase, &abortFlag) ||
                (stepNo >= kOperandStages &&
                 !mbar_wait<Order::kPair>(barTokEmpty(back), ((stepNo - kOperandStages) / kStages) & 1u, &abortFlag)))
                break;
            tc_fence_after();
            uint32_t o[32];
            if (g < groupsK) {
                // the row's 64 bytes lie as four 16-byte chunks with the 64-byte swizzle
                const uint32_t src = codeAddr(st) + m * kStepK, flip = (m >> 1) & 3u;
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    uint32_t w[4];
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                                 : "r"(src + ((c ^ flip) << 4)));
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) {
                        // Two codes as 16-bit numbers ARE a pair of bf16: q * 2^-133, subnormal up to 127.
                        // Times 2^126 they are the operand q / 128, exactly (the drain's scale makes up for
                        // the 128): two instructions for two codes, five by way of floats.
                        const uint32_t pair = __byte_perm(w[i >> 1], 0u, (i & 1u) ? 0x4342u : 0x4140u);
                        asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(o[8 * c + i]) : "r"(pair), "r"(0x7E807E80u));
                    }
                }
            } else {
                const uint32_t nt = ntOf(u);
                const uint32_t wRow = MODE == kGateUp ? nt * 64u + (m & 63u) : nt * 128u + m;
                const uint16_t *row = biases + (size_t)wRow * groupsK;
                const uint32_t g0 = ((g - groupsK) / 3u) * 64u;
#pragma unroll
                for (uint32_t i = 0; i < 32; ++i) {
                    const uint32_t ga = g0 + 2u * i;
                    const uint32_t v0 = wRow < args.N && ga < groupsK ? (uint32_t)__ldg(row + ga) : 0u;
                    const uint32_t v1 = wRow < args.N && ga + 1u < groupsK ? (uint32_t)__ldg(row + ga + 1u) : 0u;
                    o[i] = v0 | (v1 << 16);
                }
            }
            tc_store_32cols(tmemLane + op * 32u, o);
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_pair(map_to_cta(barStep(st), 0u));
                mbar_arrive(barCodeEmpty(st));
            }
            st += kDequantGroups;
            if (st >= kStages) {
                st -= kStages;
                phase ^= 1u;
            }
            op = (op + kDequantGroups) % kOperandStages;
            stepNo += kDequantGroups;
            g += kDequantGroups;
        }
    } else if (warp < (int)(2u + 4u * kDequantGroups + 4u * drainSets)) {
        // ---------------- drain: scaled sums in registers, then the outputs ----------------
        const uint32_t t = (uint32_t)threadIdx.x - (2u + 4u * kDequantGroups) * 32u;  // 0..drainThreads - 1
        const uint32_t set = t >> 7, th = t & 127u;                                   // its tokens of the tile start at kSetTokens set
        const uint32_t quarter = (uint32_t)(warp & 3), m = quarter * 32u + (uint32_t)lane;
        const uint32_t tmemLane = tmemBase + ((quarter * 32u) << 16) + set * kSetTokens;
        float *xchg = reinterpret_cast<float *>(epilogue + set * kXchgBytes);  // gate/up only
        constexpr uint32_t kTilePitch = MODE == kGateUp ? kTilePitchGateUp : kTilePitchDown;
        uint8_t *tileBuf = epilogue + (MODE == kGateUp ? kDrainSets * kXchgBytes : 0u) + set * kPassTokens * kTilePitch;
        const uint32_t leaderAccEmpty = map_to_cta(barAccEmpty(0), 0u);
        uint32_t accPhases = 0, setPhase = 0, unitNo = 0;  // a bit for each accumulator
        // every thread of this set
        auto meet = [&]() {
            mbar_arrive(barSet(set));
            const bool ok = mbar_wait_warp<false, Order::kLocal>(barSet(set), setPhase, &abortFlag);
            setPhase ^= 1u;
            return ok;
        };
        bool ok = true;
        for (uint32_t u = firstUnit; u < units && ok; u += unitStride, ++unitNo) {
            const uint32_t nt = ntOf(u), token0 = tokenOf(u), rows = rowsOf(u);
            const uint32_t setRows = min(rows, (set + 1u) * kSetTokens) - min(rows, set * kSetTokens);
            // the unit's scales: 128 rows (gate/up: 64 of either matrix), contiguous in memory
            uint16_t *scales = scaleBuf + (unitNo & 1u) * 128u * groupsK;
            for (uint32_t i = t; i < 16u * groupsK; i += drainThreads) {  // 16-byte pieces, 8 groupsK per 64 rows
                const uint32_t part = i / (8u * groupsK), piece = i - part * 8u * groupsK;
                const uint32_t row0 = MODE == kGateUp ? nt * 64u : nt * 128u + part * 64u;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (row0 < args.N)  // N is a multiple of 64
                    v = __ldg(reinterpret_cast<const uint4 *>((MODE == kGateUp && part ? args.scale[1] : args.scale[0]) +
                                                              (size_t)row0 * groupsK) + piece);
                *reinterpret_cast<uint4 *>(scales + (size_t)i * 8) = v;
            }
            mbar_arrive(barScales);
            if (!mbar_wait_warp<false, Order::kLocal>(barScales, unitNo & 1u, &abortFlag)) break;
            const uint16_t *myScale = scales + m * groupsK;
            const auto scale_of = [&](uint32_t g) { return g < groupsK ? 128.0f * bf2f(myScale[g]) : 1.0f; };  // (the codes come as q / 128)

            float sums[kSetTokens];
#pragma unroll
            for (int j = 0; j < (int)kSetTokens; ++j) sums[j] = 0.0f;
            float s = scale_of(0);
            for (uint32_t g0 = 0; g0 < steps && ok; g0 += kAccs) {
#pragma unroll
                for (uint32_t a = 0; a < kAccs; ++a) {  // unrolled: the accumulators' addresses are constants
                    const uint32_t g = g0 + a;
                    if (g >= steps) break;
                    if (!mbar_wait_warp<false, Order::kPair>(barAccFull(a), accPhases >> a & 1u, &abortFlag)) {
                        ok = false;
                        break;
                    }
                    accPhases ^= 1u << a;
                    tc_fence_after();
                    if (setRows) {
#pragma unroll
                        for (uint32_t h = 0; h < kSetTokens / 16u; ++h) {
                            uint32_t v[16];
                            tc_load_16cols(tmemLane + a * kMaxRows + 16u * h, v);
                            tc_wait_ld();
#pragma unroll
                            for (int j = 0; j < 16; ++j) sums[16 * h + j] = fmaf(s, __uint_as_float(v[j]), sums[16 * h + j]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_pair(leaderAccEmpty + 8u * a);
                    s = scale_of(g + 1u);
                }
            }
            if (!ok) break;
#pragma unroll
            for (uint32_t c = 0; c < kSetTokens / kPassTokens; ++c) {
                const uint32_t c0 = set * kSetTokens + c * kPassTokens;
                if (!ok || c0 >= rows) break;  // the same for every thread of the set (ok apart, which ends the launch)
                float sum[kPassTokens];
#pragma unroll
                for (int j = 0; j < (int)kPassTokens; ++j)
                    sum[j] = sums[c * kPassTokens + j];
                if (MODE == kGateUp) {
                    // lanes 0..63 hold gate, 64..127 up of features [64 nt, +64): either side takes 8 of the 16
                    // tokens from the other and finishes them (a row's eight floats are turned by m / 4: no bank twice)
                    const bool isUp = m >= 64u;
                    float *mine = xchg + m * 8u;
                    const uint32_t turn = (m >> 2) & 7u;
#pragma unroll
                    for (int j = 0; j < 8; ++j) mine[(uint32_t)j ^ turn] = isUp ? sum[j] : sum[8 + j];
                    if (!meet()) {
                        ok = false;
                        break;
                    }
                    const float *theirs = xchg + (m ^ 64u) * 8u;
                    uint16_t *col = reinterpret_cast<uint16_t *>(tileBuf + (isUp ? 8u : 0u) * kTilePitch) + (m & 63u);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float own = isUp ? sum[8 + j] : sum[j], other = theirs[(uint32_t)j ^ turn];
                        const float gate = bf16_round(isUp ? other : own), up = bf16_round(isUp ? own : other);
                        col[(uint32_t)j * (kTilePitch / 2)] = f2bf(gelu_tanh(gate) * up);
                    }
                } else {
                    uint16_t *col = reinterpret_cast<uint16_t *>(tileBuf) + m;
#pragma unroll
                    for (int j = 0; j < (int)kPassTokens; ++j) col[(uint32_t)j * (kTilePitch / 2)] = f2bf(sum[j]);
                }
                if (!meet()) {
                    ok = false;
                    break;
                }
                // a token's row of the tile: 8 (gate/up) or 16 (down) threads of 16 bytes
                constexpr uint32_t kPieces = MODE == kGateUp ? 8u : 16u, kPerPass = 128u / kPieces;
                const uint32_t piece = th % kPieces;
                const uint32_t col0 = nt * (kPieces * 8u) + piece * 8u;
#pragma unroll
                for (uint32_t pass = 0; pass < kPassTokens / kPerPass; ++pass) {
                    const uint32_t tok = pass * kPerPass + th / kPieces;
                    const bool store = c0 + tok < rows && col0 < args.N;
                    const size_t row = token0 + c0 + tok;
                    const uint4 val = *reinterpret_cast<const uint4 *>(tileBuf + tok * kTilePitch + piece * 16u);
                    if (store) *reinterpret_cast<uint4 *>(args.out + row * args.N + col0) = val;
                    if (MODE == kGateUp) {
                        // the tile's 64 features are one group of the down projection
                        float sg = sum8(val);
                        sg += __shfl_xor_sync(0xFFFFFFFFu, sg, 1);
                        sg += __shfl_xor_sync(0xFFFFFFFFu, sg, 2);
                        sg += __shfl_xor_sync(0xFFFFFFFFu, sg, 4);
                        if (store && piece == 0) store_group_sum(args.sums + row * sums_pitch(args.N), nt, sg);
                    }
                }
                if (MODE == kDown && !meet()) {  // the tile is rewritten next (gate/up: behind the next exchange)
                    ok = false;
                    break;
                }
            }
        }
    }

    // teardown: every thread arrives here, also after a wait that ran out
    __syncwarp();
    if (abortFlag) {
        // give copies still in flight time to land before shared memory is released
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
        if (threadIdx.x == 0) atomicExch(args.errorFlag, 3u + (uint32_t)MODE);
    }
    tc_fence_before();
    __syncthreads();
    // neither CTA leaves (or frees its tensor memory) while the other may still arrive on its
    // barriers or have MMAs reading its shared memory
    cluster_sync_all();
    tc_fence_after();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(512u) : "memory");
    }
}

// bf16 rows [rows][k], box of a CTA's half tile x 64 values; rows past the end read as zero
bool make_token_map(CUtensorMap *map, const uint16_t *base, uint64_t rows, uint64_t k, uint64_t stride, const char **error) {
    const cuuint64_t dims[2] = {k, rows}, strides[1] = {stride * 2};
    const cuuint32_t box[2] = {kStepK, kMaxRows / 2};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "INT8 GEMM", error);
}
bool make_code_map(CUtensorMap *map, const uint8_t *base, uint64_t rows, uint64_t k, const char **error) {
    const cuuint64_t dims[3] = {k, rows, 1}, strides[2] = {k, k * rows};
    const cuuint32_t box[3] = {kStepK, 64, 1};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B, "INT8 GEMM", error);
}

// Tokens per tile: the size whose waves of units take the least time.  A wave of gate/up units over 2816 inputs (47
// steps) takes 18.7, 20.1, 22.3 and 24.8 us with tiles of 32, 64, 96 and 128 tokens (4096 rows, each size forced).
uint32_t pick_tile_rows(uint32_t tokens, uint32_t nPairs, uint32_t clusters) {
    constexpr uint32_t kWave[kMaxRows / 32] = {187, 201, 223, 248};
    uint32_t best = kMaxRows;
    uint64_t bestCost = ~0ull;
    for (uint32_t r = 32; r <= kMaxRows; r += 32) {
        const uint64_t units = (uint64_t)((tokens + r - 1) / r) * nPairs;
        const uint64_t cost = ((units + clusters - 1) / clusters) * kWave[r / 32 - 1];
        if (cost <= bestCost) {
            bestCost = cost;
            best = r;
        }
    }
    return best;
}

size_t smem_bytes(int mode, uint32_t K) {
    return 1024 + (size_t)kStages * (kTokBytes + kCodeBytes) + 2 * 128 * (size_t)(K / kStepK) * 2 +
           (mode == kGateUp ? kDrainSets * (kXchgBytes + kPassTokens * kTilePitchGateUp) : kDrainSets * kPassTokens * kTilePitchDown);
}

template <int MODE>
bool launch_one(FFContext *ctx, const CUtensorMap &tok, const CUtensorMap &sums, const CUtensorMap &w0, const CUtensorMap &w1,
                Int8GemmArgs args, cudaStream_t stream, const char **error) {
    const size_t smem = smem_bytes(MODE, args.K);
    static KernelSmemMemo memo;
    if (!memo.prepare(k_int8_gemm<MODE>, ctx->device, smem, kThreads, nullptr, error)) return false;
    const uint32_t nPairs = (args.nTiles + 1) / 2, clusters = (uint32_t)ctx->smCount / 2;
    args.tileRows = pick_tile_rows(args.tokens, nPairs, clusters);
    args.rowTiles = (args.tokens + args.tileRows - 1) / args.tileRows;
    const uint32_t grid = 2u * std::max(1u, std::min(clusters, args.rowTiles * nPairs));
    {
        LaunchScope scope(ctx, stream, MODE == kGateUp ? "int8_gemm_gate_up_act" : "int8_gemm_down");
        FF_CUDA_OK(launch_pdl(k_int8_gemm<MODE>, grid, kThreads, smem, stream,
                              tok, sums, w0, w1, args),
                   error);
    }
    return true;
}

}  // namespace

bool int8_gemm_fits(uint32_t d, uint32_t f) {
    return smem_bytes(kGateUp, d) <= 226 * 1024 && smem_bytes(kDown, f) <= 226 * 1024;
}

// y = down(r16(gelu_tanh(r16(gate x)) * r16(up x))); scratch from alloc_int8_gemm.
bool launch_shared_int8_gemm(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                             uint16_t *y, cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (!ctx->xSums || !ctx->actSums) return fail(error, "context has no scratch for the INT8 shared FFN's GEMM");
    {
        LaunchScope scope(ctx, stream, "group_sums");
        const size_t threads = (size_t)tokens * (c.d / 8);
        const unsigned blocks = (unsigned)std::min<size_t>((threads + 255) / 256, (size_t)ctx->smCount * 8);
        FF_CUDA_OK(launch_pdl(k_group_sums, blocks, 256, 0, stream,
                              x, xStride, tokens, c.d, ctx->xSums),
                   error);
    }
    CUtensorMap tok, sums, w[2];
    Int8GemmArgs a{};
    for (int m = 0; m < 2; ++m) {
        a.scale[m] = L.shared8S[m];
        a.bias[m] = L.shared8B[m];
        if (!make_code_map(&w[m], L.shared8W[m], c.sharedF, c.d, error)) return false;
    }
    a.K = c.d;
    a.N = c.sharedF;
    a.nTiles = c.sharedF / 64;
    a.tokens = tokens;
    a.out = ctx->sharedActs;
    a.sums = ctx->actSums;
    a.errorFlag = ctx->errorFlag;
    if (!make_token_map(&tok, x, tokens, c.d, xStride, error) ||
        !make_token_map(&sums, ctx->xSums, tokens, sums_pitch(c.d), sums_pitch(c.d), error) ||
        !launch_one<kGateUp>(ctx, tok, sums, w[0], w[1], a, stream, error))
        return false;
    a.scale[0] = a.scale[1] = L.shared8S[2];
    a.bias[0] = a.bias[1] = L.shared8B[2];
    a.K = c.sharedF;
    a.N = c.d;
    a.nTiles = (c.d + 127) / 128;
    a.out = y;
    return make_code_map(&w[0], L.shared8W[2], c.d, c.sharedF, error) &&
           make_token_map(&tok, ctx->sharedActs, tokens, c.sharedF, c.sharedF, error) &&
           make_token_map(&sums, ctx->actSums, tokens, sums_pitch(c.sharedF), sums_pitch(c.sharedF), error) &&
           launch_one<kDown>(ctx, tok, sums, w[0], w[0], a, stream, error);
}

// Group sums of the input rows and of the activations; the columns past a row's groups stay zero.
bool alloc_int8_gemm(FFContext *ctx, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (c.maxTokens <= (uint32_t)kMaxGemvRows || ctx->actSums) return true;
    uint16_t **bufs[2] = {&ctx->xSums, &ctx->actSums};
    const size_t bytes[2] = {(size_t)c.maxTokens * sums_pitch(c.d) * 2, (size_t)c.maxTokens * sums_pitch(c.sharedF) * 2};
    for (int i = 0; i < 2; ++i) {
        if (*bufs[i]) continue;
        FF_CUDA_OK(cudaMalloc(reinterpret_cast<void **>(bufs[i]), bytes[i]), error);
        FF_CUDA_OK(cudaMemset(*bufs[i], 0, bytes[i]), error);
        ctx->scratchBytes += bytes[i];
    }
    return true;
}

}  // namespace ff
