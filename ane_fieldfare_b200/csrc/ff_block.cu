// Packed matrices against 1..16 input rows (a verify block): gate/up + GeGLU and down of the routed
// experts a block touches and of the shared FFN (INT4 or INT8), on the integer tensor cores straight
// on the codes (see ff_int_device.cuh).
//
// Work is cut into tasks: a tile of 16 weight rows (8 gate + 8 up, or 16 down rows) of one job — the
// shared FFN or an expert — against up to four of the job's input rows, which fill two MMAs' digit
// columns.  Every CTA makes the same plan from the route ids in shared memory (which routes chose each
// expert, in order; the jobs' costs) and takes a contiguous run of tasks, the same cost for every CTA,
// so it meets one or two experts, whose few input rows it stages as digits: a job's rows are staged
// where they are used, not all sixteen rows everywhere.  The CTA's warps deal the run's tiles round
// robin; a tile's rows come in parts along K as tensor copies into the warp's two slots, so one part is
// in flight while the other is multiplied, across tasks and experts.  All parts of a tile accumulate in
// the same registers, so no partial sums cross warps and results do not depend on scheduling.
//
// INT4: an input row has one scale for its digits, a group's sums are scaled once by the weights' scale,
// and the bias part is a few small bf16 MMAs on the group sums: 13 instructions per group for the
// weights and 9 for a pair of rows, per warp.  A row that has groups far below its largest value loses their
// digits, which shows where the weights of that value are zero (one value of 2^20 times the rest: 2 % error
// of the outputs), so a CTA forms its outputs of such rows once more in fp32 (redo_uneven_rows; the look at
// the groups and the code behind the loop cost 2 to 4 %: four layers of 5 rows 218.1 -> 221.5 us, of 16 rows
// 304.6 -> 315.8).  INT8: the two parts cancel in part, so they are joined group by group, and every group has
// its own scale.
//
// Reference kernels replaced (paths inside the reference project):
//   Sources/ANEFieldfareHotpath/Metal/Prefill/prefill.metal:1246-1529 (verify grouped GEMV)
//   Sources/ANEFieldfareHotpath/Metal/Quant/dequant_int4.metal:230-459 (multi-row INT4 GEMV)
//   Sources/ANEFieldfareHotpath/Metal/Quant/dequant_int8.metal:41-138 (INT8 rows)
#include <algorithm>
#include <cstring>

#include <type_traits>

#include "ff_int_device.cuh"
#include "ff_tc_device.cuh"

namespace ff {
namespace {

constexpr int kMaxWarps = 16;
constexpr int kTaskRows = 4;          // input rows of a task (2 where the rows are too wide for four as digits)
constexpr uint32_t kPartGroups = 8;   // groups of a part along K, a multiple of four
constexpr uint32_t kUneven = 10;      // INT4: a row is formed in fp32 if a group is this many powers of two below its largest value
constexpr int kMaxJobs = kMaxGemvRows * 8 + 1;

enum Mode : int { kGateUp = 0, kDown = 1 };

// One kind of job: where its weight rows and scale words are (maps) and how its rows are laid out.
struct BlockKind {
    uint32_t tiles;       // tiles of 16 weight rows
    uint32_t groups;      // groups along K
    uint32_t part;        // groups of a part (all of them when that is little more than kPartGroups)
    uint32_t pitch;       // bytes between a slot's rows (= the weight box's width)
    uint32_t sbWords;     // scale words of a row in a slot (= the scale box's width)
    const uint16_t *in;   // input rows (bf16)
    uint32_t inStride;
    uint16_t *out;        // output rows
    uint32_t outStride;
};

struct BlockArgs {
    BlockKind kind[2];    // [0] shared FFN, [1] routed experts
    const uint32_t *ids;  // [T][K] (routed), null: shared FFN only
    int T, K, E, withShared;
    uint32_t *activeExperts;  // gate/up: receives the count (may be null)
    uint32_t *errorFlag;
    uint32_t listOffset, digitsOffset, rowBytes, auxOffset, auxRow, slotsOffset, slotBytes, sbOffset;
    uint32_t planOffset;      // INT4: this CTA's run and the jobs, for redo_run
    int perExpert;            // routes of one expert at most
    int taskShift;            // log2 of a task's input rows
    float *values;            // F32OUT: the routed rows
};

struct alignas(64) BlockMaps {
    struct {
        CUtensorMap w[3];  // gate, up | down, -; scale words
    } kind[2];
};
static_assert(sizeof(BlockMaps) == sizeof(LayerStore::blockMap[0]), "copied as one");

// ---- INT8: four groups of a tile against NT pairs of input rows ------------------------------------
//
// lo / hi: this lane's 16 codes of tile rows g and g + 8 per group, dig[j] its digits of pair j (columns 0..3 one row, 4..7
// the other), sb0 / sb1 the rows' scale words, aux[j] the groups of the row this lane accounts for (t < 2
// the pair's first, else its second).  acc[j][r]: r = 0 row g, 1 row g + 8, in units of 2^16 for the high
// digits (t even), whose lanes also take the bias part (biasUnit = 2^-16, else 0).  A group's scale and
// bias parts, which cancel in part, are joined before they are added up, and four groups before they
// join the running sum.
template <int NT>
__device__ __forceinline__ void four_groups8(uint32_t lo, uint32_t hi, const uint32_t (&dig)[NT], uint32_t sb0, uint32_t sb1,
                                            const uint32_t (&aux)[NT], float biasUnit, float (&acc)[NT][2]) {
    uint4 a[4], b[4], x[NT][4], ax[NT][2];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        a[u] = lds128(lo + 64 * u);
        b[u] = lds128(hi + 64 * u);
#pragma unroll
        for (int j = 0; j < NT; ++j) x[j][u] = lds128(dig[j] + kDigitGroupBytes * u);
    }
    const uint4 s0 = lds128(sb0), s1 = lds128(sb1);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        ax[j][0] = lds128(aux[j]);
        ax[j][1] = lds128(aux[j] + 16u);
    }
    const uint32_t w0[4] = {s0.x, s0.y, s0.z, s0.w}, w1[4] = {s1.x, s1.y, s1.z, s1.w};
    int d[NT][4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            d[j][u][0] = d[j][u][1] = d[j][u][2] = d[j][u][3] = 0;
            mma_u8s8(d[j][u], a[u].x, b[u].x, a[u].y, b[u].y, x[j][u].x, x[j][u].y);
        }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_u8s8(d[j][u], a[u].z, b[u].z, a[u].w, b[u].w, x[j][u].z, x[j][u].w);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        float sum0 = 0.0f, sum1 = 0.0f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint4 &q = ax[j][u >> 1];
            const float unit = __uint_as_float((u & 1) ? q.z : q.x), xs = __uint_as_float((u & 1) ? q.w : q.y) * biasUnit;
            sum0 += fmaf(__uint_as_float(w0[u] << 16) * unit, (float)(d[j][u][0] * 256 + d[j][u][1]), __uint_as_float(w0[u] & 0xFFFF0000u) * xs);
            sum1 += fmaf(__uint_as_float(w1[u] << 16) * unit, (float)(d[j][u][2] * 256 + d[j][u][3]), __uint_as_float(w1[u] & 0xFFFF0000u) * xs);
        }
        acc[j][0] += sum0;
        acc[j][1] += sum1;
    }
}

// ---- INT4: four groups of a tile against NT pairs of input rows ------------------------------------
//
// lo / hi: this lane's eight packed bytes of tile rows g and g + 8 per group, dig[j] its digits of pair j
// (columns 0..3 one row, 4..7 the other), sb0 / sb1 the rows' scale words.  acc[j][r] += scale * digits
// (r = 0 row g, 1 row g + 8) in the input row's unit; t even holds the high digits, in units of 2^16.
template <int NT>
__device__ __forceinline__ void four_groups4(uint32_t lo, uint32_t hi, const uint32_t (&dig)[NT], uint32_t sb0, uint32_t sb1,
                                             float (&acc)[NT][2]) {
    uint2 p[4], q[4];
    uint4 x[NT][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        p[u] = lds64(lo + 32 * u);
        q[u] = lds64(hi + 32 * u);
#pragma unroll
        for (int j = 0; j < NT; ++j) x[j][u] = lds128(dig[j] + kDigitGroupBytes * u);
    }
    const uint4 s0 = lds128(sb0), s1 = lds128(sb1);
    int d[NT][4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            d[j][u][0] = d[j][u][1] = d[j][u][2] = d[j][u][3] = 0;
            mma_u8s8(d[j][u], p[u].x & 0x0F0F0F0Fu, q[u].x & 0x0F0F0F0Fu, p[u].y & 0x0F0F0F0Fu, q[u].y & 0x0F0F0F0Fu, x[j][u].x, x[j][u].y);
        }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j)
            mma_u8s8(d[j][u], p[u].x & 0xF0F0F0F0u, q[u].x & 0xF0F0F0F0u, p[u].y & 0xF0F0F0F0u, q[u].y & 0xF0F0F0F0u, x[j][u].z, x[j][u].w);
    const uint32_t w0[4] = {s0.x, s0.y, s0.z, s0.w}, w1[4] = {s1.x, s1.y, s1.z, s1.w};
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            acc[j][0] = fmaf(__uint_as_float(w0[u] << 16), (float)(d[j][u][0] * 256 + d[j][u][1]), acc[j][0]);
            acc[j][1] = fmaf(__uint_as_float(w1[u] << 16), (float)(d[j][u][2] * 256 + d[j][u][3]), acc[j][1]);
        }
}
// Bias part of eight groups: the biases (high halves of the scale words) against the group sums, which lie
// as bf16 pieces in MMA columns 0..3 (a pair's first row) and 4..7 (its second).
__device__ __forceinline__ void mma_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0));
}
constexpr uint32_t kSumBlockBytes = 128;  // [column][8 groups] bf16

// What redo_uneven_rows reads: the arguments once more (these are passed on by address), and per kind the weight rows and scale words behind the maps and what lies between experts.
struct RedoArgs {
    BlockArgs a;
    struct {
        const uint8_t *w[2];
        const uint32_t *scales;
        uint64_t stride, scaleStride;
    } kind[2];
};
// A weight row against an input row in fp32, by one thread.
__device__ __forceinline__ float fp32_row(const uint4 *w, const uint32_t *words, const uint4 *x, uint32_t groups) {
    float acc = 0.0f;
#pragma unroll 1
    for (uint32_t g = 0; g < groups; ++g) {
        float dot = 0.0f, sum = 0.0f;
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
            const uint4 q = __ldg(w + 2u * g + half);
            const uint32_t codes[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 v = __ldcg(x + 8u * g + 4u * half + (uint32_t)i);
                const uint32_t xs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float even = __uint_as_float(xs[j] << 16), odd = __uint_as_float(xs[j] & 0xFFFF0000u);
                    dot = fmaf((float)((codes[i] >> (8 * j)) & 15u), even, dot);
                    dot = fmaf((float)((codes[i] >> (8 * j + 4)) & 15u), odd, dot);
                    sum += even + odd;
                }
            }
        }
        const uint32_t word = __ldg(words + g);
        acc = fmaf(__uint_as_float(word << 16), dot, acc);
        acc = fmaf(__uint_as_float(word & 0xFFFF0000u), sum, acc);
    }
    return acc;
}
// The outputs of one of a CTA's segments (tiles [tile0, tileEnd) of job `job`'s input rows [first, last)) for the rows that
// have a group kUneven powers of two below their largest value (not all zero), once more, over what the digits gave.
// A thread a weight row.
template <int MODE, bool F32OUT>
__device__ __forceinline__ void redo_uneven_rows(const RedoArgs &r, uint32_t job, const uint8_t *list, int first, int last, uint32_t tile0,
                                                 uint32_t tileEnd) {
    constexpr uint32_t kRows = MODE == kGateUp ? 8 : 16;
    const int kind = job ? 1 : 0;
    const uint64_t expert = kind ? job - 1u : 0u;
    const BlockKind &k = r.a.kind[kind];
    const uint32_t groups = k.groups;
    for (int i = first; i < last; ++i) {
        const int outRow = kind ? (int)list[expert * kMaxGemvRows + (uint32_t)i] : i, inRow = MODE == kGateUp && kind ? outRow / r.a.K : outRow;
        const uint4 *x = reinterpret_cast<const uint4 *>(k.in + (size_t)inRow * k.inStride);
        uint32_t top = 0, least = 0xFFFFu;  // the row's largest value, the smallest of its groups' largest ones
#pragma unroll 1
        for (uint32_t g = 0; g < groups; ++g) {
            uint32_t group = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) group = max(group, top_exponent(__ldcg(x + 8u * g + j)));
            top = max(top, group);
            if (group) least = min(least, group);
        }
        if (least + (kUneven << 7) >= top) continue;
        for (uint32_t row = tile0 * kRows + threadIdx.x; row < tileEnd * kRows; row += blockDim.x) {
            const uint32_t scaleRow = row / kRows * 16u + row % kRows;
            auto dot = [&](int matrix) {
                return fp32_row(reinterpret_cast<const uint4 *>(r.kind[kind].w[matrix] + expert * r.kind[kind].stride) + (size_t)row * groups * 2u,
                                r.kind[kind].scales + expert * r.kind[kind].scaleStride + (size_t)(scaleRow + 8u * matrix) * padded_groups(groups), x,
                                groups);
            };
            const float v = dot(0);
            const size_t to = (size_t)outRow * k.outStride + row;
            if (MODE == kGateUp) {
                const float u = dot(1);
                const float gate = kind ? v : bf16_round(v), up = kind ? u : bf16_round(u);
                k.out[to] = f2bf(gelu_tanh(gate) * up);
            } else if (F32OUT && kind) {
                r.a.values[to] = v;
            } else {
                k.out[to] = f2bf(v);
            }
        }
    }
}

// redo_uneven_rows for every segment of a CTA's run, from a copy of the plan in dynamic shared memory.  (With the static
// arrays' addresses passed on, the main loop reads them again after every store.)
template <int MODE, bool F32OUT>
__device__ __noinline__ void redo_run(const RedoArgs &r, const uint8_t *smemRaw) {
    const uint32_t *plan = reinterpret_cast<const uint32_t *>(smemRaw + r.a.planOffset);
    const uint32_t endJob = plan[3], endGroup = plan[4], endTile = plan[5], nJobs = plan[6];
    uint32_t j = plan[0], rg = plan[1], tile = plan[2];
    for (; j < nJobs && j <= endJob; ++j, rg = 0, tile = 0) {
        const uint32_t job = plan[7u + j] & 0xFFFFu;
        const int rows = (int)(plan[7u + j] >> 16);
        for (; (int)(rg << r.a.taskShift) < rows; ++rg, tile = 0) {
            const bool last = j == endJob && rg == endGroup;
            const int first = (int)(rg << r.a.taskShift);
            redo_uneven_rows<MODE, F32OUT>(r, job, smemRaw + r.a.listOffset, first, min(rows, first + (1 << r.a.taskShift)), tile,
                                           last ? endTile : r.a.kind[job ? 1 : 0].tiles);
            if (last) return;
        }
    }
}

// F32OUT (down): the routed rows go to `values` unrounded.
template <int MODE, bool INT8, bool F32OUT>
__global__ void __launch_bounds__(kMaxWarps * 32, 1)
k_block_int(const BlockArgs a, const __grid_constant__ BlockMaps maps, const __grid_constant__ RedoArgs redo) {
    extern __shared__ __align__(128) uint8_t smemRaw[];
    __shared__ uint32_t sFirst[kMaxJobs + 1];   // cost of the jobs before job k (active jobs, the shared FFN first)
    __shared__ uint16_t sJob[kMaxJobs];         // 0 the shared FFN, 1 + e expert e
    __shared__ uint32_t sCount[kMaxExperts], sWarpSum[2][kMaxWarps], sTop[kMaxWarps];
    __shared__ float sUnit[kTaskRows];
    __shared__ uint32_t sUneven;  // a row of this CTA's run may be one for redo_uneven_rows
    __shared__ __align__(8) uint64_t sBar[2 * kMaxWarps];
    uint8_t *sList = smemRaw + a.listOffset;  // [expert][16] route numbers (< 128)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)(blockDim.x >> 5);
    const int g = lane >> 2, t = lane & 3;
    const uint32_t smem = sm_addr(smemRaw);
    constexpr uint32_t kGroupBytes = INT8 ? 64 : 32;
    // Plan and first weights of the down kernel need only what was there before its predecessor, those of the INT8 FFN
    // nothing that a launch writes (a decode forward of four INT8 layers 193 -> 187.5 us with them in front of the wait).
    constexpr bool kLateWait = MODE == kDown || INT8;
    if (!kLateWait) {
        pdl_wait();
        pdl_trigger();
    }
    if (threadIdx.x == 0) {
        sUneven = 0u;
        for (int i = 0; i < 2 * kMaxWarps; ++i) bar_init(sm_addr(&sBar[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // ---- the plan: routes of every expert in (token, rank) order, cost of every job ----
    const int routes = a.ids ? a.T * a.K : 0;
    for (int e = threadIdx.x; e < a.E; e += blockDim.x) sCount[e] = 0u;
    __syncthreads();
    if (warp < 4) {
        const int r = warp * 32 + lane;
        const uint32_t id = r < routes ? a.ids[r] : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, id), before = __popc(peers & ((1u << lane) - 1u));
        const bool known = id < (uint32_t)a.E;
        // A block's tokens choose distinct experts, so an expert has at most T routes (a single row may name
        // one several times); repeats beyond that and routes past the resident experts keep their rows unwritten and raise the flag
        // (the reference refuses such a route with "route expert N is out of range").
        for (int w = 0; w < 4; ++w) {  // warps in turn: a route's place counts all earlier ones
            if (warp == w && r < routes) {
                const uint32_t place = known ? sCount[id] + before : 0u;
                if (known && place < (uint32_t)a.perExpert) sList[id * kMaxGemvRows + place] = (uint8_t)r;
                else atomicExch(a.errorFlag, 12u);
            }
            __syncwarp();
            if (warp == w && r < routes && known && before == 0) sCount[id] = min(sCount[id] + (uint32_t)__popc(peers), (uint32_t)a.perExpert);
            named_barrier(1, 128);
        }
    }
    __syncthreads();
    // instructions of a tile: per group what the weights cost and what a pair of rows costs, and its set-up
    const uint32_t taskRows = 1u << a.taskShift;
    auto tile_cost = [&](int kind, int rows) { return a.kind[kind].groups * (rows > 2 ? 31u : 22u) + 100u; };
    auto job_cost = [&](int kind, int rows) {
        const uint32_t full = (uint32_t)rows >> a.taskShift, rest = (uint32_t)rows & (taskRows - 1u);
        return a.kind[kind].tiles * (full * tile_cost(kind, (int)taskRows) + (rest ? tile_cost(kind, (int)rest) : 0u));
    };
    uint32_t nJobs = a.withShared ? 1u : 0u;
    {
        uint32_t base = a.withShared ? job_cost(0, a.T) : 0u;
        if (threadIdx.x == 0) {
            sFirst[0] = 0u;
            sJob[0] = 0;
        }
        __syncthreads();
        for (int e0 = 0; e0 < a.E; e0 += (int)blockDim.x) {
            const int e = e0 + (int)threadIdx.x;
            const uint32_t n = e < a.E ? sCount[e] : 0u, cost = n ? job_cost(1, (int)n) : 0u;
            uint32_t incl = cost;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += v;
            }
            const uint32_t active = __ballot_sync(0xFFFFFFFFu, n > 0u);
            if (lane == 31) {
                sWarpSum[0][warp] = incl;
                sWarpSum[1][warp] = __popc(active);
            }
            __syncthreads();
            uint32_t costBefore = base, jobsBefore = nJobs;
            for (int w = 0; w < warps; ++w) {
                if (w < warp) {
                    costBefore += sWarpSum[0][w];
                    jobsBefore += sWarpSum[1][w];
                }
                base += sWarpSum[0][w];
                nJobs += sWarpSum[1][w];
            }
            if (n) {
                const uint32_t k = jobsBefore + __popc(active & ((1u << lane) - 1u));
                sJob[k] = (uint16_t)(1 + e);
                sFirst[k] = costBefore + incl - cost;
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) sFirst[nJobs] = base;
        if (MODE == kGateUp && threadIdx.x == 0 && blockIdx.x == 0 && a.activeExperts) *a.activeExperts = nJobs - (a.withShared ? 1u : 0u);
    }
    __syncthreads();
    if (nJobs == 0) {
        pdl_wait();
        return;
    }

    // A tile of four input rows (`rowGroup`) of a job; tiles in order are a CTA's run.
    struct Place {
        uint32_t job, rowGroup, tile;
    };
    auto kind_of = [&](uint32_t job) { return sJob[job] ? 1 : 0; };
    auto rows_of = [&](uint32_t job) { return sJob[job] ? (int)sCount[sJob[job] - 1] : a.T; };
    auto place_of = [&](uint32_t cta) {  // the first tile whose cost position is not before the CTA's share
        if (cta == gridDim.x) return Place{nJobs, 0u, 0u};
        const uint32_t target = (uint32_t)((uint64_t)sFirst[nJobs] * cta / gridDim.x);
        uint32_t lo = 0, hi = nJobs;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sFirst[mid] <= target) lo = mid;
            else hi = mid;
        }
        const int kind = kind_of(lo), rows = rows_of(lo);
        const uint32_t tiles = a.kind[kind].tiles, full = (uint32_t)rows >> a.taskShift;
        uint32_t cost = tile_cost(kind, (int)taskRows), rest = target - sFirst[lo];
        const uint32_t rg = min(full, rest / (tiles * cost));
        rest -= rg * tiles * cost;
        if (rg == full) cost = tile_cost(kind, (int)((uint32_t)rows & (taskRows - 1u)));
        return Place{lo, rg, (rest + cost - 1u) / cost};  // (may be one past the row group's last tile)
    };
    auto before = [](const Place &p, const Place &q) {
        return p.job != q.job ? p.job < q.job : p.rowGroup != q.rowGroup ? p.rowGroup < q.rowGroup : p.tile < q.tile;
    };
    auto settle = [&](Place &p) {  // tiles past a row group belong to the next
        while (p.job < nJobs) {
            const uint32_t tiles = a.kind[kind_of(p.job)].tiles;
            if (p.tile < tiles) break;
            p.tile -= tiles;
            if ((int)(++p.rowGroup << a.taskShift) >= rows_of(p.job)) {
                p.rowGroup = 0;
                ++p.job;
            }
        }
        if (p.job >= nJobs) p = Place{nJobs, 0u, 0u};
    };
    Place at = place_of(blockIdx.x), end = place_of(blockIdx.x + 1u);
    settle(at);
    settle(end);
    if (!INT8) {
        uint32_t *plan = reinterpret_cast<uint32_t *>(smemRaw + a.planOffset);
        const uint32_t run[7] = {at.job, at.rowGroup, at.tile, end.job, end.rowGroup, end.tile, nJobs};
        if (threadIdx.x < 7) {
            uint32_t v = run[0];
#pragma unroll
            for (int i = 1; i < 7; ++i) v = threadIdx.x == i ? run[i] : v;
            plan[threadIdx.x] = v;
        }
        for (uint32_t j = threadIdx.x; j < nJobs; j += blockDim.x) plan[7u + j] = sJob[j] | (uint32_t)rows_of(j) << 16;
    }

    // ---- copies: this warp's steps (tile, part) in order, two slots in turn ----
    const uint32_t slots = smem + a.slotsOffset + (uint32_t)warp * 2u * a.slotBytes;
    const uint32_t bars = sm_addr(&sBar[2 * warp]);
    Place askAt = at;
    askAt.tile += (uint32_t)warp;
    uint32_t askLimit = 0, askX = 0, askGroups = 0, askPart = 0, askBytes = 0, askHalf = 0, asked = 0;
    int askZ = 0;
    const CUtensorMap *askMap = nullptr;
    // the next row group the warp has a tile in, or none (askLimit 0)
    auto seek = [&]() {
        settle(askAt);
        askLimit = 0;
        if (!before(askAt, end)) return;
        const int kind = kind_of(askAt.job);
        const BlockKind &k = a.kind[kind];
        askLimit = askAt.job == end.job && askAt.rowGroup == end.rowGroup ? end.tile : k.tiles;
        askGroups = k.groups;
        askPart = k.part;
        askBytes = 16u * k.pitch + 64u * k.sbWords;
        askHalf = 8u * k.pitch;
        askZ = kind ? (int)sJob[askAt.job] - 1 : 0;
        askMap = &maps.kind[kind].w[0];
    };
    seek();
    auto ask = [&]() {
        if (askLimit == 0) return;
        if (lane == 0) {
            const uint32_t slot = slots + (asked & 1u) * a.slotBytes, bar = bars + 8u * (asked & 1u);
            const int row = (int)askAt.tile * (MODE == kGateUp ? 8 : 16), x = (int)(askX * (kGroupBytes / 8u));
            bar_expect(bar, askBytes);
            tma_load_3d(slot, askMap, x, row, askZ, bar);
            if (MODE == kGateUp) tma_load_3d(slot + askHalf, askMap + 1, x, row, askZ, bar);
            tma_load_3d(slot + a.sbOffset, askMap + 2, (int)askX, (int)askAt.tile * 16, askZ, bar);
        }
        ++asked;
        askX += askPart;
        if (askX >= askGroups) {
            askX = 0;
            askAt.tile += (uint32_t)warps;
            if (askAt.tile >= askLimit) seek();
        }
    };
    ask();
    ask();

    // ---- input rows as digits: row r by warps [r per, (r + 1) per) ----
    const float biasUnit = (t & 1) ? 0.0f : 1.52587890625e-5f;  // 2^-16 (INT8, see four_groups8)
    auto stage = [&](const BlockKind &k, int kind, int n, auto row_of) {
        const int per = warps / n, r = warp / per, threads = per * 32, tid = (int)threadIdx.x - r * threads;
        const int runs = (int)k.groups * 8;
        if (r >= n) return;
        int row = row_of(r);
        if (MODE == kGateUp && kind) row /= a.K;  // a route's token
        const uint4 *src = reinterpret_cast<const uint4 *>(k.in + (size_t)row * k.inStride);
        uint8_t *digits = smemRaw + a.digitsOffset + (size_t)r * a.rowBytes;
        constexpr int kHeld = 3;  // runs a thread keeps between the two passes
        uint4 held[kHeld];
#pragma unroll
        for (int i = 0; i < kHeld; ++i) {
            held[i] = make_uint4(0, 0, 0, 0);
            if (tid + i * threads < runs) held[i] = __ldcg(src + tid + i * threads);
        }
        if constexpr (INT8) {
            GroupAux *rowAux = reinterpret_cast<GroupAux *>(smemRaw + a.auxOffset + (size_t)r * a.auxRow);
            auto put = [&](int i, const uint4 &v) { digits_put<true>(i, i < runs, v, digits, rowAux + (i >> 3)); };
#pragma unroll
            for (int i = 0; i < kHeld; ++i)
                if ((tid & ~31) + i * threads < runs) put(tid + i * threads, held[i]);  // the same for the whole warp
            for (int i = tid + kHeld * threads; (i & ~31) < runs; i += threads) put(i, i < runs ? __ldcg(src + i) : make_uint4(0, 0, 0, 0));
            const int padded = ((int)k.groups + 3) & ~3;  // groups past the row add nothing
            if (tid < padded - (int)k.groups) rowAux[(int)k.groups + tid] = GroupAux{0.0f, 0.0f};
        } else {
            uint32_t top = 0, low = 0xFFFFu;  // the largest and the smallest of the runs' largest values
            auto look = [&](int i, const uint4 &v) {
                const uint32_t t = top_exponent(v);
                top = max(top, t);
                if (i < runs) low = min(low, t);
            };
#pragma unroll
            for (int i = 0; i < kHeld; ++i) look(tid + i * threads, held[i]);
            for (int i = tid + kHeld * threads; i < runs; i += threads) look(i, __ldcg(src + i));
            top = __reduce_max_sync(0xFFFFFFFFu, top);
            if (lane == 0) sTop[warp] = top;
            named_barrier(2 + r, threads);
            for (int w = 0; w < per; ++w) top = max(top, sTop[r * per + w]);
            if (!__all_sync(0xFFFFFFFFu, low + (kUneven << 7) >= top)) {  // a run of eight is that small: a whole group?
                auto check = [&](int i, const uint4 &v) {  // a group's eight lanes are a byte of the ballots
                    const uint32_t t = top_exponent(v);
                    uint32_t large = __ballot_sync(0xFFFFFFFFu, t + (kUneven << 7) >= top), some = __ballot_sync(0xFFFFFFFFu, i < runs && t != 0u);
                    large |= large >> 4 & 0x0F0F0F0Fu, some |= some >> 4 & 0x0F0F0F0Fu;
                    large |= large >> 2, some |= some >> 2;
                    large |= large >> 1, some |= some >> 1;
                    if (some & ~large & 0x01010101u) sUneven = 1u;
                };
#pragma unroll
                for (int i = 0; i < kHeld; ++i)
                    if ((tid & ~31) + i * threads < runs) check(tid + i * threads, held[i]);  // the same for the whole warp
                for (int i = tid + kHeld * threads; (i & ~31) < runs; i += threads) check(i, i < runs ? __ldcg(src + i) : make_uint4(0, 0, 0, 0));
            }
            const RowScale scale = row_scale(top);
            if (tid == 0) sUnit[r] = scale.unit;
            // pair r / 2, columns 4 (r & 1).. of the sums
            uint8_t *sums = smemRaw + a.auxOffset + (size_t)(r >> 1) * a.auxRow + (uint32_t)(r & 1) * 64u;
            auto put = [&](int i, const uint4 &v) {
                float sum = sum_of_run(v);
#pragma unroll
                for (int o = 1; o <= 4; o <<= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
                if (i >= runs) return;
                digits_store<false>(i, v, scale.toInt, digits);
                if ((i & 7) == 0) {
                    const int group = i >> 3;
                    uint16_t *dst = reinterpret_cast<uint16_t *>(sums + (uint32_t)(group >> 3) * kSumBlockBytes) + (group & 7);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {  // (a fourth piece: what is left, mostly zero)
                        const uint16_t piece = f2bf(sum);
                        dst[8 * c] = piece;
                        sum -= bf2f(piece);
                    }
                }
            };
#pragma unroll
            for (int i = 0; i < kHeld; ++i)
                if ((tid & ~31) + i * threads < runs) put(tid + i * threads, held[i]);  // the same for the whole warp
            for (int i = tid + kHeld * threads; (i & ~31) < runs; i += threads) put(i, i < runs ? __ldcg(src + i) : make_uint4(0, 0, 0, 0));
            // groups past the row up to a block of eight: their biases are zero, the sums have to be finite
            const int past = (((int)k.groups + 7) & ~7) - (int)k.groups;
            for (int i = tid; i < 4 * past; i += threads) {
                const int group = (int)k.groups + (i >> 2);
                *(reinterpret_cast<uint16_t *>(sums + (uint32_t)(group >> 3) * kSumBlockBytes) + (group & 7) + 8 * (i & 3)) = 0;
            }
        }
    };

    if (kLateWait) {
        pdl_wait();  // from here on: the input rows
        pdl_trigger();
    }
    uint32_t used = 0, done = 0;  // done: tiles of this CTA's earlier segments, modulo the warps
    while (before(at, end)) {
        // a segment: the run's tiles of one row group
        const int kind = kind_of(at.job), n = min((int)taskRows, rows_of(at.job) - (int)(at.rowGroup << a.taskShift));
        const BlockKind &k = a.kind[kind];
        const bool same = at.job == end.job && at.rowGroup == end.rowGroup;
        const uint32_t tileEnd = same ? end.tile : k.tiles;
        const uint32_t listAt = kind ? (sJob[at.job] - 1u) * kMaxGemvRows + (at.rowGroup << a.taskShift) : at.rowGroup << a.taskShift;
        auto row_of = [&](int i) { return kind ? (int)sList[listAt + (uint32_t)i] : (int)listAt + i; };  // row i: its route or token
        __syncthreads();  // the previous segment's digits are no longer read
        stage(k, kind, n, row_of);
        __syncthreads();
        // ---- this warp's tiles of the segment ----
        uint32_t tile = at.tile + ((uint32_t)warp + (uint32_t)warps - done) % (uint32_t)warps;
        const uint32_t groups = k.groups, part = k.part, half = 8u * k.pitch, sbHalf = 32u * k.sbWords;
        const uint32_t rowAt = (uint32_t)g * k.pitch + (INT8 ? 16u : 8u) * (uint32_t)t, sbAt = a.sbOffset + (uint32_t)g * k.sbWords * 4u;
        auto run_tiles = [&](auto pairs) {
            constexpr int NT = decltype(pairs)::value;
            for (; tile < tileEnd; tile += (uint32_t)warps) {
                float acc[NT][2], accBias[NT][4];
                uint32_t dig[NT], aux[NT];
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    acc[j][0] = acc[j][1] = 0.0f;
                    accBias[j][0] = accBias[j][1] = accBias[j][2] = accBias[j][3] = 0.0f;
                    const int column = min(2 * j + (g >> 2), n - 1), mine = min(2 * j + (t >> 1), n - 1);
                    dig[j] = smem + a.digitsOffset + (uint32_t)column * a.rowBytes + (uint32_t)(g & 3) * 64u + (uint32_t)t * 16u;
                    // INT8: the groups of the row this lane accounts for; INT4: its column's sums of the pair
                    aux[j] = smem + a.auxOffset + (INT8 ? (uint32_t)mine * a.auxRow : (uint32_t)j * a.auxRow + (uint32_t)g * 16u + (uint32_t)t * 4u);
                }
                for (uint32_t p0 = 0; p0 < groups; p0 += part) {
                    const uint32_t slot = slots + (used & 1u) * a.slotBytes;
                    uint32_t parity = (used >> 1) & 1u;
                    slot_wait(bars + 8u * (used & 1u), parity, a.errorFlag);
                    uint32_t lo = slot + rowAt, hi = lo + half;
                    uint32_t sb0 = slot + sbAt, sb1 = sb0 + sbHalf;
                    const uint32_t inPart = min(part, groups - p0);
                    if (!INT8) {
                        uint32_t w0 = sb0 + 8u * (uint32_t)t, w1 = sb1 + 8u * (uint32_t)t;
#pragma unroll 1
                        for (uint32_t b = 0; b < inPart; b += 8) {
                            const uint2 v0 = lds64(w0), v1 = lds64(w1);
                            const uint32_t a0 = __byte_perm(v0.x, v0.y, 0x7632), a1 = __byte_perm(v1.x, v1.y, 0x7632);
#pragma unroll
                            for (int j = 0; j < NT; ++j) {
                                uint32_t sum;
                                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sum) : "r"(aux[j] + ((p0 + b) >> 3) * kSumBlockBytes));
                                mma_1688(accBias[j], a0, a1, sum);
                            }
                            w0 += 32u;
                            w1 += 32u;
                        }
                    }
#pragma unroll 1
                    for (uint32_t b = 0; b < inPart; b += 4) {
                        if constexpr (INT8) {
                            four_groups8<NT>(lo, hi, dig, sb0, sb1, aux, biasUnit, acc);
#pragma unroll
                            for (int j = 0; j < NT; ++j) aux[j] += 32u;
                        } else {
                            four_groups4<NT>(lo, hi, dig, sb0, sb1, acc);
                        }
                        lo += 4u * kGroupBytes;
                        hi += 4u * kGroupBytes;
                        sb0 += 16u;
                        sb1 += 16u;
#pragma unroll
                        for (int j = 0; j < NT; ++j) dig[j] += 4u * kDigitGroupBytes;
                    }
                    slot_release();
                    ++used;
                    ask();
                }
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    // lane (g, t = 0): the pair's first row, t = 2: its second
                    const int mine = 2 * j + (t >> 1);
                    float r0 = fmaf(acc[j][0], 65536.0f, __shfl_xor_sync(0xFFFFFFFFu, acc[j][0], 1));
                    float r1 = fmaf(acc[j][1], 65536.0f, __shfl_xor_sync(0xFFFFFFFFu, acc[j][1], 1));
                    if (!INT8) {
                        float b0 = accBias[j][0] + accBias[j][1], b1 = accBias[j][2] + accBias[j][3];
                        b0 += __shfl_xor_sync(0xFFFFFFFFu, b0, 1);
                        b1 += __shfl_xor_sync(0xFFFFFFFFu, b1, 1);
                        const float unit = sUnit[min(mine, n - 1)];
                        r0 = fmaf(r0, unit, b0);
                        r1 = fmaf(r1, unit, b1);
                    }
                    if ((t & 1) || mine >= n) continue;
                    const size_t to = (size_t)row_of(mine) * k.outStride;
                    uint16_t *dst = k.out + to;
                    if (MODE == kGateUp) {
                        // the shared FFN rounds gate and up before the activation
                        const float gate = kind ? r0 : bf16_round(r0), up = kind ? r1 : bf16_round(r1);
                        dst[tile * 8u + (uint32_t)g] = f2bf(gelu_tanh(gate) * up);
                    } else if (F32OUT && kind) {
                        a.values[to + tile * 16u + (uint32_t)g] = r0;
                        a.values[to + tile * 16u + 8u + (uint32_t)g] = r1;
                    } else {
                        dst[tile * 16u + (uint32_t)g] = f2bf(r0);
                        dst[tile * 16u + 8u + (uint32_t)g] = f2bf(r1);
                    }
                }
            }
        };
        if (n > 2) run_tiles(std::integral_constant<int, 2>{});
        else run_tiles(std::integral_constant<int, 1>{});
        done = (done + tileEnd - at.tile) % (uint32_t)warps;
        if (same) break;
        at.tile = k.tiles;
        settle(at);
    }
    if (!INT8) {
        __syncthreads();
        if (sUneven) redo_run<MODE, F32OUT>(redo, smemRaw);
    }
}

// ---- host ------------------------------------------------------------------------------------------

bool encode3(CUtensorMap *map, CUtensorMapDataType type, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1,
             uint64_t s2, uint32_t b0, uint32_t b1, const char **error) {
    const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {s1, s2};
    const cuuint32_t box[3] = {b0, b1, 1};
    return encode_map(map, type, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, "block", error);
}

// Slot row pitch of a kind: a part's bytes, padded so that a half-warp's reads fall on different banks
// (INT4 64-bit reads of four rows: 32 or 96 modulo 128; INT8 128-bit reads of two rows: 64).
uint32_t row_pitch(uint32_t part, bool int8) {
    if (!int8) return piece_stride(part * 32);
    uint32_t p = part * 64;
    while ((p & 127u) != 64u) p += 16;
    return p;
}

// Fills a kind and, unless they are there already, its maps.  mode kGateUp: w0, w1 [rows][cols], tiles of 8 + 8 rows; kDown: w0, 16 rows.
bool setup_kind(int mode, bool int8, int kind, RedoArgs &redo, LayerStore &L, const uint8_t *w0, const uint8_t *w1, uint32_t rows, uint32_t cols,
                uint32_t experts, uint64_t stride, const uint32_t *scales, uint64_t scaleStride, const char **error) {
    BlockKind &k = redo.a.kind[kind];
    CUtensorMap(&w)[3] = L.blockMap[mode][kind];
    const uint32_t groups = cols / 64, padded = padded_groups(groups), bit = 1u << (2 * mode + kind);
    const uint64_t rowBytes = int8 ? cols : cols / 2;
    k.tiles = mode == kGateUp ? rows / 8 : rows / 16;
    k.groups = groups;
    k.part = padded <= kPartGroups + 4 ? padded : kPartGroups;
    k.pitch = row_pitch(k.part, int8);
    k.sbWords = (k.part + 7u) & ~7u;  // (words past the row read as zero)
    redo.kind[kind] = {{w0, w1}, scales, stride, scaleStride};
    if (L.blockMapsReady & bit) return true;
    L.blockMapsReady |= bit;
    const uint8_t *ws[2] = {w0, w1};
    for (int m = 0; m < (mode == kGateUp ? 2 : 1); ++m)
        if (!encode3(&w[m], CU_TENSOR_MAP_DATA_TYPE_UINT64, ws[m], rowBytes / 8, rows, experts, rowBytes, stride, k.pitch / 8,
                     mode == kGateUp ? 8 : 16, error))
            return false;
    const uint64_t scaleRows = mode == kGateUp ? (uint64_t)rows * 2 : rows;
    return encode3(&w[2], CU_TENSOR_MAP_DATA_TYPE_UINT32, scales, padded, scaleRows, experts, (uint64_t)padded * 4,
                   experts > 1 ? scaleStride * 4 : scaleRows * padded * 4, k.sbWords, 16, error);
}

template <int MODE, bool INT8, bool F32OUT = false>
bool launch_kernel(FFContext *ctx, RedoArgs redo, const BlockMaps &maps, const char *name, cudaStream_t stream, const char **error) {
    BlockArgs &a = redo.a;
    uint32_t groups = 0, slot = 0, sb = 0;
    for (int i = 0; i < 2; ++i) {
        if (!a.kind[i].tiles) continue;
        groups = std::max(groups, a.kind[i].groups);
        slot = std::max(slot, 16 * a.kind[i].pitch);
        sb = std::max(sb, 64 * a.kind[i].sbWords);
    }
    auto up128 = [](uint32_t v) { return (v + 127u) & ~127u; };
    const uint32_t padded = padded_groups(groups);
    a.sbOffset = up128(slot);
    a.slotBytes = a.sbOffset + up128(sb);
    // (a batch of four groups may read up to three groups past a slot's last row, within the scale area)
    constexpr uint32_t kLimit = 227 * 1024 - 6144;  // less the static arrays
    a.listOffset = 0;
    a.planOffset = a.ids ? (uint32_t)a.E * kMaxGemvRows : 0;
    a.digitsOffset = up128(a.planOffset + (INT8 ? 0u : 4u * (7u + kMaxJobs)));
    a.rowBytes = padded * kDigitGroupBytes;
    // INT8: a row's group entries; INT4: a pair's group sums
    a.auxRow = INT8 ? padded * (uint32_t)sizeof(GroupAux) : (groups + 7u) / 8u * kSumBlockBytes;
    // four input rows a task; two where four leave no room for four warps' slots (widths from 11072 on)
    for (a.taskShift = 2; a.taskShift >= 1; --a.taskShift) {
        const uint32_t rows = (uint32_t)std::min(std::max(a.T, a.perExpert), 1 << a.taskShift);
        a.auxOffset = a.digitsOffset + rows * a.rowBytes;
        a.slotsOffset = up128(a.auxOffset + (INT8 ? rows : (rows + 1u) / 2u) * a.auxRow);
        if (a.slotsOffset + 4 * 2 * a.slotBytes <= kLimit) break;
    }
    if (a.taskShift == 0) return fail(error, "model shape too large for the block kernels' shared memory");
    const uint32_t warps = std::min<uint32_t>(kMaxWarps, (kLimit - a.slotsOffset) / (2 * a.slotBytes));
    const size_t smem = a.slotsOffset + (size_t)warps * 2 * a.slotBytes;
    static KernelSmemMemo memo;
    if (!memo.prepare(k_block_int<MODE, INT8, F32OUT>, ctx->device, kLimit, kMaxWarps * 32, nullptr, error)) return false;
    {
        LaunchScope scope(ctx, stream, name);
        FF_CUDA_OK(launch_pdl(k_block_int<MODE, INT8, F32OUT>, ctx->smCount, warps * 32, smem, stream, a, maps, redo), error);
    }
    return true;
}

}  // namespace

// Routed experts (ids [tokens][K], partial rows to `partials`) and / or the INT4 shared FFN (rows to
// `sharedOut`) of up to 16 rows.  `values` not null: the routed rows go there as fp32 instead, and one row's
// routes may repeat an expert.
bool launch_block_int4(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                       const uint32_t *ids, bool withShared, uint16_t *partials, uint16_t *sharedOut, cudaStream_t stream,
                       const char **error, float *values) {
    const FFConfig &c = ctx->cfg;
    if (c.d % 64 || c.f % 64 || c.sharedF % 64) return fail(error, "widths must be multiples of 64");
    if (((uintptr_t)x & 15) || (xStride % 8)) return fail(error, "input rows must be 16-byte aligned");
    const uint64_t words = scale_words(c.d, c.f);
    LayerStore &Lm = const_cast<LayerStore &>(L);  // (its maps are encoded once per load)
    for (int mode = 0; mode < 2; ++mode) {
        RedoArgs redo{};
        BlockArgs &a = redo.a;
        a.ids = ids;
        a.T = (int)tokens;
        a.K = (int)c.topK;
        a.E = ids ? (int)L.expertCount : 0;
        a.perExpert = values ? (int)c.topK : (int)tokens;
        a.values = values;
        a.withShared = withShared;
        a.activeExperts = &ctx->plan->activeExperts;
        a.errorFlag = ctx->errorFlag;
        const bool down = mode == kDown;
        if (ids) {
            const uint32_t *o = &L.off.gateWOff;
            BlockKind &k = a.kind[1];
            if (!setup_kind(mode, false, 1, redo, Lm, L.experts + (down ? o[6] : o[0]), L.experts + o[3], down ? c.d : c.f,
                            down ? c.f : c.d, L.expertCount, L.stride,
                            L.routedScales + (down ? (uint64_t)(c.f / 8) * 16 * padded_groups(c.d / 64) : 0), words, error))
                return false;
            k.in = down ? ctx->acts : x;
            k.inStride = down ? c.f : xStride;
            k.out = down ? partials : ctx->acts;
            k.outStride = down ? c.d : c.f;
        }
        if (withShared) {
            const uint32_t *o = &L.sharedOff.gateWOff;
            BlockKind &k = a.kind[0];
            if (!setup_kind(mode, false, 0, redo, Lm, L.shared + (down ? o[6] : o[0]), L.shared + o[3], down ? c.d : c.sharedF,
                            down ? c.sharedF : c.d, 1, (uint64_t)c.d * c.sharedF / 2,
                            L.sharedScales + (down ? (uint64_t)(c.sharedF / 8) * 16 * padded_groups(c.d / 64) : 0), 0, error))
                return false;
            k.in = down ? ctx->sharedActs : x;
            k.inStride = down ? c.sharedF : xStride;
            k.out = down ? sharedOut : ctx->sharedActs;
            k.outStride = down ? c.d : c.sharedF;
        }
        BlockMaps maps;
        memcpy(&maps, Lm.blockMap[mode], sizeof(maps));
        const bool ok = values && down ? launch_kernel<kDown, false, true>(ctx, redo, maps, "int4_block_down", stream, error)
                        : down ? launch_kernel<kDown, false>(ctx, redo, maps, "int4_block_down", stream, error)
                             : launch_kernel<kGateUp, false>(ctx, redo, maps, "int4_block_gate_up_act", stream, error);
        if (!ok) return false;
    }
    return true;
}

// The INT8 shared FFN of up to 16 rows.
bool launch_block_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens, uint16_t *y,
                       cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    LayerStore &Lm = const_cast<LayerStore &>(L);  // (its maps are encoded once per load)
    for (int mode = 0; mode < 2; ++mode) {
        RedoArgs redo{};
        BlockArgs &a = redo.a;
        a.T = (int)tokens;
        a.K = 1;
        a.perExpert = (int)tokens;
        a.withShared = 1;
        a.errorFlag = ctx->errorFlag;
        const bool down = mode == kDown;
        BlockKind &k = a.kind[0];
        if (!setup_kind(mode, true, 0, redo, Lm, L.shared8W[down ? 2 : 0], L.shared8W[1], down ? c.d : c.sharedF,
                        down ? c.sharedF : c.d, 1, (uint64_t)c.d * c.sharedF,
                        L.sharedScales + (down ? (uint64_t)(c.sharedF / 8) * 16 * padded_groups(c.d / 64) : 0), 0, error))
            return false;
        k.in = down ? ctx->sharedActs : x;
        k.inStride = down ? c.sharedF : xStride;
        k.out = down ? y : ctx->sharedActs;
        k.outStride = down ? c.d : c.sharedF;
        BlockMaps maps;
        memcpy(&maps, Lm.blockMap[mode], sizeof(maps));
        const bool ok = down ? launch_kernel<kDown, true>(ctx, redo, maps, "shared_int8_down", stream, error)
                             : launch_kernel<kGateUp, true>(ctx, redo, maps, "shared_int8_gate_up_act", stream, error);
        if (!ok) return false;
    }
    return true;
}

}  // namespace ff
