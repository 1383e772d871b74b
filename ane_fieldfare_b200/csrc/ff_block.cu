// Packed matrices against 1..16 input rows (a verify block): gate/up + GeGLU and down of the routed
// experts a block touches and of the shared FFN (INT4 or INT8), on the integer tensor cores straight
// on the codes (see ff_int_device.cuh).
//
// Work is cut into tasks: a tile of 16 weight rows (8 gate + 8 up, or 16 down rows) of one job — the
// shared FFN or an expert — against up to four of the job's input rows, which fill two MMAs' digit
// columns.  Every CTA makes the same plan from the route ids in shared memory (which routes chose each
// expert, in order; prefix sums of tasks) and takes one contiguous run of tasks, so it meets one or two
// experts, whose few input rows it stages as digits: a job's rows are staged where they are used, not
// all sixteen rows everywhere.  The CTA's warps deal the run's tiles round robin; a tile's rows come in
// parts along K as tensor copies into the warp's two slots, so one part is in flight while the other is
// multiplied, across tasks and experts.  All parts of a tile accumulate in the same registers, so no
// partial sums cross warps and results do not depend on scheduling.
//
// What bounds it: HBM for a block of many experts (16 rows, 48 experts: 170 MB), the staging of a job's
// rows and the last tasks of a run for few.  With codes turned into bf16 pairs, the integer pipe
// bounded it: gate/up 56 us and down 39 us for 16 rows.
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

constexpr int kMaxWarps = 12;
constexpr int kTaskRows = 4;          // input rows of a task
constexpr uint32_t kPartGroups = 12;  // groups of a part along K (INT8: 8), a multiple of four
constexpr uint32_t kPartGroups8 = 8;

enum Mode : int { kGateUp = 0, kDown = 1 };

// One kind of job: where its weight rows and scale words are (maps) and how its rows are laid out.
struct BlockKind {
    uint32_t tiles;       // tiles of 16 weight rows
    uint32_t groups;      // groups along K
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
};

struct alignas(64) BlockMaps {
    CUtensorMap w[2][2];  // [kind][gate, up] or [kind][down]
    CUtensorMap sb[2];
};

__device__ __forceinline__ void box3(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}

// Four groups of a tile against NT pairs of input rows.  lo / hi: this lane's packed bytes of tile rows g
// and g + 8 (INT4 8 bytes, INT8 16 per group), dig[j] its digits of pair j (columns 0..3 one row, 4..7
// the other), sb0 / sb1 the rows' scale words, aux[j] the groups of the row this lane accounts for (t < 2
// the pair's first, else its second).  acc[j][r]: r = 0 row g, 1 row g + 8, in units of 2^16 for the high
// digits (t even), whose lanes also take the bias part (biasUnit = 2^-16, else 0).  A group's scale and
// bias parts, which cancel in part, are joined before they are added up, and four groups before they
// join the running sum.
template <int NT, bool INT8>
__device__ __forceinline__ void four_groups(uint32_t lo, uint32_t hi, const uint32_t (&dig)[NT], uint32_t sb0, uint32_t sb1,
                                            const uint32_t (&aux)[NT], float biasUnit, float (&acc)[NT][2]) {
    constexpr uint32_t kStep = INT8 ? 64 : 32;
    uint4 a[4], b[4], x[NT][4], ax[NT][2];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (INT8) {
            a[u] = lds128(lo + kStep * u);
            b[u] = lds128(hi + kStep * u);
        } else {
            const uint2 p = lds64(lo + kStep * u), q = lds64(hi + kStep * u);
            a[u] = make_uint4(p.x & 0x0F0F0F0Fu, p.y & 0x0F0F0F0Fu, p.x & 0xF0F0F0F0u, p.y & 0xF0F0F0F0u);
            b[u] = make_uint4(q.x & 0x0F0F0F0Fu, q.y & 0x0F0F0F0Fu, q.x & 0xF0F0F0F0u, q.y & 0xF0F0F0F0u);
        }
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

template <int MODE, bool INT8>
__global__ void __launch_bounds__(kMaxWarps * 32, 1)
k_block_int(const BlockArgs a, const __grid_constant__ BlockMaps maps) {
    extern __shared__ __align__(128) uint8_t smemRaw[];
    __shared__ uint32_t sFirst[kMaxExperts + 2];  // first task of job j: 0 shared, 1 + e expert e
    __shared__ uint32_t sCount[kMaxExperts], sWarpSum[2][kMaxWarps];
    __shared__ __align__(8) uint64_t sBar[2 * kMaxWarps];
    uint8_t *sList = smemRaw + a.listOffset;  // [expert][16] route numbers (< 128)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (int)(blockDim.x >> 5);
    const int g = lane >> 2, t = lane & 3;
    const uint32_t smem = sm_addr(smemRaw);
    constexpr uint32_t kPart = INT8 ? kPartGroups8 : kPartGroups, kGroupBytes = INT8 ? 64 : 32;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * kMaxWarps; ++i) bar_init(sm_addr(&sBar[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // ---- the plan: routes of every expert in (token, rank) order, tasks per job ----
    const int routes = a.ids ? a.T * a.K : 0;
    for (int e = threadIdx.x; e < kMaxExperts; e += blockDim.x) sCount[e] = 0u;
    __syncthreads();
    if (warp < 4) {
        const int r = warp * 32 + lane;
        const uint32_t id = r < routes ? a.ids[r] : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, id), before = __popc(peers & ((1u << lane) - 1u));
        const bool known = id < (uint32_t)a.E;
        // A token's routes are distinct experts, so an expert is chosen by at most T routes; repeats
        // beyond that and routes past the resident experts keep their rows unwritten and raise the flag
        // (the reference refuses such a route with "route expert N is out of range").
        for (int w = 0; w < 4; ++w) {  // warps in turn: a route's place counts all earlier ones
            if (warp == w && r < routes) {
                const uint32_t place = known ? sCount[id] + before : 0u;
                if (known && place < (uint32_t)a.T) sList[id * kMaxGemvRows + place] = (uint8_t)r;
                else atomicExch(a.errorFlag, 12u);
            }
            __syncwarp();
            if (warp == w && r < routes && known && before == 0) sCount[id] = min(sCount[id] + (uint32_t)__popc(peers), (uint32_t)a.T);
            named_barrier(1, 128);
        }
    }
    __syncthreads();
    {
        // tasks of expert e = threadIdx.x (two passes cover 256 experts whatever the block size)
        uint32_t base = a.withShared ? a.kind[0].tiles * ((uint32_t)(a.T + kTaskRows - 1) / kTaskRows) : 0u, active = 0;
        if (threadIdx.x == 0) sFirst[0] = 0u;
        for (int e0 = 0; e0 < a.E; e0 += (int)blockDim.x) {
            const int e = e0 + (int)threadIdx.x;
            const uint32_t n = e < a.E ? sCount[e] : 0u;
            uint32_t tasks = a.kind[1].tiles * ((n + kTaskRows - 1) / kTaskRows), incl = tasks;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += v;
            }
            const uint32_t act = __popc(__ballot_sync(0xFFFFFFFFu, n > 0u));
            if (lane == 31) {
                sWarpSum[0][warp] = incl;
                sWarpSum[1][warp] = act;
            }
            __syncthreads();
            uint32_t earlier = base;
            for (int w = 0; w < warps; ++w) {
                if (w < warp) earlier += sWarpSum[0][w];
                base += sWarpSum[0][w];
                active += sWarpSum[1][w];
            }
            if (e < a.E) sFirst[1 + e] = earlier + incl - tasks;
            __syncthreads();
        }
        if (threadIdx.x == 0) sFirst[1 + a.E] = base;
        if (MODE == kGateUp && threadIdx.x == 0 && blockIdx.x == 0 && a.activeExperts) *a.activeExperts = active;
    }
    __syncthreads();
    const uint32_t total = sFirst[1 + a.E];
    const uint32_t first = (uint32_t)((uint64_t)blockIdx.x * total / gridDim.x),
                   last = (uint32_t)((uint64_t)(blockIdx.x + 1) * total / gridDim.x);
    if (first >= last) return;

    // A run of tasks that share their input rows: rows [4 * rowGroup, +4) of job `job`.
    struct Segment {
        uint32_t job, rowGroup, begin, end;
    };
    auto segment_of = [&](uint32_t task) {  // last job whose first task is not behind `task`
        uint32_t lo = 0, hi = (uint32_t)a.E + 1u;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sFirst[mid] <= task) lo = mid;
            else hi = mid;
        }
        const uint32_t tiles = a.kind[lo ? 1 : 0].tiles, rg = (task - sFirst[lo]) / tiles;
        return Segment{lo, rg, sFirst[lo] + rg * tiles, sFirst[lo] + (rg + 1u) * tiles};
    };
    auto rows_of = [&](const Segment &s) { return min(kTaskRows, (s.job ? (int)sCount[s.job - 1] : a.T) - (int)s.rowGroup * kTaskRows); };

    // ---- copies: this warp's steps (task, part) in order, two slots in turn ----
    const uint32_t slots = smem + a.slotsOffset + (uint32_t)warp * 2u * a.slotBytes;
    const uint32_t bars = sm_addr(&sBar[2 * warp]);
    uint32_t askTask = first + (uint32_t)warp, askPart = 0, asked = 0;
    Segment askSeg{0, 0, 0, 0};
    auto ask = [&]() {
        if (askTask >= last) return;
        if (askTask >= askSeg.end || askTask < askSeg.begin) askSeg = segment_of(askTask);
        const int kind = askSeg.job ? 1 : 0;
        const BlockKind &k = a.kind[kind];
        if (lane == 0) {
            const uint32_t slot = slots + (asked & 1u) * a.slotBytes, bar = bars + 8u * (asked & 1u);
            const int tile = (int)(askTask - askSeg.begin), z = askSeg.job ? (int)askSeg.job - 1 : 0;
            const int x = (int)(askPart * kPart * kGroupBytes / 8u);
            bar_expect(bar, 16u * k.pitch + 64u * k.sbWords);
            if (MODE == kGateUp) {
                box3(slot, &maps.w[kind][0], x, tile * 8, z, bar);
                box3(slot + 8u * k.pitch, &maps.w[kind][1], x, tile * 8, z, bar);
            } else {
                box3(slot, &maps.w[kind][0], x, tile * 16, z, bar);
            }
            box3(slot + a.sbOffset, &maps.sb[kind], (int)(askPart * kPart), tile * 16, z, bar);
        }
        ++asked;
        if (++askPart * kPart >= k.groups) {
            askPart = 0;
            askTask += (uint32_t)warps;
        }
    };
    ask();
    ask();

    const float biasUnit = (t & 1) ? 0.0f : 1.52587890625e-5f;  // 2^-16
    uint32_t used = 0;
    for (uint32_t at = first; at < last;) {
        const Segment seg = segment_of(at);
        const int kind = seg.job ? 1 : 0, n = rows_of(seg);
        const BlockKind &k = a.kind[kind];
        const uint32_t segEnd = min(seg.end, last);
        auto row_of = [&](int i) {  // row i of the segment: its route (routed) or token (shared)
            const int r = (int)seg.rowGroup * kTaskRows + i;
            return kind ? (int)sList[(seg.job - 1u) * kMaxGemvRows + (uint32_t)r] : r;
        };
        __syncthreads();  // the previous segment's digits are no longer read
        // ---- stage the rows as digits, two runs in flight per thread ----
        {
            const int runsPerRow = (int)k.groups * 8, runs = n * runsPerRow;
            auto fetch = [&](int i, bool ok) {
                if (!ok) return make_uint4(0, 0, 0, 0);
                const int r = i / runsPerRow;
                int row = row_of(r);
                if (MODE == kGateUp && kind) row /= a.K;  // a route's token
                return __ldcg(reinterpret_cast<const uint4 *>(k.in + (size_t)row * k.inStride) + (i - r * runsPerRow));
            };
            auto put = [&](int i, bool ok, const uint4 &v) {
                const int r = ok ? i / runsPerRow : 0, in = ok ? i - r * runsPerRow : 0;
                digits_put<INT8>(in, ok, v, smemRaw + a.digitsOffset + (size_t)r * a.rowBytes,
                                 reinterpret_cast<GroupAux *>(smemRaw + a.auxOffset + (size_t)r * a.auxRow) + (in >> 3));
            };
            for (int base = warp * 32; base < runs; base += 2 * (int)blockDim.x) {
                const int i = base + lane, j = i + (int)blockDim.x;
                const uint4 v = fetch(i, i < runs), w = fetch(j, j < runs);
                put(i, i < runs, v);
                if (base + (int)blockDim.x < runs) put(j, j < runs, w);  // the same for the whole warp
            }
            // groups past the row, up to a batch of four: nothing is added for them
            const int padded = ((int)k.groups + 3) & ~3;
            for (int i = threadIdx.x; i < n * 4; i += blockDim.x) {
                const int group = padded - 4 + (i & 3);
                if (group >= (int)k.groups)
                    *(reinterpret_cast<GroupAux *>(smemRaw + a.auxOffset + (size_t)(i >> 2) * a.auxRow) + group) = GroupAux{0.0f, 0.0f};
            }
        }
        __syncthreads();
        // ---- this warp's tiles of the segment ----
        const uint32_t phase = (at - first) % (uint32_t)warps;
        uint32_t task = at + ((uint32_t)warp + (uint32_t)warps - phase) % (uint32_t)warps;
        auto run_tiles = [&](auto pairs) {
            constexpr int NT = decltype(pairs)::value;
            for (; task < segEnd; task += (uint32_t)warps) {
                float acc[NT][2];
                uint32_t dig[NT], aux[NT];
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    acc[j][0] = acc[j][1] = 0.0f;
                    const int column = min(2 * j + (g >> 2), n - 1), mine = min(2 * j + (t >> 1), n - 1);
                    dig[j] = smem + a.digitsOffset + (uint32_t)column * a.rowBytes + (uint32_t)(g & 3) * 64u + (uint32_t)t * 16u;
                    aux[j] = smem + a.auxOffset + (uint32_t)mine * a.auxRow;
                }
                for (uint32_t p0 = 0; p0 < k.groups; p0 += kPart) {
                    const uint32_t slot = slots + (used & 1u) * a.slotBytes;
                    uint32_t parity = (used >> 1) & 1u;
                    slot_wait(bars + 8u * (used & 1u), parity, a.errorFlag);
                    uint32_t lo = slot + (uint32_t)g * k.pitch + (INT8 ? 16u : 8u) * t, hi = lo + 8u * k.pitch;
                    uint32_t sb0 = slot + a.sbOffset + (uint32_t)g * k.sbWords * 4u, sb1 = sb0 + 32u * k.sbWords;
                    const int batches = ((int)min(kPart, k.groups - p0) + 3) >> 2;
#pragma unroll 1
                    for (int b = 0; b < batches; ++b) {
                        four_groups<NT, INT8>(lo, hi, dig, sb0, sb1, aux, biasUnit, acc);
                        lo += 4u * kGroupBytes;
                        hi += 4u * kGroupBytes;
                        sb0 += 16u;
                        sb1 += 16u;
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            dig[j] += 4u * kDigitGroupBytes;
                            aux[j] += 32u;
                        }
                    }
                    slot_release();
                    ++used;
                    ask();
                }
                const uint32_t tile = task - seg.begin;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    // lane (g, t = 0): the pair's first row, t = 2: its second
                    const float r0 = fmaf(acc[j][0], 65536.0f, __shfl_xor_sync(0xFFFFFFFFu, acc[j][0], 1));
                    const float r1 = fmaf(acc[j][1], 65536.0f, __shfl_xor_sync(0xFFFFFFFFu, acc[j][1], 1));
                    const int mine = 2 * j + (t >> 1);
                    if ((t & 1) || mine >= n) continue;
                    uint16_t *dst = k.out + (size_t)row_of(mine) * k.outStride;
                    if (MODE == kGateUp) {
                        // the shared FFN rounds gate and up before the activation
                        const float gate = kind ? r0 : bf16_round(r0), up = kind ? r1 : bf16_round(r1);
                        dst[tile * 8u + (uint32_t)g] = f2bf(gelu_tanh(gate) * up);
                    } else {
                        dst[tile * 16u + (uint32_t)g] = f2bf(r0);
                        dst[tile * 16u + 8u + (uint32_t)g] = f2bf(r1);
                    }
                }
            }
        };
        if (n > 2) run_tiles(std::integral_constant<int, 2>{});
        else run_tiles(std::integral_constant<int, 1>{});
        at = segEnd;
    }
}

// ---- host ------------------------------------------------------------------------------------------

bool encode3(CUtensorMap *map, CUtensorMapDataType type, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1,
             uint64_t s2, uint32_t b0, uint32_t b1, const char **error) {
    EncodeTiledFn fn = encode_tiled(error);
    if (!fn) return false;
    const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {s1, s2};
    const cuuint32_t box[3] = {b0, b1, 1}, elem[3] = {1, 1, 1};
    const CUresult rc = fn(map, type, 3, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) return fail(error, "cuTensorMapEncodeTiled(block) failed: " + std::to_string((int)rc));
    return true;
}

// Slot row pitch of a kind: a part's bytes, padded so that a half-warp's reads fall on different banks
// (INT4 64-bit reads of four rows: 32 or 96 modulo 128; INT8 128-bit reads of two rows: 64).
uint32_t row_pitch(uint32_t groups, bool int8) {
    if (!int8) return piece_stride(std::min(groups, kPartGroups) * 32);
    uint32_t p = std::min(groups, kPartGroups8) * 64;
    while ((p & 127u) != 64u) p += 16;
    return p;
}

// Fills a kind and its maps.  mode kGateUp: w0, w1 [rows][cols], tiles of 8 + 8 rows; kDown: w0, 16 rows.
bool setup_kind(int mode, bool int8, BlockKind &k, CUtensorMap (&w)[2], CUtensorMap &sb, const uint8_t *w0, const uint8_t *w1,
                uint32_t rows, uint32_t cols, uint32_t experts, uint64_t stride, const uint32_t *scales, uint64_t scaleStride,
                const char **error) {
    const uint32_t groups = cols / 64, padded = padded_groups(groups), part = int8 ? kPartGroups8 : kPartGroups;
    const uint64_t rowBytes = int8 ? cols : cols / 2;
    k.tiles = mode == kGateUp ? rows / 8 : rows / 16;
    k.groups = groups;
    k.pitch = row_pitch(groups, int8);
    k.sbWords = std::min(padded, part);
    const uint8_t *ws[2] = {w0, w1};
    for (int m = 0; m < (mode == kGateUp ? 2 : 1); ++m)
        if (!encode3(&w[m], CU_TENSOR_MAP_DATA_TYPE_UINT64, ws[m], rowBytes / 8, rows, experts, rowBytes, stride, k.pitch / 8,
                     mode == kGateUp ? 8 : 16, error))
            return false;
    const uint64_t scaleRows = mode == kGateUp ? (uint64_t)rows * 2 : rows;
    return encode3(&sb, CU_TENSOR_MAP_DATA_TYPE_UINT32, scales, padded, scaleRows, experts, (uint64_t)padded * 4,
                   experts > 1 ? scaleStride * 4 : scaleRows * padded * 4, k.sbWords, 16, error);
}

template <int MODE, bool INT8>
bool launch_kernel(FFContext *ctx, BlockArgs a, const BlockMaps &maps, const char *name, cudaStream_t stream, const char **error) {
    uint32_t groups = 0, slot = 0, sb = 0;
    for (int i = 0; i < 2; ++i) {
        if (!a.kind[i].tiles) continue;
        groups = std::max(groups, a.kind[i].groups);
        slot = std::max(slot, 16 * a.kind[i].pitch);
        sb = std::max(sb, 64 * a.kind[i].sbWords);
    }
    auto up128 = [](uint32_t v) { return (v + 127u) & ~127u; };
    const uint32_t rows = (uint32_t)std::min(a.T, kTaskRows), padded = padded_groups(groups);
    a.listOffset = 0;
    a.digitsOffset = a.ids ? up128((uint32_t)a.E * kMaxGemvRows) : 0;
    a.rowBytes = padded * kDigitGroupBytes;
    a.auxOffset = a.digitsOffset + rows * a.rowBytes;
    a.auxRow = padded * (uint32_t)sizeof(GroupAux);
    a.slotsOffset = up128(a.auxOffset + rows * a.auxRow);
    a.sbOffset = up128(slot);
    a.slotBytes = a.sbOffset + up128(sb);
    const uint32_t limit = 227 * 1024 - 4096;  // less the static arrays
    // (a batch of four groups may read up to three groups past a slot's last row: within the scale area
    // or the next slot; behind the last slot a group's worth is kept)
    const uint32_t slack = 3 * 64 * 2;
    if (a.slotsOffset + 4 * 2 * a.slotBytes + slack > limit) return fail(error, "model shape too large for the block kernels' shared memory");
    const uint32_t warps = std::min<uint32_t>(kMaxWarps, (limit - slack - a.slotsOffset) / (2 * a.slotBytes));
    const size_t smem = a.slotsOffset + (size_t)warps * 2 * a.slotBytes + slack;
    static KernelSmemMemo memo;
    if (!memo.prepare(k_block_int<MODE, INT8>, ctx->device, 227 * 1024 - 4096, kMaxWarps * 32, nullptr, error)) return false;
    {
        LaunchScope scope(ctx, stream, name);
        k_block_int<MODE, INT8><<<ctx->smCount, warps * 32, smem, stream>>>(a, maps);
    }
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

}  // namespace

// Routed experts (ids [tokens][K], partial rows to `partials`) and / or the INT4 shared FFN (rows to
// `sharedOut`) of up to 16 rows.
bool launch_block_int4(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                       const uint32_t *ids, bool withShared, uint16_t *partials, uint16_t *sharedOut, cudaStream_t stream,
                       const char **error) {
    const FFConfig &c = ctx->cfg;
    if (c.d % 64 || c.f % 64 || c.sharedF % 64) return fail(error, "widths must be multiples of 64");
    if (((uintptr_t)x & 15) || (xStride % 8)) return fail(error, "input rows must be 16-byte aligned");
    const uint64_t words = scale_words(c.d, c.f);
    for (int mode = 0; mode < 2; ++mode) {
        BlockArgs a{};
        BlockMaps maps;
        memset(&maps, 0, sizeof(maps));
        a.ids = ids;
        a.T = (int)tokens;
        a.K = (int)c.topK;
        a.E = ids ? (int)L.expertCount : 0;
        a.withShared = withShared;
        a.activeExperts = &ctx->plan->activeExperts;
        a.errorFlag = ctx->errorFlag;
        const bool down = mode == kDown;
        if (ids) {
            const uint32_t *o = &L.off.gateWOff;
            BlockKind &k = a.kind[1];
            if (!setup_kind(mode, false, k, maps.w[1], maps.sb[1], L.experts + (down ? o[6] : o[0]), L.experts + o[3], down ? c.d : c.f,
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
            if (!setup_kind(mode, false, k, maps.w[0], maps.sb[0], L.shared + (down ? o[6] : o[0]), L.shared + o[3], down ? c.d : c.sharedF,
                            down ? c.sharedF : c.d, 1, (uint64_t)c.d * c.sharedF / 2,
                            L.sharedScales + (down ? (uint64_t)(c.sharedF / 8) * 16 * padded_groups(c.d / 64) : 0), 0, error))
                return false;
            k.in = down ? ctx->sharedActs : x;
            k.inStride = down ? c.sharedF : xStride;
            k.out = down ? sharedOut : ctx->sharedActs;
            k.outStride = down ? c.d : c.sharedF;
        }
        const bool ok = down ? launch_kernel<kDown, false>(ctx, a, maps, "int4_block_down", stream, error)
                             : launch_kernel<kGateUp, false>(ctx, a, maps, "int4_block_gate_up_act", stream, error);
        if (!ok) return false;
    }
    return true;
}

// The INT8 shared FFN of up to 16 rows.
bool launch_block_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens, uint16_t *y,
                       cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    for (int mode = 0; mode < 2; ++mode) {
        BlockArgs a{};
        BlockMaps maps;
        memset(&maps, 0, sizeof(maps));
        a.T = (int)tokens;
        a.K = 1;
        a.withShared = 1;
        a.errorFlag = ctx->errorFlag;
        const bool down = mode == kDown;
        BlockKind &k = a.kind[0];
        if (!setup_kind(mode, true, k, maps.w[0], maps.sb[0], L.shared8W[down ? 2 : 0], L.shared8W[1], down ? c.d : c.sharedF,
                        down ? c.sharedF : c.d, 1, (uint64_t)c.d * c.sharedF,
                        L.sharedScales + (down ? (uint64_t)(c.sharedF / 8) * 16 * padded_groups(c.d / 64) : 0), 0, error))
            return false;
        k.in = down ? ctx->sharedActs : x;
        k.inStride = down ? c.sharedF : xStride;
        k.out = down ? y : ctx->sharedActs;
        k.outStride = down ? c.d : c.sharedF;
        const bool ok = down ? launch_kernel<kDown, true>(ctx, a, maps, "shared_int8_down", stream, error)
                             : launch_kernel<kGateUp, true>(ctx, a, maps, "shared_int8_gate_up_act", stream, error);
        if (!ok) return false;
    }
    return true;
}

}  // namespace ff
