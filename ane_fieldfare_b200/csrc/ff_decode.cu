// One token through the whole MoE block in ONE cooperative kernel: router, top-8, routed
// gate/up/GeGLU, shared FFN, routed down and the weighted combine.
//
// The step streams 37.5 MB of weights once; at B200's HBM rate that is under 6 us, so separate
// kernels (launch gaps, cold starts) cannot come near the roofline.  Here one CTA per SM runs
// three phases:
//   A  router logits (one warp per expert) and the shared gate/up/GeGLU rows; the shared down
//      rows are already requested;
//   B  every CTA ranks the 128 logits itself (top-8, softmax, gain), then routed gate/up/GeGLU
//      rows and the shared down rows; the routed down rows are requested as the warps finish;
//   C  routed down rows and the fixed-order combine onto the shared output (or the caller's
//      residual).
// Values cross from CTA to CTA as tagged 64-bit words that the readers poll (logits, shared activations,
// routed activations, shared output rows): value and validity in one L2 round trip, nothing is cleared.
// Tile counters beside them are hints when it is worth polling a long row; they order nothing.
//
// Weight rows reach the SM as asynchronous copies (completion counted on a per-warp mbarrier) into a
// per-warp shared-memory slot: cp.async.bulk.tensor over row-box maps of the layer (one request brings 8
// or 16 row pieces of one matrix), cp.async.bulk for a tile's scale | bias words.
//
// Row arithmetic runs on the integer tensor cores straight on the codes (ff_int_device.cuh): a warp task
// is a tile of 16 weight rows, two runs of eight — gate and up rows of the same features, sixteen rows
// of the shared down projection, or the same eight output rows of two routed experts, whose
// activations then fill the eight digit columns of the MMA.  Long rows are split along K between the
// warps of a pair (quad, triple) of one CTA and added in a fixed order, the experts' down rows in rank
// order, so results do not depend on scheduling.
//
// What bounds a step: the chain router row -> logits through L2 -> routes -> routed rows from HBM (3.8
// us for 19.5 MB) -> activations through L2 -> down rows: 15.7 us a step in a graph (2396 GB/s).
//
// Cooperative launch guarantees that all CTAs are resident.  Every spin (tagged words, hints, copy
// completion) is bounded: on running out it raises the context's error flag and carries on, so the
// launch always ends.  Shapes past one CTA's shared memory take launch_decode_general.
//
// Reference kernels replaced (paths inside the reference project):
//   Sources/ANEFieldfareHotpath/Metal/MoE/moe.metal:65-120,242-319,500-517,548-570,597-638
//   Sources/ANEFieldfareHotpath/Metal/Quant/dequant_int4.metal:78-169
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <string>

#include "ff_int_device.cuh"

namespace ff {

constexpr int kFusedThreads = 512;
constexpr int kFusedWarps = kFusedThreads / 32;
constexpr int kBigWarps = 10;      // warps 0..9: gate/up pairs and the routed down tiles
constexpr int kSharedGuWarps = 8;  // warps 0..7 take the shared gate/up tiles in phase A (K quarters)
constexpr int kRouterWarps = 2;    // warps 8, 9 the router rows
constexpr int kRouterChunks = 12;  // 16-byte pieces of a router row a lane holds: 3072 inputs
constexpr int kRankWarp = 9;       // polls the logits
static_assert(kRankWarp < kBigWarps && 8 <= kBigWarps, "warps 0..9 rank");
constexpr uint32_t kBarrierSpinLimit = 1u << 24;
constexpr uint32_t kHintSpinLimit = 1u << 12;

struct DecodeArgs {
    const uint16_t *routerW, *routerScale, *gain;
    const float *logitBias;
    const uint32_t *scales;       // routed scale | bias words, scaleStride words per expert (see pack_scales)
    uint64_t scaleStride;
    const uint32_t *sharedScales;
    const uint8_t *shared;  // null: no shared FFN, `residual` is added instead
    const uint16_t *x;
    const uint16_t *residual;
    const uint32_t *idsIn;  // non-null: routes are given, the router is skipped
    const uint16_t *weightsIn;
    // Values handed from CTA to CTA travel as 64-bit words (launch tag << 32 | payload) that the
    // readers poll: a word is valid when its tag is the running launch's, so nothing is cleared.
    unsigned long long *taggedLogits;  // [CTA / 4][kMaxExperts] payload: the logit's bits
    unsigned long long *taggedActs;    // [K * F / 2] payload: two routed activations (bf16)
    unsigned long long *taggedH1;      // [D / 2] payload: two rows of the shared FFN's output (bf16)
    unsigned long long *taggedShared;  // [Fs / 2] payload: two shared activations (bf16)
    uint32_t *ids;
    uint16_t *weights;
    uint16_t *y;
    unsigned long long *barrier;  // ticket and hand-off counters
    uint32_t *hints;              // [kHintSets][2]: finished shared and routed gate/up tiles
    uint32_t *errorFlag;
    unsigned long long *stamps;  // null, or the phase / per-warp timestamp slots (ns)
    int E, D, F, Fs, K;          // K = 0: shared FFN only (y receives its output)
    int expertCount;             // resident experts of the layer: routes at or past it are refused
    // host hand-off (null when unused): the last CTA to finish copies y to `hostY` (host memory the
    // device can write), then stores (error flag << 32 | epoch) to `mailbox`, which the host polls
    uint16_t *hostY;
    unsigned long long *mailbox;
    uint32_t epoch;
    // shared-memory carve-up (fused_layout)
    uint32_t regionOffset, regionAux, actsAux, partialOffset, downOffset, slotsOffset, rowsBytes, pairBytes, tripleBytes, downBytes;
    uint32_t strideGU, strideGUA, strideSD, strideRD;
};

// Row-box tensor maps of the layer (kernel parameters): routed gate, routed up, shared gate, shared
// up, shared down, routed down.  A tile's eight (sixteen) row pieces arrive as one tensor copy per matrix.
struct alignas(64) DecodeMaps {
    CUtensorMap m[kDecodeMaps];
};
enum : int { kMapRoutedGate = 0, kMapRoutedUp = 1, kMapSharedGate = 2, kMapSharedUp = 3, kMapSharedDown = 4, kMapRoutedDown = 5 };

// Fetches a tensor map's descriptor ahead of its first use (the first copy through a map otherwise
// waits for it).
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Values cross CTAs as tagged words only.  Two 64-bit counters that only grow go with them: at its
// start every CTA draws a ticket from counter [3]; ticket / gridDim is the launch's generation (launches
// on a context are serialised, so all CTAs of a launch get the same one), and the generation gives the
// launch's 32-bit tag (never 0, different for consecutive launches).  [2] counts finished CTAs for the
// host hand-off.  No reset, no host-side state.
// Polling all of a row's words from every CTA would fill L2's bandwidth and hold up the stores it
// waits for, so tile counters say when it is worth looking: four sets used in turn, the one of the
// launch after next cleared by CTA 0.  They are hints, not ordered with the words; the words' tags
// decide.
enum : int { kCountDone = 2, kCountTicket = 3, kHintSets = 4 };
__device__ __forceinline__ void hint_add(uint32_t *hint) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(hint) : "memory");
}
// By one thread, bounded (the words behind the hint are waited for in any case).
__device__ __forceinline__ void hint_wait(const uint32_t *hint, uint32_t count) {
    uint32_t v = 0;
    for (uint32_t spins = 0; spins < kHintSpinLimit && v < count; ++spins)
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(hint) : "memory");
}

__device__ __forceinline__ void named_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// The thread that waits for the CTA: lane 0 of the last warp.
__device__ __forceinline__ bool is_waiting_thread() { return threadIdx.x == blockDim.x - 32; }

__device__ __forceinline__ void st_tagged(unsigned long long *p, uint32_t tag, uint32_t payload) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)tag << 32) | payload) : "memory");
}
__device__ __forceinline__ unsigned long long ld_tagged(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void stamp(const DecodeArgs &a, int slot) {
    if (a.stamps && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        a.stamps[slot] = t;
    }
}

// Per-warp timestamps of two CTAs (first and last) when tracing: slot 8 + ((cta01 * 3 + phase) * 16 +
// warp) * 3 + which, which = 0 requests issued, 1 data arrived, 2 rows done.
__device__ __forceinline__ void warp_stamp(const DecodeArgs &a, int phase, int which) {
    if (a.stamps && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1) && (threadIdx.x & 31) == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        const int c = blockIdx.x == 0 ? 0 : 1;
        a.stamps[8 + ((c * 3 + phase) * 16 + (threadIdx.x >> 5)) * 3 + which] = t;
    }
}

// Rows of bf16 values as digits (flat run index over all rows) by `threads` threads, this one number
// `tid`; fetch(i, j, v, w) reads runs i and j (negative: none).  Rows of `groups` groups have their aux
// entries `auxGroups` apart (0: one row).  No barrier at the end.
template <typename Fetch>
__device__ __forceinline__ void stage_digits(int runs, int tid, int threads, uint8_t *digits, GroupAux *aux, int groups, int auxGroups, Fetch fetch) {
    auto auxOf = [&](int run) {
        const int group = run >> 3;
        return aux + (auxGroups ? group / groups * auxGroups + group % groups : group);
    };
    // two runs in flight
    for (int base = tid & ~31; base < runs; base += 2 * threads) {
        const int i = base + (tid & 31), j = i + threads;
        uint4 v = make_uint4(0, 0, 0, 0), w = make_uint4(0, 0, 0, 0);
        fetch(i < runs ? i : -1, j < runs ? j : -1, v, w);
        digits_put(i, i < runs, v, digits, auxOf(i));
        if (base + threads < runs) digits_put(j, j < runs, w, digits, auxOf(j));  // the same for the whole warp
    }
}
// Runs of eight values that other CTAs are still writing as four tagged words each, polled (bounded);
// i, j < 0: none.
__device__ __forceinline__ void fetch_tagged(const unsigned long long *src, uint32_t tag, int i, int j, uint4 &v, uint4 &w,
                                             uint32_t *errorFlag) {
    auto one = [&](int r, uint4 &out) {
        const unsigned long long *p = src + 4 * (size_t)r;
        unsigned long long w0, w1, w2, w3;
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w0), "=l"(w1) : "l"(p) : "memory");
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w2), "=l"(w3) : "l"(p + 2) : "memory");
        out = make_uint4((uint32_t)w0, (uint32_t)w1, (uint32_t)w2, (uint32_t)w3);
        return (uint32_t)(w0 >> 32) == tag && (uint32_t)(w1 >> 32) == tag && (uint32_t)(w2 >> 32) == tag && (uint32_t)(w3 >> 32) == tag;
    };
    bool okI = i < 0, okJ = j < 0;
    for (uint32_t spins = 0; spins < kBarrierSpinLimit && !(okI && okJ); ++spins) {
        const bool askI = !okI, askJ = !okJ;
        if (askI) okI = one(i, v);
        if (askJ) okJ = one(j, w);
    }
    if (!(okI && okJ)) atomicExch(errorFlag, 9u);
}

// The K largest logits, by warps 0..9: one of them polls the CTA's copy of the tagged words and puts
// their keys into shared memory (0: never taken — -inf or NaN, or past the experts); then two threads
// per expert count the larger keys, half of them each.  Equal keys leave a place empty; then the count
// is repeated with the lower id first.  (Dependent instructions cost here, one warp waits 5 cycles for
// each: taking the maximum eight times cost 2 us, a rolled count with the tie rule in it 1.3 us.)
// sKey: two halves of kKeyHalf words.  Ends with a barrier of the ten warps.
constexpr uint32_t kNoRoute = 0xFFFFFFFFu;
constexpr int kKeyHalf = kMaxExperts / 2 + 4;  // (+4: the halves' 128-bit reads fall on different banks)
__device__ __forceinline__ void poll_and_rank(const DecodeArgs &a, uint32_t tag, uint32_t *sKey, uint32_t *sIds, float *sScore) {
    const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int half = ((a.E + 1) / 2 + 15) & ~15;  // keys of a half, a multiple of sixteen
    if (warp == kRankWarp) {
        const unsigned long long *words = a.taggedLogits + (size_t)(blockIdx.x >> 2) * kMaxExperts;
        for (int base = 0; base < 2 * half; base += 64) {
            const int e = base + 2 * lane;  // (both words in one half)
            if (e >= 2 * half) break;
            unsigned long long w[2] = {0, 0};
            bool ok = false;
            for (uint32_t spins = 0; spins < kBarrierSpinLimit && !ok; ++spins) {
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w[0]), "=l"(w[1]) : "l"(words + e) : "memory");
                ok = (e >= a.E || (uint32_t)(w[0] >> 32) == tag) && (e + 1 >= a.E || (uint32_t)(w[1] >> 32) == tag);
            }
            if (!ok) atomicExch(a.errorFlag, 9u);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float v = __uint_as_float((uint32_t)w[i]);
                sKey[(e >= half ? kKeyHalf + e - half : e) + i] = e + i < a.E && v > -INFINITY ? ordered_key(v) : 0u;
            }
        }
    }
    if (tid < 8) {
        sIds[tid] = kNoRoute;
        sScore[tid] = -INFINITY;
    }
    named_barrier(9, kBigWarps * 32);
    auto key_of = [&](int e) { return e < a.E ? sKey[e >= half ? kKeyHalf + e - half : e] : 0u; };
    auto place = [&](int e, uint32_t key, int rank) {
        if (key && rank < a.K) {
            sIds[rank] = (uint32_t)e;
            sScore[rank] = __uint_as_float((key >> 31) ? (key & 0x7FFFFFFFu) : ~key);
        }
    };
    for (int base = 0; base < a.E && tid < 256; base += 128) {
        const int e = base + (tid >> 1), h = tid & 1;
        const uint32_t mine = key_of(e);
        int n[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int o = 0; o < half; o += 16) {
            uint4 k[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) k[i] = *reinterpret_cast<const uint4 *>(sKey + h * kKeyHalf + o + 4 * i);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                n[0] += k[i].x > mine ? 1 : 0;
                n[1] += k[i].y > mine ? 1 : 0;
                n[2] += k[i].z > mine ? 1 : 0;
                n[3] += k[i].w > mine ? 1 : 0;
            }
        }
        int rank = (n[0] + n[1]) + (n[2] + n[3]);
        rank += __shfl_xor_sync(0xFFFFFFFFu, rank, 1);
        if (h == 0) place(e, mine, rank);
    }
    named_barrier(9, kBigWarps * 32);
    bool empty = false;
    for (int r = 0; r < a.K; ++r) empty |= sIds[r] == kNoRoute;
    if (empty) {  // the same for the ten warps
        named_barrier(9, kBigWarps * 32);
        if (tid < 8) sIds[tid] = 0u;  // what stays without a route: expert 0, weight 0
        named_barrier(9, kBigWarps * 32);
        for (int e = tid; e < a.E; e += kBigWarps * 32) {
            const uint32_t mine = key_of(e);
            int rank = 0;
            for (int o = 0; o < a.E; ++o) rank += key_of(o) >= mine + (o < e ? 0u : 1u) ? 1 : 0;
            place(e, mine, rank);
        }
        named_barrier(9, kBigWarps * 32);
    }
}

// The input row travelling inside the kernel's parameters (no host-to-device copy before the
// launch): up to 4096 bf16 values.
struct InlineRow {
    uint4 v[512];
};

// xInline: null, or the input row in parameter space (read with plain loads).
__device__ __forceinline__ void decode_body(const DecodeArgs &a, const DecodeMaps &maps, const uint16_t *xInline) {
    extern __shared__ __align__(128) uint8_t smemRaw[];
    __shared__ uint32_t sIds[8];
    __shared__ __align__(16) uint32_t sKey[2 * kKeyHalf];
    __shared__ float sWeights[8], sScore[8];
    __shared__ __align__(8) uint64_t sCopyBar[kFusedWarps];
    __shared__ uint32_t *sHints;            // this launch's tile counters
    __shared__ uint32_t sTag;               // the launch's tag for polled words, from the generation

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = (int)gridDim.x, cta = (int)blockIdx.x;
    const int D = a.D, F = a.F, Fs = a.Fs, K = a.K, E = a.E;
    const int g = lane >> 2, t = lane & 3;
    const int groupsD = D >> 6, groupsF = F >> 6, groupsFs = Fs >> 6;
    const int auxGroups = (groupsF + 1) & ~1;  // a routed row's aux groups, 16-byte aligned

    // shared memory: x as digits | its group sums | the shared activations as digits | their group sums; over
    // these, once phase B is done, the routed activations as digits | their group sums || K-split partial sums |
    // routed down rows per expert | slots: five pairs (two tile parts, the tile's scales), two triples of the
    // other six warps.  The fifth pair has no tile in phase A: its slot holds x as fp32 for the router until then.
    const uint32_t smem = sm_addr(smemRaw);
    uint8_t *region = smemRaw + a.regionOffset;
    GroupAux *regionAux = reinterpret_cast<GroupAux *>(smemRaw + a.regionAux);
    GroupAux *actsAux = reinterpret_cast<GroupAux *>(smemRaw + a.actsAux);
    const uint32_t x32Offset = a.slotsOffset + (kSharedGuWarps / 2) * a.pairBytes;
    const bool routing = !a.idsIn && K > 0;
    GroupAux *xAux = reinterpret_cast<GroupAux *>(smemRaw + D * 4);
    float *partial = reinterpret_cast<float *>(smemRaw + a.partialOffset);  // [warp][16]
    float *downRows = reinterpret_cast<float *>(smemRaw + a.downOffset);    // [row tile][expert][8]
    const int pair = warp >> 1;
    const int triple = warp >= kBigWarps ? (warp - kBigWarps) / 3 : 0;
    const int part3 = warp >= kBigWarps ? (warp - kBigWarps) % 3 : 0;
    const uint32_t tripleBase = smem + a.slotsOffset + (kBigWarps / 2) * a.pairBytes + (uint32_t)triple * a.tripleBytes;
    const uint32_t slot = warp < kBigWarps ? smem + a.slotsOffset + (uint32_t)pair * a.pairBytes + (uint32_t)(warp & 1) * a.rowsBytes
                                            : tripleBase + (uint32_t)part3 * 16u * a.strideSD;
    const uint32_t downSlot = warp < kBigWarps ? slot : tripleBase + (uint32_t)part3 * a.downBytes;
    auto scalesOfPair = [&](int p) { return smem + a.slotsOffset + (uint32_t)p * a.pairBytes + 2u * a.rowsBytes; };
    auto barOf = [&](int w) { return sm_addr(&sCopyBar[w]); };
    const uint32_t myBar = barOf(warp);
    uint32_t parity = 0;

    if (threadIdx.x == 0) {
        for (int w = 0; w < kFusedWarps; ++w) bar_init(barOf(w), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp >= 10 && lane == 0) prefetch_tensormap(&maps.m[warp - 10]);  // warps 10..15: the six maps
    // the ticket: drawn now by a thread with nothing to request (warp 9), published to the CTA
    // further down so that nobody waits for the atomic's round trip here
    unsigned long long ticket = 0;
    if (threadIdx.x == 9 * 32) ticket = atomicAdd(a.barrier + kCountTicket, 1ull);
    // this thread's share of the input row is requested before anything else
    const bool xPlain = xInline != nullptr;
    const uint16_t *xSrc = xPlain ? xInline : a.x;
    auto fetchX = [&](int i) {  // plain loads for a row in the kernel's parameters
        return xPlain ? reinterpret_cast<const uint4 *>(xSrc)[i] : __ldcg(reinterpret_cast<const uint4 *>(xSrc) + i);
    };
    // Router rows: warps 8, 9 take one expert each and hold its row in registers, 3072 inputs at a time
    // (through shared memory the row's loads waited for the barriers' set-up, and the chain for the loads).
    const int rw = warp - kSharedGuWarps, chunksD = D >> 3;
    int eA = (routing && rw >= 0 && rw < kRouterWarps) ? rw * G + cta : 0x7FFFFFFF;
    uint4 wr[kRouterChunks];
    auto load_router = [&](int first) {
        const uint4 *row = reinterpret_cast<const uint4 *>(a.routerW + (size_t)eA * D);
#pragma unroll
        for (int i = 0; i < kRouterChunks; ++i) {
            const int c = first + 32 * i + lane;
            wr[i] = c < chunksD ? __ldcs(row + c) : make_uint4(0, 0, 0, 0);
        }
    };
    if (eA < E) load_router(0);
    uint4 xMine = make_uint4(0, 0, 0, 0);
    if ((int)threadIdx.x < (D >> 3)) xMine = fetchX((int)threadIdx.x);
    __syncthreads();
    stamp(a, 0);

    const uint8_t *sh = a.shared;
    const int tilesSGU = sh ? Fs >> 3 : 0;  // 8 gate + 8 up rows per tile, four K quarters
    const int tilesSD = sh ? D >> 4 : 0;    // 16 down rows per tile, three K parts

    // Requests of part `part` of `parts` (along K) of a gate/up tile: one box of eight row pieces per
    // matrix (`pitch` bytes per row in the slot: the box is as wide as the pitch, what it reads past
    // the part is not used); with the first part the tile's scale | bias words over the full K to `sb`.
    const uint32_t wordsGU = 16u * padded_groups((uint32_t)groupsD), wordsSD = 16u * padded_groups((uint32_t)groupsFs),
                   wordsRD = 8u * padded_groups((uint32_t)groupsF);
    auto issue_gate_up = [&](const CUtensorMap *gateMap, const CUtensorMap *upMap, int expert, const uint32_t *words, int tile,
                             int part, int parts, uint32_t pitch, uint32_t sb) {
        int gb, ge;
        even_range(groupsD, parts, part, gb, ge);
        if (lane == 0) {
            bar_expect(myBar, (ge > gb ? 16u * pitch : 0u) + (part == 0 ? 4u * wordsGU : 0u));
            if (ge > gb) {
                tma_load_3d(slot, gateMap, gb * 4, tile * 8, expert, myBar);
                tma_load_3d(slot + 8u * pitch, upMap, gb * 4, tile * 8, expert, myBar);
            }
            if (part == 0) bulk_copy(sb, words + (size_t)tile * wordsGU, 4u * wordsGU, myBar);
        }
        __syncwarp();
    };
    // A gate/up tile's part: lane (g, t = 0) gets gate row g and up row g.
    auto gate_up = [&](int part, int parts, uint32_t pitch, uint32_t sb) {
        int gb, ge;
        even_range(groupsD, parts, part, gb, ge);
        const uint32_t s = sb + 4u * ((uint32_t)g * padded_groups((uint32_t)groupsD) + (uint32_t)gb);
        return tile_int4<false>(slot + (uint32_t)g * pitch + 8u * t, slot + (uint32_t)(g + 8) * pitch + 8u * t,
                                smem + (uint32_t)gb * kDigitGroupBytes + (uint32_t)(g & 3) * 64u + (uint32_t)t * 16u, s, s + 2u * wordsGU,
                                sm_addr(xAux) + 8u * (uint32_t)gb, ge - gb);
    };
    auto issue_shared_down = [&](int tile, int part) {
        int gb, ge;
        even_range(groupsFs, 3, part, gb, ge);
        if (lane == 0) {
            bar_expect(myBar, (ge > gb ? 16u * a.strideSD : 0u) + (part == 0 ? 4u * wordsSD : 0u));
            if (ge > gb) tma_load_3d(slot, &maps.m[kMapSharedDown], gb * 4, tile * 16, 0, myBar);
            if (part == 0) bulk_copy(tripleBase + 48u * a.strideSD, a.sharedScales + (Fs >> 3) * wordsGU + (size_t)tile * wordsSD, 4u * wordsSD, myBar);
        }
        __syncwarp();
    };
    // A warp's copies and, for the scales, those of the first warp of its pair, quad or triple.  (All
    // warps of a group take the same number of tiles, so one parity serves both barriers.)
    auto wait_tile = [&](int first) {
        if (warp != first) {
            uint32_t p = parity;
            slot_wait(barOf(first), p, a.errorFlag);
        }
        slot_wait(myBar, parity, a.errorFlag);
    };

    // ---------------- phase A: router logits, shared gate/up/GeGLU ----------------
    // shared gate/up tiles: four warps per tile (K quarters), two tiles per CTA and round
    const int partA = warp & 3;
    int tA = warp < kSharedGuWarps ? (warp >> 2) * G + cta : 0x7FFFFFFF;
    auto issue_shared_gate_up = [&](int tile) {
        issue_gate_up(&maps.m[kMapSharedGate], &maps.m[kMapSharedUp], 0, a.sharedScales, tile, partA, 4, a.strideGUA,
                      scalesOfPair((warp & ~3) >> 1));
    };
    if (tA < tilesSGU) issue_shared_gate_up(tA);
    int tSD = warp >= kBigWarps ? triple * G + cta : 0x7FFFFFFF;
    if (tSD < tilesSD) issue_shared_down(tSD, part3);
    warp_stamp(a, 0, 0);
    if (threadIdx.x == 9 * 32) {
        const unsigned long long generation = ticket / gridDim.x;
        sTag = (uint32_t)((generation + 1ull) % 0xFFFFFFFFull) + 1u;  // 1 .. 2^32-1: never 0, consecutive launches differ
        sHints = a.hints + 2 * (generation % kHintSets);
        if (cta == 0) *reinterpret_cast<uint2 *>(a.hints + 2 * ((generation + 2) % kHintSets)) = make_uint2(0u, 0u);
    }
    // the input row, as digits and (for the router) as it is
    stage_digits(D >> 3, (int)threadIdx.x, kFusedThreads, smemRaw, xAux, groupsD, 0, [&](int i, int j, uint4 &v, uint4 &w) {
        // as fp32 [step of 32 runs][half][lane] for the router's chains
        float4 *x32 = reinterpret_cast<float4 *>(smemRaw + x32Offset);
        auto keep = [&](int r, const uint4 &q) {
            if (!routing) return;
            const uint32_t qq[4] = {q.x, q.y, q.z, q.w};
            float f[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                f[2 * k] = __uint_as_float(qq[k] << 16);
                f[2 * k + 1] = __uint_as_float(qq[k] & 0xFFFF0000u);
            }
            if (a.routerScale) {  // times the router's per-input scales
                const uint4 sv = __ldg(reinterpret_cast<const uint4 *>(a.routerScale) + r);
                const uint32_t ss[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    f[2 * k] = f[2 * k] * __uint_as_float(ss[k] << 16);
                    f[2 * k + 1] = f[2 * k + 1] * __uint_as_float(ss[k] & 0xFFFF0000u);
                }
            }
            x32[2 * r - (r & 31)] = make_float4(f[0], f[1], f[2], f[3]);
            x32[2 * r - (r & 31) + 32] = make_float4(f[4], f[5], f[6], f[7]);
        };
        if (i >= 0) keep(i, v = i == (int)threadIdx.x ? xMine : fetchX(i));
        if (j >= 0) keep(j, w = fetchX(j));
    });
    __syncthreads();  // the tag is published, too
    const uint32_t tag = sTag;
    for (; tA < tilesSGU; tA += (kSharedGuWarps / 4) * G) {
        wait_tile(warp & ~3);
        warp_stamp(a, 0, 1);
        const float2 v = gate_up(partA, 4, a.strideGUA, scalesOfPair((warp & ~3) >> 1));
        float *mine = partial + warp * 16;
        if (partA && t == 0) {
            mine[g] = v.x;
            mine[8 + g] = v.y;
        }
        named_barrier(1 + (warp >> 2), 128);  // every part is read, too: the slots are free
        const int next = tA + (kSharedGuWarps / 4) * G;
        if (next < tilesSGU) issue_shared_gate_up(next);
        if (!partA) {
            const float *m = mine + g;
            const float gate = ((v.x + m[16]) + m[32]) + m[48], up = ((v.y + m[24]) + m[40]) + m[56];
            // two activations of a tile per tagged word, the odd neighbour's by shuffle
            const uint32_t act = f2bf(gelu_tanh(bf16_round(gate)) * bf16_round(up));
            const uint32_t two = act | (__shfl_down_sync(0xFFFFFFFFu, act, 4) << 16);
            if (t == 0 && !(g & 1)) st_tagged(a.taggedShared + ((tA * 8 + g) >> 1), tag, two);
            if (lane == 0) hint_add(sHints);
        }
        named_barrier(1 + (warp >> 2), 128);
    }
    while (eA < E) {
        const float biasE = a.logitBias ? __ldg(a.logitBias + eA) : 0.0f;
        // lane l chains fmaf over elements [256 i + 8 l, +8): the order of every router kernel.  (Chunks
        // past the row are skipped: a lane's last step may not exist.)
        float acc = 0.0f;
        for (int first = 0; first < chunksD; first += 32 * kRouterChunks) {
            if (first) load_router(first);
#pragma unroll
            for (int i = 0; i < kRouterChunks; ++i) {
                const int c = first + 32 * i + lane;
                if (c < chunksD) {
                    const uint32_t at = smem + x32Offset + 16u * (uint32_t)(2 * c - lane);
                    const uint4 lo = lds128(at), hi = lds128(at + 512u);
                    const uint32_t xx[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                    const uint32_t ww[4] = {wr[i].x, wr[i].y, wr[i].z, wr[i].w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        acc = fmaf(__uint_as_float(ww[k] << 16), __uint_as_float(xx[2 * k]), acc);
                        acc = fmaf(__uint_as_float(ww[k] & 0xFFFF0000u), __uint_as_float(xx[2 * k + 1]), acc);
                    }
                }
            }
        }
#pragma unroll
        for (int offset = 16; offset >= 1; offset >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, offset);
        // Value and validity in one 64-bit store, a copy for every four CTAs: the readers poll their own
        // copies (all CTAs' polls on eight lines held the stores up for microseconds).
        const float logit = a.logitBias ? acc + biasE : acc;
        for (int c = lane; c < (G + 3) / 4; c += 32) st_tagged(a.taggedLogits + (size_t)c * kMaxExperts + eA, tag, __float_as_uint(logit));
        eA += kRouterWarps * G;
        if (eA < E) load_router(0);
    }
    // The fifth pair's first copies, behind the ranking's barriers, overwrite x as fp32.  (By the warp that mostly has
    // no router row, hence no stores in flight that the fence would wait for.)
    if (routing && warp == kRankWarp) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    warp_stamp(a, 0, 2);
    stamp(a, 1);

    // ---------------- top-8 ----------------
    const int tilesF = F >> 3;
    const int tilesRouted = K * tilesF;
    int tB = warp < kBigWarps ? pair * G + cta : 0x7FFFFFFF;
    int kB = 0x7FFFFFFF;  // route and tile inside its expert, ready before the routes are
    int tileB = 0;
    auto place = [&](int tile) {
        kB = tile / tilesF;
        tileB = tile - kB * tilesF;
    };
    if (tB < tilesRouted) place(tB);
    if (K > 0 && warp < kBigWarps) {
        if (!a.idsIn) {
            poll_and_rank(a, tag, sKey, sIds, sScore);
        } else {
            // Given routes.  A route past the resident experts would address memory outside the layer:
            // it is replaced by expert 0 with weight 0 and reported through the error flag (the
            // reference refuses such a route with "route expert N is out of range").
            if ((int)threadIdx.x < K) {
                uint32_t id = a.idsIn[threadIdx.x];
                float w = bf2f(a.weightsIn[threadIdx.x]);
                if (id >= (uint32_t)a.expertCount) {
                    atomicExch(a.errorFlag, 12u);
                    id = 0u;
                    w = 0.0f;
                }
                sIds[threadIdx.x] = id;
                sWeights[threadIdx.x] = w;
            }
            named_barrier(9, kBigWarps * 32);
        }
        named_arrive(10, kFusedThreads);  // for the warps of the shared down rows
    }
    stamp(a, 2);
    stamp(a, 3);
    auto issue_routed_gate_up = [&]() {
        issue_gate_up(&maps.m[kMapRoutedGate], &maps.m[kMapRoutedUp], (int)sIds[kB], a.scales + (size_t)sIds[kB] * a.scaleStride, tileB,
                      warp & 1, 2, a.strideGU, scalesOfPair(pair));
    };
    if (tB < tilesRouted) issue_routed_gate_up();
    if (warp < kBigWarps) warp_stamp(a, 1, 0);
    if (routing && warp == kSharedGuWarps) {
        // softmax over the chosen scores: exponentials in parallel, the sum in rank order
        const float myScore = lane < K ? sScore[lane] : -INFINITY;
        const float top = __shfl_sync(0xFFFFFFFFu, myScore, 0);
        const float ex = lane < K ? expf(myScore - top) : 0.0f;
        float sum = 0.0f;
        for (int r = 0; r < K; ++r) sum += __shfl_sync(0xFFFFFFFFu, ex, r);
        if (lane < K) {
            const uint32_t myId = sIds[lane];
            float w = ex / sum;
            if (a.gain) w = w * bf2f(a.gain[myId]);
            const uint16_t wb = f2bf(w);
            sWeights[lane] = bf2f(wb);  // read in phase C
            if (blockIdx.x == 0) {
                a.ids[lane] = myId;
                a.weights[lane] = wb;
            }
        }
    }

    // ---------------- phase B: routed gate/up/GeGLU (warps 0..9), shared down rows (10..15) ----------
    // Routed down task j of a round (16 / pairsK row tiles of eight rows, pairsK expert pairs each), tasks
    // in the order of warps 10..15, 0..9: the shared down warps are done first.
    const int tilesRD = D >> 3, pairsK = (K + 1) >> 1, perRound = pairsK ? kFusedWarps / pairsK : 1;
    const int task = warp >= kBigWarps ? warp - kBigWarps : warp + (kFusedWarps - kBigWarps);
    const int myTile = pairsK ? task / pairsK : 0, myPair = pairsK ? task - myTile * pairsK : 0;
    const int eLo = 2 * myPair, eHi = min(2 * myPair + 1, K - 1);
    auto tileOf = [&](int round) { return cta + G * (round * perRound + myTile); };
    auto has_task = [&](int round) { return K > 0 && myTile < perRound && tileOf(round) < tilesRD; };
    auto issue_routed_down = [&](int tile) {
        // the two experts' rows (one box each) and scale words
        if (lane == 0) {
            bar_expect(myBar, 16u * a.strideRD + 8u * wordsRD);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t id = sIds[i ? eHi : eLo];
                tma_load_3d(downSlot + (uint32_t)i * 8u * a.strideRD, &maps.m[kMapRoutedDown], 0, tile * 8, (int)id, myBar);
                bulk_copy(downSlot + 16u * a.strideRD + (uint32_t)i * 4u * wordsRD,
                          a.scales + (size_t)id * a.scaleStride + (F >> 3) * wordsGU + (size_t)tile * wordsRD, 4u * wordsRD, myBar);
            }
        }
        __syncwarp();
    };
    if (warp >= kBigWarps && sh) {
        // the shared activations, staged by the six warps that use them
        if (is_waiting_thread()) hint_wait(sHints, (uint32_t)tilesSGU);
        named_barrier(8, (kFusedWarps - kBigWarps) * 32);
        stage_digits(Fs >> 3, (int)threadIdx.x - kBigWarps * 32, (kFusedWarps - kBigWarps) * 32, region, regionAux, groupsFs, 0,
                     [&](int i, int j, uint4 &v, uint4 &w) { fetch_tagged(a.taggedShared, tag, i, j, v, w, a.errorFlag); });
        named_barrier(8, (kFusedWarps - kBigWarps) * 32);
    }
    for (; tB < tilesRouted; tB += (kBigWarps / 2) * G) {
        wait_tile(warp & ~1);
        warp_stamp(a, 1, 1);
        const float2 v = gate_up(warp & 1, 2, a.strideGU, scalesOfPair(pair));
        float *mine = partial + warp * 16;
        if ((warp & 1) && t == 0) {
            mine[g] = v.x;
            mine[8 + g] = v.y;
        }
        named_barrier(1 + pair, 64);
        const int next = tB + (kBigWarps / 2) * G;
        if (next < tilesRouted) {
            place(next);
            issue_routed_gate_up();
        }
        if (!(warp & 1)) {
            // the tile's eight activations are one run of the staged row: four tagged words,
            // written by the lanes t == 0 of even g (the odd neighbour's value comes by shuffle)
            const float gate = v.x + mine[16 + g], up = v.y + mine[24 + g];
            const uint32_t act = f2bf(gelu_tanh(gate) * up);
            const uint32_t two = act | (__shfl_down_sync(0xFFFFFFFFu, act, 4) << 16);
            if (t == 0 && !(g & 1)) st_tagged(a.taggedActs + ((tB * 8 + g) >> 1), tag, two);
            if (lane == 0) hint_add(sHints + 1);
        }
        named_barrier(1 + pair, 64);
    }
    for (; tSD < tilesSD; tSD += 2 * G) {
        wait_tile(kBigWarps + 3 * triple);
        warp_stamp(a, 1, 1);
        int gb, ge;
        even_range(groupsFs, 3, part3, gb, ge);
        const uint32_t padded = padded_groups((uint32_t)groupsFs), s = tripleBase + 48u * a.strideSD + 4u * ((uint32_t)g * padded + (uint32_t)gb);
        const float2 v = tile_int4<false>(slot + (uint32_t)g * a.strideSD + 8u * t, slot + (uint32_t)(g + 8) * a.strideSD + 8u * t,
                                          sm_addr(region) + (uint32_t)gb * kDigitGroupBytes + (uint32_t)(g & 3) * 64u + (uint32_t)t * 16u, s,
                                          s + 32u * padded, sm_addr(regionAux) + 8u * (uint32_t)gb, ge - gb);
        float *mine = partial + warp * 16;
        if (part3 && t == 0) {
            mine[g] = v.x;
            mine[8 + g] = v.y;
        }
        named_barrier(6 + triple, 96);
        const int next = tSD + 2 * G;
        if (next < tilesSD) issue_shared_down(next, part3);
        if (!part3) {
            const float *m = mine + g;
            const uint32_t r0 = f2bf((v.x + m[16]) + m[32]), r1 = f2bf((v.y + m[24]) + m[40]);
            const int row = tSD * 16 + g;  // and row + 8
            if (K > 0) {
                // read as the residual of the routed rows in phase C: tagged words of two rows
                const uint32_t two0 = r0 | (__shfl_down_sync(0xFFFFFFFFu, r0, 4) << 16);
                const uint32_t two1 = r1 | (__shfl_down_sync(0xFFFFFFFFu, r1, 4) << 16);
                if (t == 0 && !(g & 1)) {
                    st_tagged(a.taggedH1 + (row >> 1), tag, two0);
                    st_tagged(a.taggedH1 + ((row + 8) >> 1), tag, two1);
                }
            } else if (t == 0) {
                a.y[row] = (uint16_t)r0;
                a.y[row + 8] = (uint16_t)r1;
            }
        }
        named_barrier(6 + triple, 96);
    }
    // warps 10..15 meet the routes only here: the shared down rows need none
    if (K > 0 && warp >= kBigWarps) named_barrier(10, kFusedThreads);
    if (has_task(0)) issue_routed_down(tileOf(0));
    warp_stamp(a, 1, 2);
    stamp(a, 4);
    if (K == 0) {
        stamp(a, 5);
        stamp(a, 6);
        return;
    }

    // No grid barrier before phase C: the routed activations and the shared output rows are polled
    // as tagged words while they are staged.
    warp_stamp(a, 2, 0);
    // (seven eighths: the last tiles' words are polled for, by the few threads that stage them)
    if (is_waiting_thread()) hint_wait(sHints + 1, (uint32_t)(tilesRouted - tilesRouted / 8));
    __syncthreads();  // the routed activations take the place of the rows that phase B's warps read
    stamp(a, 5);

    // ---------------- phase C: routed down rows and the combine ----------------
    // Warp w combines a round's row tile w, lane r its row r; the residual (two rows of the shared
    // output in a tagged word, or the caller's row) is asked for ahead of the activations.
    auto combine_tile = [&](int round) { return cta + G * (round * perRound + warp); };
    auto combines = [&](int round) { return warp < perRound && combine_tile(round) < tilesRD && lane < 8; };
    unsigned long long resWord = 0;
    float residual = 0.0f;
    auto ask_residual = [&](int round) {
        if (!combines(round)) return;
        const int row = combine_tile(round) * 8 + lane;
        if (a.shared) resWord = ld_tagged(a.taggedH1 + (row >> 1));
        else residual = a.residual ? bf2f(__ldcg(a.residual + row)) : 0.0f;
    };
    ask_residual(0);
    stage_digits(K * (F >> 3), (int)threadIdx.x, kFusedThreads, smemRaw, actsAux, groupsF, auxGroups,
                 [&](int i, int j, uint4 &v, uint4 &w) { fetch_tagged(a.taggedActs, tag, i, j, v, w, a.errorFlag); });
    __syncthreads();
    for (int round = 0; cta + G * round * perRound < tilesRD; ++round) {
        if (has_task(round)) {
            slot_wait(myBar, parity, a.errorFlag);
            warp_stamp(a, 2, 1);
            // rows 0..7 of the tile: expert eLo, columns 0..3; rows 8..15: expert eHi, columns 4..7
            const int mine = t < 2 ? eLo : eHi, column = g < 4 ? eLo : eHi;
            const uint32_t s = downSlot + 16u * a.strideRD + 4u * ((t < 2 ? 0u : wordsRD) + (uint32_t)g * padded_groups((uint32_t)groupsF));
            const float v = tile_int4<true>(downSlot + (uint32_t)g * a.strideRD + 8u * t, downSlot + (uint32_t)(g + 8) * a.strideRD + 8u * t,
                                            smem + (uint32_t)(column * groupsF) * kDigitGroupBytes + (uint32_t)(g & 3) * 64u + (uint32_t)t * 16u,
                                            s, s, sm_addr(actsAux) + 8u * (uint32_t)(mine * auxGroups), groupsF)
                                .x;
            if (!(t & 1) && (t == 0 || eHi > eLo)) downRows[(myTile * 8 + mine) * 8 + g] = v;
        }
        __syncthreads();
        if (has_task(round + 1)) issue_routed_down(tileOf(round + 1));
        if (combines(round)) {
            const int row = combine_tile(round) * 8 + lane;
            float acc = residual;
            if (a.shared) {
                uint32_t spins = 0;
                while ((uint32_t)(resWord >> 32) != tag) {
                    if (++spins > kBarrierSpinLimit) {
                        atomicExch(a.errorFlag, 9u);
                        break;
                    }
                    resWord = ld_tagged(a.taggedH1 + (row >> 1));
                }
                acc = bf2f((uint16_t)((lane & 1) ? (uint32_t)resWord >> 16 : (uint32_t)resWord & 0xFFFFu));
            }
            for (int k = 0; k < K; ++k) acc = __fadd_rn(acc, __fmul_rn(sWeights[k], downRows[(warp * 8 + k) * 8 + lane]));
            a.y[row] = f2bf(acc);
        }
        ask_residual(round + 1);
        __syncthreads();  // the rows are rewritten in the next round
    }
    warp_stamp(a, 2, 2);
    stamp(a, 6);

    // ---------------- host hand-off by the last CTA to finish ----------------
    if (a.mailbox) {
        __shared__ uint32_t sLast;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const unsigned long long old = atomicAdd(a.barrier + kCountDone, 1ull);
            sLast = (old % gridDim.x == gridDim.x - 1) ? 1u : 0u;
        }
        __syncthreads();
        if (sLast) {
            __threadfence();
            for (int i = threadIdx.x; i < (D >> 3); i += blockDim.x)
                reinterpret_cast<uint4 *>(a.hostY)[i] = __ldcg(reinterpret_cast<const uint4 *>(a.y) + i);
            // one system-scope release by one thread publishes the row (ordered before it by the CTA
            // barrier) together with the error flag and the epoch, as one 64-bit word
            __syncthreads();
            if (threadIdx.x == 0) {
                const unsigned long long word =
                    ((unsigned long long)__ldcg(a.errorFlag) << 32) | (unsigned long long)a.epoch;
                asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(a.mailbox), "l"(word) : "memory");
            }
        }
    }
}

__global__ void __launch_bounds__(kFusedThreads, 1)
k_decode_fused(const DecodeArgs a, const __grid_constant__ DecodeMaps maps) {
    decode_body(a, maps, nullptr);
}

__global__ void __launch_bounds__(kFusedThreads, 1)
k_decode_fused_inline_x(const DecodeArgs a, const __grid_constant__ DecodeMaps maps,
                        const __grid_constant__ InlineRow row) {
    decode_body(a, maps, reinterpret_cast<const uint16_t *>(&row));
}

// Scale | bias words of `count` blobs, tile by tile: [F/8 gate/up tiles][8 gate rows, 8 up rows] of
// padded_groups(D/64) words, then [D down rows] of padded_groups(F/64).
uint64_t scale_words_gate_up(uint32_t D, uint32_t F) { return (uint64_t)(F / 8) * 16 * padded_groups(D / 64); }
uint64_t scale_words(uint32_t D, uint32_t F) { return scale_words_gate_up(D, F) + (uint64_t)D * padded_groups(F / 64); }
__global__ void __launch_bounds__(256)
k_pack_scales(ScaleSource src, uint32_t D, uint32_t F, uint32_t *out, uint64_t words) {
    const uint32_t gD = D / 64, gF = F / 64, pD = padded_groups(gD), pF = padded_groups(gF);
    const uint64_t gateUp = (uint64_t)(F / 8) * 16 * pD;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t g, row, groups, matrix;
        if (i < gateUp) {
            const uint32_t r = (uint32_t)(i / pD), in = r & 15u;  // rows of a tile: 8 gate, 8 up
            g = (uint32_t)(i % pD);
            row = (r >> 4) * 8u + (in & 7u);
            groups = gD;
            matrix = in < 8u ? 0u : 1u;
        } else {
            g = (uint32_t)((i - gateUp) % pF);
            row = (uint32_t)((i - gateUp) / pF);  // down rows stay in order: tiles of any height are contiguous
            groups = gF;
            matrix = 2u;
        }
        uint32_t word = 0u;
        if (g < groups) {
            const size_t at = ((size_t)row * groups + g) * 2 + blockIdx.y * src.stride;
            word = (uint32_t)*reinterpret_cast<const uint16_t *>(src.scales[matrix] + at) |
                   ((uint32_t)*reinterpret_cast<const uint16_t *>(src.biases[matrix] + at) << 16);
        }
        out[blockIdx.y * words + i] = word;
    }
}
// Lays out `count` blobs' scales; *out is allocated when null (its size depends on the shape alone).
bool pack_scales(FFContext *ctx, const ScaleSource &src, uint32_t D, uint32_t F, uint32_t count,
                 uint32_t **out, const char **error) {
    const uint64_t words = scale_words(D, F);
    if (!*out) {
        FF_CUDA_OK(cudaMalloc(reinterpret_cast<void **>(out), words * count * 4), error);
        ctx->scratchBytes += words * count * 4;
    }
    k_pack_scales<<<dim3((unsigned)((words + 1023) / 1024), count), 256>>>(src, D, F, *out, words);
    FF_CUDA_OK(cudaGetLastError(), error);
    FF_CUDA_OK(cudaStreamSynchronize(nullptr), error);
    return true;
}

struct FusedLayout {
    uint32_t regionOffset, regionAux, actsAux, partialOffset, downOffset, slotsOffset, rowsBytes, pairBytes, tripleBytes, downBytes;
    uint32_t strideGU, strideGUA, strideSD, strideRD;
    size_t total;
};

static FusedLayout fused_layout(const FFConfig &c) {
    const uint32_t D = c.d, F = c.f, Fs = c.sharedF, K = c.topK;
    const uint32_t groupsD = D / 64, groupsF = F / 64, groupsFs = Fs / 64;
    auto up128 = [](uint32_t v) { return (v + 127u) & ~127u; };
    auto longest = [](uint32_t groups, int parts) {  // groups of the first (longest) part
        int begin, end;
        even_range((int)groups, parts, 0, begin, end);
        return (uint32_t)(end - begin);
    };
    FusedLayout l{};
    l.strideGU = piece_stride(longest(groupsD, 2) * 32);   // routed tiles: K halves
    l.strideGUA = piece_stride(longest(groupsD, 4) * 32);  // shared tiles: K quarters
    l.strideSD = Fs ? piece_stride(longest(groupsFs, 3) * 32) : 32;
    l.strideRD = piece_stride(groupsF * 32);
    // x and the shared activations, with their aux; in their place, later, K (even) rows of routed ones
    l.regionOffset = up128(D * 4 + groupsD * (uint32_t)sizeof(GroupAux));
    l.regionAux = l.regionOffset + Fs * 4;
    const uint32_t rows = (K + 1) / 2 * 2;
    l.actsAux = rows * F * 4;
    l.partialOffset = up128(std::max(l.regionAux + (uint32_t)sizeof(GroupAux) * (groupsFs + 2),
                                     l.actsAux + (uint32_t)sizeof(GroupAux) * (rows * ((groupsF + 1) & ~1u) + 2)));
    l.downOffset = l.partialOffset + kFusedWarps * 16 * 4;
    l.slotsOffset = up128(l.downOffset + kFusedWarps * 8 * 8 * 4);
    l.downBytes = up128(16 * l.strideRD + 64 * padded_groups(groupsF));
    l.rowsBytes = up128(std::max({16 * l.strideGU, 16 * l.strideGUA, l.downBytes}));
    l.pairBytes = up128(std::max(2 * l.rowsBytes + 64 * padded_groups(groupsD), (D + 255) / 256 * 1024));  // x as fp32, too
    l.tripleBytes = up128(std::max(Fs ? 48 * l.strideSD + 64 * padded_groups(groupsFs) : 0u, 3 * l.downBytes));
    l.total = (size_t)l.slotsOffset + (size_t)(kBigWarps / 2) * l.pairBytes + 2 * (size_t)l.tripleBytes;
    return l;
}

// Whether the fused kernel's shared memory (its static arrays included) and its row boxes hold the shape.
bool decode_fused_fits(const FFConfig &c) {
    static const size_t staticBytes = [] {
        size_t most = 0;
        cudaFuncAttributes f{};
        for (const void *k : {reinterpret_cast<const void *>(k_decode_fused), reinterpret_cast<const void *>(k_decode_fused_inline_x)})
            most = std::max(most, cudaFuncGetAttributes(&f, k) == cudaSuccess ? f.sharedSizeBytes : (size_t)4096);
        return most;
    }();
    const FusedLayout l = fused_layout(c);
    return l.total + staticBytes <= 227 * 1024 && std::max({l.strideGU, l.strideGUA, l.strideSD, l.strideRD}) <= 2048;
}

// y = bf16(residual + sum_k w_k v_k) of one row, in rank order as the fused kernel adds.
__global__ void __launch_bounds__(256)
k_combine_values(const float *values, const uint32_t *ids, const uint16_t *weights, const uint16_t *residual, int D, int K,
                 int expertCount, uint16_t *y) {
    pdl_enter();
    const int row = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (row >= D) return;
    float acc = residual ? bf2f(residual[row]) : 0.0f;
    for (int k = 0; k < K; ++k)  // (a route past the experts has no values: weight 0, as in the fused kernel)
        if (ids[k] < (uint32_t)expertCount) acc = __fadd_rn(acc, __fmul_rn(bf2f(weights[k]), values[(size_t)k * D + row]));
    y[row] = f2bf(acc);
}

// The same step as separate launches (router, block kernels with fp32 output rows, combine), for the shapes whose
// rows and slots are too large for one CTA's shared memory: 2880 x 1024 with a shared width of 2112, for instance.
static bool launch_decode_general(FFContext *ctx, const LayerStore &L, const uint16_t *x, const uint32_t *idsIn,
                                  const uint16_t *weightsIn, bool withShared, bool routed, const uint16_t *residual,
                                  uint16_t *y, cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (!routed) return launch_block_int4(ctx, L, x, c.d, 1, nullptr, true, nullptr, y, stream, error);
    if (!idsIn) {
        if (!launch_router_topk(ctx, L, x, c.d, 1, ctx->ids, ctx->weights, nullptr, stream, error)) return false;
        idsIn = ctx->ids;
        weightsIn = ctx->weights;
    }
    if (!launch_block_int4(ctx, L, x, c.d, 1, idsIn, withShared, nullptr, ctx->h1, stream, error, ctx->decodeValues)) return false;
    LaunchScope scope(ctx, stream, "combine_values");
    FF_CUDA_OK(launch_pdl(k_combine_values, (c.d + 255) / 256, 256, 0, stream, ctx->decodeValues, idsIn, weightsIn,
                          withShared ? ctx->h1 : residual, (int)c.d, (int)c.topK, (int)L.expertCount, y),
               error);
    return true;
}

// One decode row through router (unless ids are given), routed experts and the shared FFN (or
// the caller's residual), as one cooperative launch where the shape fits.  routed = false: the shared FFN alone, y
// receives its output.
bool launch_decode_fused(FFContext *ctx, const LayerStore &L, const uint16_t *x, const uint32_t *idsIn,
                         const uint16_t *weightsIn, bool withShared, bool routed, const uint16_t *residual,
                         uint16_t *y, cudaStream_t stream, const char **error, const DecodeHostHandoff *host) {
    const FFConfig &c = ctx->cfg;
    if (routed && !L.experts) return fail(error, "layer has no resident experts");
    if (routed && !idsIn && !L.has_router()) return fail(error, "layer has no resident router");
    if (routed && !idsIn && L.routerQ) {
        // The kernel's own router reads bf16 rows.  An INT8 router runs as its own launches in
        // front (logits, top-K), and the kernel takes the routes as given.
        if (host) return fail(error, "the host hand-off needs a bf16 router");
        if (L.routerExperts != L.expertCount) return fail(error, "router and layer disagree on the expert count");
        if (!launch_router_topk(ctx, L, x, ctx->cfg.d, 1, ctx->ids, ctx->weights, nullptr, stream, error))
            return false;
        idsIn = ctx->ids;
        weightsIn = ctx->weights;
    }
    if (withShared && !L.shared) return fail(error, "layer has no resident shared FFN");
    if (!routed && !withShared) return fail(error, "nothing to compute");
    if (c.topK > 8) return fail(error, "decode supports at most 8 routes");
    if (c.d % 64 || c.f % 64 || c.sharedF % 64) return fail(error, "widths must be multiples of 64");
    DecodeArgs a{};
    a.routerW = L.routerW;
    a.routerScale = L.routerScale;
    a.gain = L.gain;
    a.logitBias = L.logitBias;
    a.scales = L.routedScales;
    a.scaleStride = scale_words(c.d, c.f);
    a.sharedScales = L.sharedScales;
    a.shared = withShared ? L.shared : nullptr;
    a.x = x;
    a.residual = residual;
    a.idsIn = idsIn;
    a.weightsIn = weightsIn;
    a.taggedLogits = ctx->taggedLogits;
    a.taggedActs = ctx->taggedActs;
    a.taggedH1 = ctx->taggedActs + (size_t)c.topK * c.f / 2;
    a.taggedShared = a.taggedH1 + c.d / 2;
    a.ids = ctx->ids;
    a.weights = ctx->weights;
    a.y = y;
    a.barrier = reinterpret_cast<unsigned long long *>(ctx->gridBarrier);
    a.hints = ctx->gridBarrier + 16;
    a.errorFlag = ctx->errorFlag;
    a.stamps = ctx->tracing ? ctx->phaseStamps : nullptr;
    a.E = idsIn ? (int)L.expertCount : (int)L.routerExperts;
    a.expertCount = (int)L.expertCount;
    if (routed && !idsIn && L.routerExperts != L.expertCount)
        return fail(error, "router has " + std::to_string(L.routerExperts) + " experts, the layer " +
                               std::to_string(L.expertCount));
    a.D = (int)c.d;
    a.F = (int)c.f;
    a.Fs = withShared ? (int)c.sharedF : 0;
    a.K = routed ? (int)c.topK : 0;
    if (a.E > kMaxExperts) return fail(error, "too many experts for the decode kernel");
    const FusedLayout lay = fused_layout(c);
    const size_t smem = lay.total;
    // bulk copies need 16-byte aligned sources: every sub-tensor offset and the blob stride
    const uint32_t *ro = &L.off.gateWOff, *so = &L.sharedOff.gateWOff;
    for (int i = 0; i < 9; ++i)
        if ((routed && (ro[i] % 16 || L.stride % 16)) || (withShared && so[i] % 16))
            return fail(error, "sub-tensor offsets must be multiples of 16 bytes for the decode kernel");
    if (!(host && host->inlineX) && ((uintptr_t)x & 15) != 0) return fail(error, "input row must be 16-byte aligned");
    if (!decode_fused_fits(c)) {
        if (host) return fail(error, "the host hand-off needs the fused decode kernel");
        return launch_decode_general(ctx, L, x, idsIn, weightsIn, withShared, routed, residual, y, stream, error);
    }
    // row-box tensor maps of the layer, built once per loaded layer
    LayerStore &Lm = const_cast<LayerStore &>(L);
    if (!Lm.decodeMapsReady) {
        memset(Lm.decodeMap, 0, sizeof(Lm.decodeMap));
        if (L.experts) {
            const uint32_t *o = &L.off.gateWOff;
            for (int m = 0; m < 2; ++m)
                if (!make_row_box_map(&Lm.decodeMap[kMapRoutedGate + m], L.experts + o[3 * m], c.f, c.d / 2,
                                      L.expertCount, L.stride, lay.strideGU, 8, error))
                    return false;
            if (!make_row_box_map(&Lm.decodeMap[kMapRoutedDown], L.experts + o[6], c.d, c.f / 2, L.expertCount, L.stride,
                                  lay.strideRD, 8, error))
                return false;
        }
        if (L.shared && c.sharedF) {
            const uint32_t *o = &L.sharedOff.gateWOff;
            for (int m = 0; m < 2; ++m)
                if (!make_row_box_map(&Lm.decodeMap[kMapSharedGate + m], L.shared + o[3 * m], c.sharedF, c.d / 2, 1,
                                      0, lay.strideGUA, 8, error))
                    return false;
            if (!make_row_box_map(&Lm.decodeMap[kMapSharedDown], L.shared + o[6], c.d, c.sharedF / 2, 1, 0,
                                  lay.strideSD, 16, error))
                return false;
        }
        Lm.decodeMapsReady = true;
    }
    static thread_local DecodeMaps maps;
    memcpy(maps.m, L.decodeMap, sizeof(maps.m));
    a.regionOffset = lay.regionOffset;
    a.regionAux = lay.regionAux;
    a.actsAux = lay.actsAux;
    a.partialOffset = lay.partialOffset;
    a.downOffset = lay.downOffset;
    a.slotsOffset = lay.slotsOffset;
    a.rowsBytes = lay.rowsBytes;
    a.pairBytes = lay.pairBytes;
    a.tripleBytes = lay.tripleBytes;
    a.downBytes = lay.downBytes;
    a.strideGU = lay.strideGU;
    a.strideGUA = lay.strideGUA;
    a.strideSD = lay.strideSD;
    a.strideRD = lay.strideRD;
    static KernelSmemMemo memo, memoInline;
    int perSm = 0;
    if (!memo.prepare(k_decode_fused, ctx->device, smem, kFusedThreads, &perSm, error)) return false;
    if (perSm < 1) return fail(error, "fused decode kernel does not fit on an SM");
    if (!memoInline.prepare(k_decode_fused_inline_x, ctx->device, smem, kFusedThreads, &perSm, error)) return false;
    if (perSm < 1) return fail(error, "fused decode kernel does not fit on an SM");
    const int grid = ctx->smCount;
    if (host) {
        a.hostY = host->hostY;
        a.mailbox = host->mailbox;
        a.epoch = host->epoch;
    }
    LaunchScope scope(ctx, stream, "decode_fused");
    if (host && host->inlineX) {
        if (c.d > 4096) return fail(error, "input row too long to travel in the kernel parameters");
        static thread_local InlineRow row;
        memcpy(&row, host->inlineX, (size_t)c.d * 2);
        void *params[] = {&a, &maps, &row};
        FF_CUDA_OK(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_decode_fused_inline_x),
                                               dim3(grid), dim3(kFusedThreads), params, smem, stream),
                   error);
    } else {
        void *params[] = {&a, &maps};
        FF_CUDA_OK(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(k_decode_fused), dim3(grid),
                                               dim3(kFusedThreads), params, smem, stream),
                   error);
    }
    return true;
}

}  // namespace ff
