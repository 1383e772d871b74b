// Internal declarations shared by the translation units of libfieldfare_cuda.so.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <vector>

#include "fieldfare_cuda.h"

namespace ff {

constexpr int kGroup = 64;        // codes per scale/bias pair
constexpr int kMaxGemvRows = 16;  // input rows one GEMV job can carry (a verify block)
constexpr int kRouterCounts = 64;
// rows of one expert per unit of the prefill GEMM (accumulator columns): see routed_tile_rows and dense_tile_rows
constexpr uint32_t kRowTile = 192, kRowTileSmall = 128;
constexpr int kDecodeMaps = 6;
constexpr int kMaxExperts = 256;  // router width limit, as in the reference's prefill router

// ---- error plumbing ------------------------------------------------------------------------

// Stores a strdup'd message in *error (when the caller asked for one) and returns false.
bool fail(const char **error, const std::string &message);

#define FF_CUDA_OK(call, error)                                                              \
    do {                                                                                     \
        cudaError_t ff_status_ = (call);                                                     \
        if (ff_status_ != cudaSuccess)                                                       \
            return ff::fail(error, std::string(#call) + ": " + cudaGetErrorString(ff_status_)); \
    } while (0)

// Per-kernel memo of "dynamic shared-memory limit raised on this device" and of the occupancy at
// the last requested size.  The library's entry points may be called from one host thread per GPU
// (and context-free entry points from any thread), so the memo is guarded by a mutex.
constexpr int kMaxDevices = 64;
class KernelSmemMemo {
public:
    // Makes `kernel` launchable with `smem` bytes of dynamic shared memory on `device` and returns
    // the resident CTAs per SM at (threads, smem) in *perSm (when asked for).
    template <typename Kernel>
    bool prepare(Kernel kernel, int device, size_t smem, int threads, int *perSm, const char **error) {
        if (device < 0 || device >= kMaxDevices) return fail(error, "device ordinal out of range");
        std::lock_guard<std::mutex> guard(lock_);
        Entry &e = entries_[device];
        if (e.limit < smem || !e.touched) {
            FF_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), error);
            e.limit = smem;
            e.touched = true;
        }
        if (perSm) {
            if (e.occSmem != smem || e.occThreads != threads) {
                int n = 0;
                FF_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem), error);
                e.occ = n;
                e.occSmem = smem;
                e.occThreads = threads;
            }
            *perSm = e.occ;
        }
        return true;
    }

private:
    struct Entry {
        size_t limit = 0, occSmem = 0;
        int occ = 0, occThreads = -1;
        bool touched = false;
    };
    std::mutex lock_;
    Entry entries_[kMaxDevices];
};

// ---- work descriptions the kernels read ----------------------------------------------------

// One affine INT4 matrix (or a gate/up pair sharing inputs) applied to up to 16 input rows.
struct GemvJob {
    const uint8_t *w0;   // gate (or the only) matrix: packed codes
    const uint16_t *s0;  // scales
    const uint16_t *b0;  // biases
    const uint8_t *w1;   // up matrix (dual jobs only)
    const uint16_t *s1;
    const uint16_t *b1;
    const uint16_t *in;  // bf16 input rows
    uint16_t *out;       // bf16 output rows
    uint32_t rows;       // weight rows = outputs per input row
    uint32_t cols;       // weight columns = input width
    uint32_t inStride;   // elements between input rows
    uint32_t outStride;  // elements between output rows
    uint32_t n;          // input rows used, 1..16
    uint32_t flags;      // kJobRoundGateUp
    uint32_t inRow[kMaxGemvRows];
    uint32_t outRow[kMaxGemvRows];
};
constexpr uint32_t kJobRoundGateUp = 1u;  // round gate and up to bf16 before the activation

// What a decode/verify block reports.
struct RoutePlan {
    uint32_t activeExperts;  // distinct routed experts in the block
    uint32_t pad[3];
};

// How far an exact logit (without its bias) can be from its approximation on the tensor cores: perNorm |x| + floor,
// for rows of |x| < limit (see ff_router.cu).
struct RouterBound {
    float perNorm, floor, limit;
};

struct LayerStore {
    uint8_t *experts = nullptr;  // expertCount blobs, stride apart (a layer file, verbatim)
    uint64_t stride = 0;
    uint32_t expertCount = 0;
    FFExpertOffsets off{};
    uint8_t *shared = nullptr;  // gate, up, down of the shared FFN in the same nine-part order
    FFExpertOffsets sharedOff{};
    uint32_t *routedScales = nullptr, *sharedScales = nullptr;  // scale | bias words, tile by tile (pack_scales)
    uint16_t *routerW = nullptr;
    uint16_t *routerScale = nullptr;
    uint16_t *gain = nullptr;
    float *logitBias = nullptr;
    uint32_t routerExperts = 0;
    // INT8 affine router (the shipped checkpoints' form): codes [experts][d], one bf16 scale and
    // bias per group of 64 inputs; set instead of routerW
    uint8_t *routerQ = nullptr;
    uint16_t *routerQScale = nullptr, *routerQBias = nullptr;
    // for a prefill chunk's routes: the weights as the tensor cores multiply them (null: routerW), and a
    // bound of each approximate logit's error
    uint16_t *routerFolded = nullptr;
    RouterBound *routerBounds = nullptr;
    uint16_t *routerLanes = nullptr;  // INT8 router rows in lane order, and their scales | biases
    uint32_t *routerAux = nullptr;
    bool has_router() const { return routerW != nullptr || routerQ != nullptr; }
    // INT8 affine shared FFN (the shipped checkpoints' form): gate, up [sharedF][d] and down
    // [d][sharedF] as codes with one bf16 scale and bias per group of 64; set instead of `shared`
    uint8_t *shared8W[3] = {nullptr, nullptr, nullptr};
    uint16_t *shared8S[3] = {nullptr, nullptr, nullptr}, *shared8B[3] = {nullptr, nullptr, nullptr};
    bool has_shared8() const { return shared8W[0] != nullptr; }
    bool has_shared() const { return shared != nullptr || has_shared8(); }
    // prefill: tensor maps over the packed weights (gate, up, down) of routed and shared blobs
    bool mapsReady = false;
    CUtensorMap routedMap[3];
    CUtensorMap sharedMap[3];
    // one-token kernel: row-box maps of routed gate, routed up, shared gate, shared up, shared down,
    // routed down
    bool decodeMapsReady = false;
    CUtensorMap decodeMap[kDecodeMaps];
    // verify block: [gate/up, down][shared, routed] maps of the weights and scale words
    uint32_t blockMapsReady = 0;  // bit 2 * mode + kind
    CUtensorMap blockMap[2][2][3];
};

}  // namespace ff

constexpr int kPhaseStampSlots = 8 + 2 * 3 * 16 * 3;

struct FFContext {
    int device = 0;
    int smCount = 0;
    FFConfig cfg{};
    std::vector<ff::LayerStore> layers;
    cudaStream_t hostStream = nullptr;  // used by the *_host entry points

    // decode / verify scratch
    float *logits = nullptr;        // [min(maxTokens,16)][experts]
    float *logitsRows = nullptr;    // [maxTokens][experts], allocated with the first INT8 router
    uint32_t *ids = nullptr;        // [maxTokens][topK]
    uint16_t *weights = nullptr;    // [maxTokens][topK]
    ff::RoutePlan *plan = nullptr;
    uint32_t *routerCounts = nullptr;  // [kRouterCounts] CTAs that have formed the logits of a row (a block) or of a tile of rows
    uint16_t *acts = nullptr;       // [maxTokens*topK][f]
    uint16_t *sharedActs = nullptr; // [maxTokens][sharedF]
    uint16_t *h1 = nullptr;         // [maxTokens][d]
    uint16_t *partials = nullptr;   // [maxTokens*topK][d]
    float *decodeValues = nullptr;  // [topK][d] one row's routed outputs, where the shape does not fit the fused decode kernel
    uint16_t *xDev = nullptr;       // [maxTokens][d] staging for *_host
    uint16_t *yDev = nullptr;

    // prefill scratch (allocated when maxTokens > 16)
    uint16_t *xSorted = nullptr;            // [maxTokens*topK][d] rows in expert order
    uint32_t *rowOfRoute = nullptr;         // [maxTokens*topK] row of a token's route in that order
    uint16_t *xShared = nullptr;            // [maxTokens][d] rows for the shared FFN's GEMM
    // The shared FFN of a prefill block runs on a stream of its own beside the router and the sort, whose
    // kernels leave most SMs idle: forked off and joined within the call.
    cudaStream_t sideStream = nullptr;
    cudaEvent_t forked = nullptr, joined = nullptr;
    FFTokenExpertPair *sortedPairs = nullptr;
    uint32_t *expertOffsets = nullptr;      // [experts+1]
    uint32_t *blockCounts = nullptr;        // permute: [blocks][experts]
    uint32_t *units = nullptr;              // GEMM work units
    uint32_t *unitCount = nullptr;          // [4]
    uint32_t maxUnits = 0;
    float *routerParts = nullptr;           // approximate logits of a prefill chunk
    uint16_t *xSums = nullptr, *actSums = nullptr;  // group sums of the INT8 shared FFN's GEMM
    uint32_t *errorFlag = nullptr;          // device: set by a kernel that gave up waiting
    unsigned long long *phaseStamps = nullptr;  // device: 8 phase + 288 per-warp timestamps of the fused decode kernel
    unsigned long long *taggedLogits = nullptr;  // device: [SMs][kMaxExperts] router logits of the fused decode kernel
    unsigned long long *taggedActs = nullptr;    // device: [topK * f / 2 + d / 2 + sharedF / 2] routed activations, shared output rows, shared activations, as polled words
    uint32_t *gridBarrier = nullptr;        // device: counters of the fused decode kernel (eight 64-bit, then eight 32-bit)
    volatile unsigned long long *mailbox = nullptr;  // pinned host word the decode kernel reports to
    uint32_t hostEpoch = 0;

    // tracing: CUDA events around every kernel launch, aggregated per kernel name
    bool tracing = false;
    struct TraceRecord {
        const char *name;
        cudaEvent_t begin, end;
    };
    std::vector<TraceRecord> trace;

    // counters
    uint64_t kernelLaunches = 0;
    uint64_t weightBytes = 0;
    uint64_t scratchBytes = 0;
    uint32_t lastTokens = 0;
};

namespace ff {

// Counts a kernel launch and, when tracing is on, brackets it with CUDA events on its stream.
struct LaunchScope {
    FFContext *ctx;
    cudaStream_t stream;
    cudaEvent_t begin = nullptr, end = nullptr;
    const char *name;
    LaunchScope(FFContext *c, cudaStream_t s, const char *n) : ctx(c), stream(s), name(n) {
        ctx->kernelLaunches++;
        if (ctx->tracing) {
            cudaEventCreate(&begin);
            cudaEventCreate(&end);
            cudaEventRecord(begin, stream);
        }
    }
    ~LaunchScope() {
        if (begin) {
            cudaEventRecord(end, stream);
            ctx->trace.push_back({name, begin, end});
        }
    }
};

// Programmatic dependent launch: a kernel launched with launch_pdl may start while its predecessor on the
// stream still runs.  Every thread calls pdl_wait before it reads what the predecessor writes or writes
// anything the predecessor (or one before it) may still read; it returns when the predecessor is
// complete.  pdl_trigger, after pdl_wait, lets the successor start: what the successor does in front of
// its own pdl_wait may then use everything from before this kernel.  Saves the 2 us between kernels.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
    pdl_wait();
    pdl_trigger();
}
template <typename... Params, typename... Args>
cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args) {
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// ff_gemv.cu
bool launch_router_topk(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                        uint32_t tokens, uint32_t *ids, uint16_t *weights, float *logits,
                        cudaStream_t stream, const char **error);
bool launch_block_small(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                        uint32_t tokens, const uint32_t *ids, const uint16_t *weights,
                        bool withShared, bool decodeCombine, const uint16_t *residual,
                        uint16_t *partials, uint16_t *sharedOut, uint16_t *y,
                        cudaStream_t stream, const char **error);
bool launch_reduce(FFContext *ctx, const uint16_t *partials, const uint16_t *weights,
                   const uint16_t *residual, uint16_t *y, uint32_t tokens, cudaStream_t stream,
                   const char **error, const uint32_t *rowIndex = nullptr);
bool launch_gemv_rows(FFContext *ctx, const FFProjection &p, const uint16_t *x, uint32_t xStride,
                      uint32_t rows, uint16_t *y, uint32_t yStride, cudaStream_t stream,
                      const char **error);
bool launch_shared_small(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                         uint32_t tokens, uint16_t *y, cudaStream_t stream, const char **error);
bool launch_rmsnorm(FFContext *ctx, const uint16_t *x, const uint16_t *w, float eps,
                    uint32_t tokens, uint16_t *y, cudaStream_t stream, const char **error);
bool launch_dequant_probe(FFContext *ctx, const uint8_t *w, const uint16_t *s, const uint16_t *b,
                          uint32_t rows, uint32_t cols, float *out32, uint16_t *out16,
                          cudaStream_t stream, const char **error);

// ff_decode.cu
uint64_t scale_words(uint32_t D, uint32_t F);          // words of one blob
uint64_t scale_words_gate_up(uint32_t D, uint32_t F);  // of those, in front of the down rows
// Scales and biases of gate, up and down (bytes, blobs `stride` apart).
struct ScaleSource {
    const uint8_t *scales[3], *biases[3];
    uint64_t stride;
};
bool pack_scales(FFContext *ctx, const ScaleSource &src, uint32_t D, uint32_t F, uint32_t count, uint32_t **out, const char **error);
bool make_row_box_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t rowBytes, uint64_t experts,
                      uint64_t expertStride, uint32_t boxBytes, uint32_t boxRows, const char **error);

// ff_block.cu
bool launch_block_int4(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                       const uint32_t *ids, bool withShared, uint16_t *partials, uint16_t *sharedOut, cudaStream_t stream,
                       const char **error, float *values = nullptr);
bool launch_block_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens, uint16_t *y,
                       cudaStream_t stream, const char **error);

// Host hand-off of the one-token kernel: `inlineX` (host memory) travels in the kernel parameters
// instead of `x`; the last CTA copies the output to `hostY` (host memory mapped for the device) and
// stores (error flag << 32 | epoch) to the mailbox word.
struct DecodeHostHandoff {
    const uint16_t *inlineX;
    uint16_t *hostY;
    unsigned long long *mailbox;
    uint32_t epoch;
};
bool decode_fused_fits(const FFConfig &c);  // else launch_decode_fused takes the general kernels (no host hand-off)
bool launch_decode_fused(FFContext *ctx, const LayerStore &L, const uint16_t *x, const uint32_t *idsIn,
                         const uint16_t *weightsIn, bool withShared, bool routed, const uint16_t *residual,
                         uint16_t *y, cudaStream_t stream, const char **error,
                         const DecodeHostHandoff *host = nullptr);

// ff_prefill.cu
bool prefill_prepare_layer(FFContext *ctx, LayerStore &L, const char **error);
bool launch_prefill_routed(FFContext *ctx, LayerStore &L, const uint16_t *x, uint32_t xStride,
                           uint32_t tokens, const uint32_t *ids, uint16_t *partials,
                           cudaStream_t stream, const char **error);
bool launch_prefill_shared(FFContext *ctx, LayerStore &L, const uint16_t *x, uint32_t xStride,
                           uint32_t tokens, uint16_t *y, cudaStream_t stream, const char **error);
bool launch_post_attn_setup(FFContext *ctx, uint16_t *hidden, const uint16_t *attn, const uint16_t *wPostAttn,
                            const uint16_t *wPreFfn, const uint16_t *wPreFfn2, float eps, uint32_t tokens,
                            uint16_t *denseX, uint16_t *routedX, uint16_t *routerX, cudaStream_t stream,
                            const char **error);
bool launch_layer_tail(FFContext *ctx, const uint16_t *h2, const uint16_t *h1, uint16_t *hidden,
                       const uint16_t *wPostFfn2, const uint16_t *wPostFfn, float eps, float layerScalar,
                       uint32_t tokens, cudaStream_t stream, const char **error);
bool launch_shared_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                        uint16_t *y, cudaStream_t stream, const char **error);
bool launch_route_sort(FFContext *ctx, const uint32_t *groupIds, uint32_t tokens, uint32_t groups,
                       FFTokenExpertPair *sortedPairs, uint32_t *offsets, cudaStream_t stream, const char **error);
bool launch_router_prefill(FFContext *ctx, const LayerStore &L, const uint16_t *x,
                           uint32_t xStride, uint32_t tokens, uint32_t *ids, uint16_t *weights,
                           float *logits, cudaStream_t stream, const char **error);

// ff_router.cu
size_t router_parts_rows(size_t maxTokens, int smCount);
bool router_prepare(FFContext *ctx, LayerStore &L, const char **error);
bool launch_router_select(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                          uint32_t *ids, uint16_t *weights, cudaStream_t stream, const char **error);

// Where a logits kernel's last CTA per row puts the row's top-K (ids null: logits only; at most
// kMaxGemvRows rows).
struct RouterTail {
    uint32_t *ids;
    uint16_t *weights;
    const uint16_t *gain;
    uint32_t *counts;  // [kMaxGemvRows], zero between launches
    int K;
};
bool launch_router_logits_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                               float *logits, const RouterTail &tail, cudaStream_t stream, const char **error);

// ff_int8_gemm.cu
bool int8_gemm_fits(uint32_t d, uint32_t f);  // contraction lengths within the kernel's shared memory
bool launch_shared_int8_gemm(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                             uint16_t *y, cudaStream_t stream, const char **error);
bool alloc_int8_gemm(FFContext *ctx, const char **error);

// nine offsets for a blob holding gate/up [f][d] and down [d][f]
FFExpertOffsets packed_offsets(uint32_t d, uint32_t f, uint64_t *payload);

}  // namespace ff
