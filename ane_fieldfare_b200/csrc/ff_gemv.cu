// Bandwidth kernels of the INT4 MoE block: router rows, INT4 GEMV of one matrix or a gate/up pair for
// 1..16 token rows, decode combine, token-major reduce, RMSNorm and the fused steps either side of the
// block, and the dequantization probe.
//
// GEMV scheme (every matrix, every row count): a weight row of `cols` 4-bit codes is cut into
// 16-byte chunks of 32 codes.  Eight lanes share a row; lane j takes chunks j, j+8, j+16, ...
// with one 128-bit load each, unpacks the codes in registers, and for every input row
// accumulates  acc = fma(scale, sum(q*x), acc); acc = fma(bias, sum(x), acc)  per chunk; the
// eight lane sums are added by an xor butterfly (4, 2, 1).  A warp therefore covers four weight
// rows, and the per-(weight row, input row) arithmetic does not depend on how many input rows a
// job carries.  Input rows are staged once per job in shared memory as fp32, in an order that
// makes the eight lanes' 128-bit reads contiguous.
//
// Reference kernels this file stands in for (paths inside the reference project):
//   Sources/ANEFieldfareHotpath/Metal/MoE/moe.metal:65-103,186-319,382-517,548-638
//   Sources/ANEFieldfareHotpath/Metal/Prefill/prefill.metal:544-565,1246-1529
//   Sources/ANEFieldfareHotpath/Metal/Quant/dequant_int4.metal:78-347
#include <algorithm>
#include <initializer_list>

#include "ff_gemv_device.cuh"
#include "ff_internal.cuh"

namespace ff {

template <int NT, bool DUAL>
__device__ __forceinline__ void run_item(const GemvJob &job, int row0, const float *xs,
                                         const float *xsum) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = row0 + warp * 4 + (lane >> 3);
    const bool live = row < (int)job.rows;
    int sel[NT];  // staged row each input reads
#pragma unroll
    for (int t = 0; t < NT; ++t) sel[t] = t < (int)job.n ? t : 0;
    float a0[NT], a1[NT];
    row_dot<NT, DUAL>(job.w0, job.s0, job.b0, job.w1, job.s1, job.b1, row, (int)job.cols, live, xs,
                      xsum, sel, a0, a1);
    if (live && (lane & 7) == 0) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            if (t < (int)job.n) {
                float v = a0[t];
                if (DUAL) {
                    float g = a0[t], u = a1[t];
                    if (job.flags & kJobRoundGateUp) {
                        g = bf16_round(g);
                        u = bf16_round(u);
                    }
                    v = gelu_tanh(g) * u;
                }
                job.out[(size_t)job.outRow[t] * job.outStride + row] = f2bf(v);
            }
        }
    }
}

// Persistent GEMV over a job's row blocks: its input rows are staged once per CTA.
template <int MAXNT, bool DUAL>
__global__ void __launch_bounds__(kGemvThreads) k_int4_gemv(const __grid_constant__ GemvJob job, uint32_t blocks) {
    extern __shared__ float smem[];
    __shared__ GemvJob sjob;
    float *xs = smem;
    float *xsum = smem + MAXNT * staged_stride((int)job.cols);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&job);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&sjob);
    for (int i = threadIdx.x; i < (int)(sizeof(GemvJob) / 4); i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    const int n = (int)sjob.n;
    stage_rows(sjob.in, sjob.inStride, sjob.inRow, min(n, MAXNT), (int)sjob.cols, xs, xsum);
    for (uint32_t block = blockIdx.x; block < blocks; block += gridDim.x) {
        const int row0 = (int)block * kRowsPerItem;
        if (n <= 1) {
            run_item<1, DUAL>(sjob, row0, xs, xsum);
        } else if (MAXNT >= 2 && n <= 2) {
            run_item<(MAXNT >= 2 ? 2 : 1), DUAL>(sjob, row0, xs, xsum);
        } else if (MAXNT >= 4 && n <= 4) {
            run_item<(MAXNT >= 4 ? 4 : 1), DUAL>(sjob, row0, xs, xsum);
        } else if (MAXNT >= 8 && n <= 8) {
            run_item<(MAXNT >= 8 ? 8 : 1), DUAL>(sjob, row0, xs, xsum);
        } else if (MAXNT >= 16) {
            run_item<(MAXNT >= 16 ? 16 : 1), DUAL>(sjob, row0, xs, xsum);
        }
    }
}

// ---- router --------------------------------------------------------------------------------

// One warp per (expert, token).  The reduction order is part of the contract (top-K indices are
// compared for equality with the CPU oracle): lane l chains fmaf over elements
// [256 i + 8 l, +8) for i = 0, 1, ... in increasing index, the lane sums are added by an xor
// butterfly (16, 8, 4, 2, 1), then the per-expert logit bias is added.
// The expert's row of the first kRowChunks * 256 inputs, and the per-input scale (by way of shared memory: the CTA's eight
// warps need the same), are requested in front of the wait for the launch before, the token's row all together behind it.
// Bound by its latencies.  us in a graph, 128 experts, in loads of a few chunks / eleven chunks with the scale fetched where
// it is used / now: 2816 inputs, one row 5.3 / 5.5 / 5.0, 16 rows 6.6 / 6.8 / 6.3; scaled 6.3 / 6.8 / 5.2, 7.5 / 7.9 / 6.7; 4096
// inputs, scaled, one row 7.4 / 8.2 / 5.7.  Eleven chunks, all of 2816 inputs, are no faster there than twelve and take a second
// turn for 2880 to 3072 (scaled, 16 rows 7.3 / 6.9).  kRowChunks 0: loads where they are used, in few registers (39).
template <int kRowChunks>
__global__ void __launch_bounds__(256)
k_router_logits(const uint16_t *W, const uint16_t *scale, const float *bias, const uint16_t *x,
                uint32_t xStride, int E, int D, float *logits, RouterTail tail) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = min((int)blockIdx.x * 8 + warp, E - 1);  // (a warp past the experts repeats the last)
    const int t = blockIdx.y;
    const uint16_t *wr = W + (size_t)e * D;
    const uint16_t *xr = x + (size_t)t * xStride;
    float acc = 0.0f;
    auto add_chunk = [&](const uint4 &w, const uint4 &v, const uint4 &s) {
        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
        const uint32_t xx[4] = {v.x, v.y, v.z, v.w};
        const uint32_t ss[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float x0 = __uint_as_float(xx[k] << 16), x1 = __uint_as_float(xx[k] & 0xFFFF0000u);
            if (scale) {
                x0 = x0 * __uint_as_float(ss[k] << 16);
                x1 = x1 * __uint_as_float(ss[k] & 0xFFFF0000u);
            }
            acc = fmaf(__uint_as_float(ww[k] << 16), x0, acc);
            acc = fmaf(__uint_as_float(ww[k] & 0xFFFF0000u), x1, acc);
        }
    };
    if constexpr (kRowChunks == 0) {
        pdl_enter();
        for (int base = 8 * lane; base < D; base += 256) {
            const uint4 w = *reinterpret_cast<const uint4 *>(wr + base);
            const uint4 v = *reinterpret_cast<const uint4 *>(xr + base);
            uint4 s = make_uint4(0, 0, 0, 0);
            if (scale) s = *reinterpret_cast<const uint4 *>(scale + base);
            add_chunk(w, v, s);
        }
    } else {
        __shared__ __align__(16) uint4 sScale[kRowChunks * 32];
        uint4 wv[kRowChunks];
        auto fetch = [&](int first) {
#pragma unroll
            for (int i = 0; i < kRowChunks; ++i) {
                const int base = first + 256 * i + 8 * lane;
                if (base < D) wv[i] = __ldg(reinterpret_cast<const uint4 *>(wr + base));
            }
            if (scale)
                for (int i = threadIdx.x; i < kRowChunks * 32 && first + 8 * i < D; i += 256)
                    sScale[i] = __ldg(reinterpret_cast<const uint4 *>(scale + first) + i);
        };
        fetch(0);
        pdl_enter();
        for (int first = 0; first < D; first += 256 * kRowChunks) {
            if (first) {
                if (scale) __syncthreads();  // every warp is done with the scales before
                fetch(first);
            }
            uint4 xv[kRowChunks];
#pragma unroll
            for (int i = 0; i < kRowChunks; ++i) {
                const int base = first + 256 * i + 8 * lane;
                if (base < D) xv[i] = *reinterpret_cast<const uint4 *>(xr + base);
            }
            if (scale) __syncthreads();
#pragma unroll
            for (int i = 0; i < kRowChunks; ++i) {
                if (first + 256 * i + 8 * lane >= D) break;
                uint4 s = make_uint4(0, 0, 0, 0);
                if (scale) s = sScale[32 * i + lane];
                add_chunk(wv[i], xv[i], s);
            }
        }
    }
#pragma unroll
    for (int offset = 16; offset >= 1; offset >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, offset);
    if (lane == 0) logits[(size_t)t * E + e] = bias ? acc + bias[e] : acc;
    if (tail.ids)
        topk_by_last_cta(logits + (size_t)t * E, E, tail.K, tail.gain, tail.ids + t * tail.K, tail.weights + t * tail.K, tail.counts + t,
                         gridDim.x);
}

// Metal/Prefill/prefill.metal:544-565 plus an optional residual row added after the ranks.
// rowIndex (optional): the partial row of route (t, r) is row rowIndex[t * K + r] of `partials`
// instead of row t * K + r — rows that came back from other GPUs in another order are reduced
// where they lie.
__global__ void __launch_bounds__(256)
k_reduce_token_major(const uint16_t *partials, const uint32_t *rowIndex, const uint16_t *weights,
                     const uint16_t *residual, uint16_t *y, int T, int K, int D) {
    const int t = blockIdx.y;
    const int d = (blockIdx.x * blockDim.x + threadIdx.x) * 2;
    if (t >= T || d >= D) return;
    float acc0 = 0.0f, acc1 = 0.0f;
    for (int r = 0; r < K; ++r) {
        const float w = bf2f(weights[(size_t)t * K + r]);
        const size_t row = rowIndex ? (size_t)rowIndex[(size_t)t * K + r] : (size_t)t * K + r;
        const uint32_t two = *reinterpret_cast<const uint32_t *>(partials + row * D + d);
        acc0 = fmaf(w, __uint_as_float(two << 16), acc0);
        acc1 = fmaf(w, __uint_as_float(two & 0xFFFF0000u), acc1);
    }
    if (residual) {
        const uint32_t two = *reinterpret_cast<const uint32_t *>(residual + (size_t)t * D + d);
        acc0 += __uint_as_float(two << 16);
        acc1 += __uint_as_float(two & 0xFFFF0000u);
    }
    *reinterpret_cast<uint32_t *>(y + (size_t)t * D + d) =
        (uint32_t)f2bf(acc0) | ((uint32_t)f2bf(acc1) << 16);
}

// The same reduce, eight outputs per thread with 128-bit loads (every element's chain is the one
// above: rank ascending, then the residual); for rows that are 16-byte aligned.  B = 8: the loads
// of eight ranks are issued together, for blocks of at most a wave, where their latencies one after another
// are the time (77 rows 4.4 -> 3.5 us); B = 1 beyond, where more warps in flight beat more loads of each (32768
// rows 363 us, with B = 8 450 us).  STREAM: the partial rows are streamed, which pays from four of them a row on: eight a row,
// written and reduced, 1500 rows of 2816 36.2 -> 33.7 us, 4096 102.0 -> 91.0 (a layer of 4096 rows 614 -> 607); four, 4096 rows
// 54.9 -> 48.8; three 39.5 -> 41.5, two 26.9 -> 28.6.  With B = 8 from eight on: 200 rows of 2816 2.7 -> 2.4; six, 40 rows of 6144
// 2.1 -> 2.5, five, 128 rows of 1024 1.9 -> 2.3.
template <int B, bool STREAM>
__global__ void __launch_bounds__(256)
k_reduce_token_major_x8(const uint16_t *partials, const uint32_t *rowIndex, const uint16_t *weights,
                        const uint16_t *residual, uint16_t *y, int T, int K, int D) {
    pdl_enter();
    const int perRow = D >> 3;
    const size_t item = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= (size_t)T * perRow) return;
    const int t = (int)(item / perRow), d = (int)(item - (size_t)t * perRow) * 8;
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
    uint4 rest = make_uint4(0, 0, 0, 0);
    if (residual) rest = *reinterpret_cast<const uint4 *>(residual + (size_t)t * D + d);
    for (int r0 = 0; r0 < K; r0 += B) {
        uint4 v[B];
        float w[B];
#pragma unroll
        for (int r = 0; r < B; ++r) {
            if (r0 + r < K) {
                const size_t route = (size_t)t * K + r0 + r, row = rowIndex ? (size_t)rowIndex[route] : route;
                w[r] = bf2f(weights[route]);
                const uint4 *src = reinterpret_cast<const uint4 *>(partials + row * D + d);
                v[r] = STREAM ? __ldcs(src) : *src;  // read once
            }
        }
#pragma unroll
        for (int r = 0; r < B; ++r) {
            if (r0 + r < K) {
                const uint32_t p[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[2 * i] = fmaf(w[r], __uint_as_float(p[i] << 16), acc[2 * i]);
                    acc[2 * i + 1] = fmaf(w[r], __uint_as_float(p[i] & 0xFFFF0000u), acc[2 * i + 1]);
                }
            }
        }
    }
    if (residual) {
        const uint32_t p[4] = {rest.x, rest.y, rest.z, rest.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[2 * i] += __uint_as_float(p[i] << 16);
            acc[2 * i + 1] += __uint_as_float(p[i] & 0xFFFF0000u);
        }
    }
    uint4 o;
    o.x = (uint32_t)f2bf(acc[0]) | ((uint32_t)f2bf(acc[1]) << 16);
    o.y = (uint32_t)f2bf(acc[2]) | ((uint32_t)f2bf(acc[3]) << 16);
    o.z = (uint32_t)f2bf(acc[4]) | ((uint32_t)f2bf(acc[5]) << 16);
    o.w = (uint32_t)f2bf(acc[6]) | ((uint32_t)f2bf(acc[7]) << 16);
    *reinterpret_cast<uint4 *>(y + (size_t)t * D + d) = o;
}

// ---- row kernels: RMSNorm and the fused steps either side of the block ----------------------------
//
// One CTA of 256 threads per row.  A row moves as 16-byte pieces (thread t takes pieces t, t + 256, ...;
// every operand is asked for before the first sum is formed), and goes through shared memory for the
// sum of squares, whose order is fixed: thread t chains fmaf over elements t, t + 256, ..., butterfly
// inside a warp, warps in order.  Bound by HBM for many rows (32768 rows of 2816: RMSNorm 213 us with
// 2-byte accesses) and by one load latency and the two sums for one row (the step in front of the block
// 21 us, the one behind it 15 us, when every pass read its row again).

constexpr int kRowThreads = 256;

// Piece c of a row; WIDE: 16-byte aligned rows.
template <bool WIDE>
__device__ __forceinline__ uint4 load_piece(const uint16_t *row, int c) {
    uint4 v;
    if (WIDE) {
        v = *(reinterpret_cast<const uint4 *>(row) + c);
    } else {
        uint16_t h[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = row[8 * c + i];
        v = make_uint4(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16), h[4] | ((uint32_t)h[5] << 16), h[6] | ((uint32_t)h[7] << 16));
    }
    return v;
}
template <bool WIDE>
__device__ __forceinline__ void store_piece(uint16_t *row, int c, const uint4 &v) {
    if (WIDE) {
        *(reinterpret_cast<uint4 *>(row) + c) = v;
        return;
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        row[8 * c + 2 * i] = (uint16_t)w[i];
        row[8 * c + 2 * i + 1] = (uint16_t)(w[i] >> 16);
    }
}
// out[i] = f(a[i], b[i], c[i]) over the eight elements of pieces, f giving bf16 bits.
template <typename F>
__device__ __forceinline__ uint4 map_pieces(const uint4 &a, const uint4 &b, const uint4 &c, F f) {
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w}, cw[4] = {c.x, c.y, c.z, c.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t lo = f(__uint_as_float(aw[i] << 16), __uint_as_float(bw[i] << 16), __uint_as_float(cw[i] << 16));
        const uint32_t hi = f(__uint_as_float(aw[i] & 0xFFFF0000u), __uint_as_float(bw[i] & 0xFFFF0000u),
                              __uint_as_float(cw[i] & 0xFFFF0000u));
        o[i] = lo | (hi << 16);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// 1 / rms of `row` (in shared memory, written by the caller's threads just before).
__device__ __forceinline__ float row_rms_inv(const uint16_t *row, int D, float eps, float *warpSums) {
    __syncthreads();  // the row is there, and warpSums no longer read
    float sq = 0.0f;
#pragma unroll 8
    for (int i = threadIdx.x; i < D; i += kRowThreads) {
        const float v = bf2f(row[i]);
        sq = fmaf(v, v, sq);
    }
#pragma unroll
    for (int offset = 16; offset >= 1; offset >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, offset);
    if ((threadIdx.x & 31) == 0) warpSums[threadIdx.x >> 5] = sq;
    __syncthreads();
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < kRowThreads / 32; ++i) total += warpSums[i];
    return 1.0f / sqrtf(total / (float)D + eps);
}

// y = x * w * rsqrt(mean(x^2) + eps).  C: pieces per thread.
template <int C, bool WIDE>
__global__ void __launch_bounds__(kRowThreads)
k_rmsnorm(const uint16_t *x, const uint16_t *w, float eps, int D, uint16_t *y) {
    pdl_enter();
    extern __shared__ __align__(16) uint16_t glueRow[];
    __shared__ float warpSums[kRowThreads / 32];
    const size_t row = (size_t)blockIdx.x * D;
    const uint4 ones = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    uint4 xv[C], wv[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D) {
            xv[i] = load_piece<WIDE>(x + row, c);
            wv[i] = w ? load_piece<WIDE>(w, c) : ones;
            reinterpret_cast<uint4 *>(glueRow)[c] = xv[i];
        }
    }
    const float inv = row_rms_inv(glueRow, D, eps, warpSums);
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D)
            store_piece<WIDE>(y + row, c, map_pieces(xv[i], wv[i], wv[i], [&](float a, float b, float) { return (uint32_t)f2bf(a * b * inv); }));
    }
}

// The same for rows too wide for the row buffer.
__global__ void __launch_bounds__(kRowThreads)
k_rmsnorm_long(const uint16_t *x, const uint16_t *w, float eps, int D, uint16_t *y) {
    pdl_enter();
    __shared__ float warpSums[kRowThreads / 32];
    const size_t row = (size_t)blockIdx.x * D;
    const float inv = row_rms_inv(x + row, D, eps, warpSums);
    for (int i = threadIdx.x; i < D; i += kRowThreads) y[row + i] = f2bf(bf2f(x[row + i]) * (w ? bf2f(w[i]) : 1.0f) * inv);
}

// prefill_post_attn_setup_block (Metal/Prefill/prefill.metal:244-318):
//   a = r16(attn * rms_inv(attn) * w_post_attn);  hidden = r16(hidden + a);
//   n = hidden * rms_inv(hidden);  dense_x = r16(n * w_pre_ffn);  routed_x = r16(n * w_pre_ffn2);
//   router_x = r16(n).
template <int C, bool WIDE>
__global__ void __launch_bounds__(kRowThreads)
k_post_attn_setup(uint16_t *hidden, const uint16_t *attn, const uint16_t *wPostAttn, const uint16_t *wPreFfn,
                  const uint16_t *wPreFfn2, float eps, int D, uint16_t *denseX, uint16_t *routedX,
                  uint16_t *routerX) {
    pdl_enter();
    extern __shared__ __align__(16) uint16_t glueRow[];
    __shared__ float warpSums[kRowThreads / 32];
    const size_t row = (size_t)blockIdx.x * D;
    uint4 av[C], hv[C], wA[C], w1[C], w2[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D) {
            av[i] = load_piece<WIDE>(attn + row, c);
            hv[i] = load_piece<WIDE>(hidden + row, c);
            wA[i] = load_piece<WIDE>(wPostAttn, c);
            w1[i] = load_piece<WIDE>(wPreFfn, c);
            w2[i] = load_piece<WIDE>(wPreFfn2, c);
            reinterpret_cast<uint4 *>(glueRow)[c] = av[i];
        }
    }
    const float attnInv = row_rms_inv(glueRow, D, eps, warpSums);  // (every read of the row is behind its barrier)
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D) {
            hv[i] = map_pieces(av[i], hv[i], wA[i],
                               [&](float a, float h, float w) { return (uint32_t)f2bf(h + bf16_round(a * attnInv * w)); });
            reinterpret_cast<uint4 *>(glueRow)[c] = hv[i];
            store_piece<WIDE>(hidden + row, c, hv[i]);
        }
    }
    const float inv = row_rms_inv(glueRow, D, eps, warpSums);
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D) {
            store_piece<WIDE>(denseX + row, c, map_pieces(hv[i], w1[i], w1[i], [&](float h, float w, float) { return (uint32_t)f2bf(h * inv * w); }));
            store_piece<WIDE>(routedX + row, c, map_pieces(hv[i], w2[i], w2[i], [&](float h, float w, float) { return (uint32_t)f2bf(h * inv * w); }));
            store_piece<WIDE>(routerX + row, c, map_pieces(hv[i], hv[i], hv[i], [&](float h, float, float) { return (uint32_t)f2bf(h * inv); }));
        }
    }
}

// prefill_layer_tail_block (Metal/Prefill/prefill.metal:321-399; one row: Metal/Fusions/fused.metal:470-474):
//   t = r16(h2 * rms_inv(h2) * w_postffn2);  h12 = r16(h1 + t);
//   u = r16(h12 * rms_inv(h12) * w_postffn);  hidden = r16(r16(hidden + u) * r16(layer_scalar)).
template <int C, bool WIDE>
__global__ void __launch_bounds__(kRowThreads)
k_layer_tail(const uint16_t *h2, const uint16_t *h1, uint16_t *hidden, const uint16_t *wPostFfn2,
             const uint16_t *wPostFfn, float eps, float layerScalar, int D) {
    pdl_enter();
    extern __shared__ __align__(16) uint16_t glueRow[];
    __shared__ float warpSums[kRowThreads / 32];
    const size_t row = (size_t)blockIdx.x * D;
    uint4 bv[C], av[C], hv[C], w2[C], w1[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D) {
            bv[i] = load_piece<WIDE>(h2 + row, c);
            av[i] = load_piece<WIDE>(h1 + row, c);
            hv[i] = load_piece<WIDE>(hidden + row, c);
            w2[i] = load_piece<WIDE>(wPostFfn2, c);
            w1[i] = load_piece<WIDE>(wPostFfn, c);
            reinterpret_cast<uint4 *>(glueRow)[c] = bv[i];
        }
    }
    const float inv2 = row_rms_inv(glueRow, D, eps, warpSums);
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D) {
            av[i] = map_pieces(bv[i], av[i], w2[i],
                               [&](float b, float a, float w) { return (uint32_t)f2bf(a + bf16_round(b * inv2 * w)); });
            reinterpret_cast<uint4 *>(glueRow)[c] = av[i];
        }
    }
    const float inv12 = row_rms_inv(glueRow, D, eps, warpSums);
    const float scale = bf16_round(layerScalar);
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int c = threadIdx.x + kRowThreads * i;
        if (8 * c < D)
            store_piece<WIDE>(hidden + row, c, map_pieces(av[i], hv[i], w1[i], [&](float a, float h, float w) {
                                  return (uint32_t)f2bf(bf16_round(h + bf16_round(a * inv12 * w)) * scale);
                              }));
    }
}

// A row kernel by the pieces a thread holds (rows of 4096 values and less: two) and the rows' alignment.
#define FF_ROW_KERNEL(NAME, D, WIDE, ...)                                                                              \
    do {                                                                                                               \
        const size_t smem_ = (size_t)(D) * 2;                                                                          \
        static KernelSmemMemo memo_[6];                                                                                \
        auto go_ = [&](auto kernel, KernelSmemMemo &memo) {                                                            \
            if (!memo.prepare(kernel, ctx->device, smem_, kRowThreads, nullptr, error)) return false;                  \
            LaunchScope scope(ctx, stream, #NAME);                                                                     \
            FF_CUDA_OK(launch_pdl(kernel, tokens, kRowThreads, smem_, stream, __VA_ARGS__), error);                      \
            return true;                                                                                               \
        };                                                                                                             \
        const bool ok_ = (D) <= 4096    ? ((WIDE) ? go_(k_##NAME<2, true>, memo_[0]) : go_(k_##NAME<2, false>, memo_[1]))  \
                         : (D) <= 16384 ? ((WIDE) ? go_(k_##NAME<8, true>, memo_[2]) : go_(k_##NAME<8, false>, memo_[3]))  \
                                        : ((WIDE) ? go_(k_##NAME<24, true>, memo_[4]) : go_(k_##NAME<24, false>, memo_[5])); \
        if (!ok_) return false;                                                                                        \
    } while (0)

static bool aligned16(std::initializer_list<const void *> pointers) {
    uintptr_t all = 0;
    for (const void *p : pointers) all |= reinterpret_cast<uintptr_t>(p);
    return (all & 15u) == 0;
}

bool launch_rmsnorm(FFContext *ctx, const uint16_t *x, const uint16_t *w, float eps, uint32_t tokens, uint16_t *y,
                    cudaStream_t stream, const char **error) {
    if (tokens == 0) return true;
    const int D = (int)ctx->cfg.d;
    if ((size_t)D * 2 > 96 * 1024) {
        LaunchScope scope(ctx, stream, "rmsnorm");
        k_rmsnorm_long<<<tokens, kRowThreads, 0, stream>>>(x, w, eps, D, y);
        FF_CUDA_OK(cudaGetLastError(), error);
        return true;
    }
    FF_ROW_KERNEL(rmsnorm, D, aligned16({x, w, y}), x, w, eps, D, y);
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

bool launch_post_attn_setup(FFContext *ctx, uint16_t *hidden, const uint16_t *attn, const uint16_t *wPostAttn,
                            const uint16_t *wPreFfn, const uint16_t *wPreFfn2, float eps, uint32_t tokens,
                            uint16_t *denseX, uint16_t *routedX, uint16_t *routerX, cudaStream_t stream,
                            const char **error) {
    if (tokens == 0) return true;
    const int D = (int)ctx->cfg.d;
    if ((size_t)D * 2 > 96 * 1024) return fail(error, "model width too large for the row buffer");
    FF_ROW_KERNEL(post_attn_setup, D, aligned16({hidden, attn, wPostAttn, wPreFfn, wPreFfn2, denseX, routedX, routerX}), hidden, attn,
                  wPostAttn, wPreFfn, wPreFfn2, eps, D, denseX, routedX, routerX);
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

bool launch_layer_tail(FFContext *ctx, const uint16_t *h2, const uint16_t *h1, uint16_t *hidden,
                       const uint16_t *wPostFfn2, const uint16_t *wPostFfn, float eps, float layerScalar,
                       uint32_t tokens, cudaStream_t stream, const char **error) {
    if (tokens == 0) return true;
    const int D = (int)ctx->cfg.d;
    if ((size_t)D * 2 > 96 * 1024) return fail(error, "model width too large for the row buffer");
    FF_ROW_KERNEL(layer_tail, D, aligned16({h2, h1, hidden, wPostFfn2, wPostFfn}), h2, h1, hidden, wPostFfn2, wPostFfn, eps, layerScalar, D);
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

// w = q*scale + bias for a whole matrix, fp32 and/or bf16 (one rounding of the exact value:
// a bf16 fused multiply-add).  One thread per 8 codes.
__global__ void __launch_bounds__(256)
k_dequant_probe(const uint8_t *w, const uint16_t *s, const uint16_t *b, int rows, int cols,
                float *out32, uint16_t *out16) {
    const size_t word = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t wordsPerRow = (size_t)cols / 8;
    if (word >= (size_t)rows * wordsPerRow) return;
    const size_t row = word / wordsPerRow;
    const int col = (int)(word - row * wordsPerRow) * 8;
    const uint32_t packed = reinterpret_cast<const uint32_t *>(w)[word];
    const size_t g = row * (size_t)(cols / kGroup) + (size_t)(col / kGroup);
    const float scale = bf2f(s[g]), bias = bf2f(b[g]);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float q = (float)((packed >> (4 * k)) & 0xFu);
        if (out32) out32[row * cols + col + k] = fmaf(q, scale, bias);
        if (out16) {
            // exact in double, then one rounding to bf16 via round-to-odd fp32
            const double exact = (double)q * (double)scale + (double)bias;
            float f = __double2float_rz(exact);
            if ((double)f != exact) f = __uint_as_float(__float_as_uint(f) | 1u);
            out16[row * cols + col + k] = f2bf(f);
        }
    }
}

// ---- host launchers ------------------------------------------------------------------------

static size_t gemv_smem_bytes(int rows, uint32_t maxCols) {
    return (size_t)rows * (staged_stride((int)maxCols) + (maxCols >> 5)) * sizeof(float);
}

constexpr size_t kGemvSmemLimit = 200 * 1024;
static uint32_t gemv_rows_class(uint32_t n) { return n <= 1 ? 1 : n <= 2 ? 2 : n <= 4 ? 4 : n <= 8 ? 8 : 16; }
// Input rows one launch can stage for a job of `n` rows and `cols` columns: the job's row class,
// or the largest smaller class that fits in shared memory; 0 when not even one row fits.
static uint32_t gemv_pass_rows(uint32_t n, uint32_t cols) {
    for (uint32_t c = gemv_rows_class(n); c >= 1; c >>= 1)
        if (gemv_smem_bytes((int)c, cols) <= kGemvSmemLimit) return c;
    return 0;
}

static uint32_t blocks_of(uint32_t rows) { return (rows + kRowsPerItem - 1) / kRowsPerItem; }

template <int MAXNT, bool DUAL>
static bool launch_gemv_kernel(FFContext *ctx, const GemvJob &job, cudaStream_t stream, const char **error) {
    auto kernel = k_int4_gemv<MAXNT, DUAL>;
    const size_t smem = gemv_smem_bytes(MAXNT, job.cols);
    if (smem > kGemvSmemLimit)
        return fail(error, "input rows do not fit in shared memory: " + std::to_string(MAXNT) +
                               " rows x " + std::to_string(job.cols) + " columns");
    // attribute + occupancy are looked up once per (kernel, device, shared-memory size): nothing but
    // the launch itself happens on later calls, which keeps the call legal under stream capture
    static KernelSmemMemo memo;
    int perSm = 0;
    if (!memo.prepare(kernel, ctx->device, smem, kGemvThreads, &perSm, error)) return false;
    if (perSm < 1) return fail(error, "GEMV kernel does not fit on an SM");
    const uint32_t blocks = blocks_of(job.rows);
    const uint32_t grid = std::min(blocks, (uint32_t)(ctx->smCount * perSm));
    if (grid == 0) return true;
    {
        LaunchScope scope(ctx, stream, DUAL ? "int4_gemv_gate_up_act" : "int4_gemv_down");
        kernel<<<grid, kGemvThreads, smem, stream>>>(job, blocks);
    }
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

template <bool DUAL>
static bool launch_gemv_class(FFContext *ctx, const GemvJob &job, cudaStream_t stream, const char **error) {
    if (job.n <= 1) return launch_gemv_kernel<1, DUAL>(ctx, job, stream, error);
    if (job.n <= 2) return launch_gemv_kernel<2, DUAL>(ctx, job, stream, error);
    if (job.n <= 4) return launch_gemv_kernel<4, DUAL>(ctx, job, stream, error);
    if (job.n <= 8) return launch_gemv_kernel<8, DUAL>(ctx, job, stream, error);
    return launch_gemv_kernel<16, DUAL>(ctx, job, stream, error);
}

// One job given by value (a matrix, or a gate/up pair, against job.n <= 16 input rows).  When the
// rows of the job's class do not fit in shared memory together (wide matrices), the job runs as
// passes of fewer rows: the arithmetic per (weight row, input row) does not depend on how many
// rows a launch carries, so the bits are those of a single pass.
template <bool DUAL>
static bool launch_inline_job(FFContext *ctx, const GemvJob &job, cudaStream_t stream, const char **error) {
    const uint32_t pass = gemv_pass_rows(job.n, job.cols);
    if (pass == 0)
        return fail(error, "one input row of " + std::to_string(job.cols) + " columns does not fit in shared memory");
    for (uint32_t first = 0; first < job.n; first += pass) {
        GemvJob part = job;
        part.n = std::min(pass, job.n - first);
        for (uint32_t i = 0; i < (uint32_t)kMaxGemvRows; ++i) {
            part.inRow[i] = i < part.n ? job.inRow[first + i] : 0u;
            part.outRow[i] = i < part.n ? job.outRow[first + i] : 0u;
        }
        if (!launch_gemv_class<DUAL>(ctx, part, stream, error)) return false;
    }
    return true;
}

constexpr int kInt8Rows = 4;  // input rows of a warp

// INT8 affine shared FFN (Metal/Quant/dequant_int8.metal:41-138; Kernels/MoE/SharedExpertInt8.swift) for the
// shapes and alignments the tensor-core kernels do not take: one warp per output row and up to four
// input rows, in the reference kernels' order made definite:
// lane l takes elements 64 g + 2 l and + 1 of every group g in increasing g,
//   acc = fma(s_g, fma(q1, x1, q0 * x0), acc);  acc = fma(b_g, x0 + x1, acc);
// lane sums by an xor butterfly (16..1).  DUAL: gate and up rows of the same index, both rounded to
// 16 bits, then act = r16(gelu_tanh(gate) * up); otherwise one matrix, out = r16(sum).
template <bool DUAL>
__global__ void __launch_bounds__(256)
k_int8_rows(const uint8_t *W0, const uint16_t *S0, const uint16_t *B0, const uint8_t *W1, const uint16_t *S1,
            const uint16_t *B1, const uint16_t *x, uint32_t xStride, int T, int rows, int cols, uint16_t *out,
            uint32_t outStride) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * 8 + warp;
    const int t0 = blockIdx.y * kInt8Rows;
    if (r >= rows) return;
    const int groups = cols / 64;
    const uint8_t *w0 = W0 + (size_t)r * cols, *w1 = DUAL ? W1 + (size_t)r * cols : nullptr;
    const uint16_t *s0 = S0 + (size_t)r * groups, *b0 = B0 + (size_t)r * groups;
    const uint16_t *s1 = DUAL ? S1 + (size_t)r * groups : nullptr, *b1 = DUAL ? B1 + (size_t)r * groups : nullptr;
    float acc0[kInt8Rows], acc1[kInt8Rows];
#pragma unroll
    for (int i = 0; i < kInt8Rows; ++i) acc0[i] = acc1[i] = 0.0f;
    for (int g = 0; g < groups; ++g) {
        const int idx = g * 64 + 2 * lane;
        const uint32_t q = *reinterpret_cast<const uint16_t *>(w0 + idx);
        const float q00 = (float)(q & 0xFFu), q01 = (float)(q >> 8);
        const float sa = bf2f(s0[g]), ba = bf2f(b0[g]);
        float q10 = 0.0f, q11 = 0.0f, sb = 0.0f, bb = 0.0f;
        if (DUAL) {
            const uint32_t p = *reinterpret_cast<const uint16_t *>(w1 + idx);
            q10 = (float)(p & 0xFFu);
            q11 = (float)(p >> 8);
            sb = bf2f(s1[g]);
            bb = bf2f(b1[g]);
        }
#pragma unroll
        for (int i = 0; i < kInt8Rows; ++i) {
            const int t = min(t0 + i, T - 1);
            const uint32_t xv = *reinterpret_cast<const uint32_t *>(x + (size_t)t * xStride + idx);
            const float x0 = __uint_as_float(xv << 16), x1 = __uint_as_float(xv & 0xFFFF0000u);
            const float sumX = x0 + x1;
            acc0[i] = fmaf(sa, fmaf(q01, x1, q00 * x0), acc0[i]);
            acc0[i] = fmaf(ba, sumX, acc0[i]);
            if (DUAL) {
                acc1[i] = fmaf(sb, fmaf(q11, x1, q10 * x0), acc1[i]);
                acc1[i] = fmaf(bb, sumX, acc1[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kInt8Rows; ++i) {
        float a = acc0[i], b = acc1[i];
#pragma unroll
        for (int offset = 16; offset >= 1; offset >>= 1) {
            a += __shfl_xor_sync(0xFFFFFFFFu, a, offset);
            if (DUAL) b += __shfl_xor_sync(0xFFFFFFFFu, b, offset);
        }
        if (lane == 0 && t0 + i < T) {
            uint16_t v;
            if (DUAL) v = f2bf(gelu_tanh(bf16_round(a)) * bf16_round(b));
            else v = f2bf(a);
            out[(size_t)(t0 + i) * outStride + r] = v;
        }
    }
}

// y = down(r16(gelu_tanh(r16(gate x)) * r16(up x))) for any number of rows; the activations go through
// the context's shared-activation scratch.
bool launch_shared_int8(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride, uint32_t tokens,
                        uint16_t *y, cudaStream_t stream, const char **error) {
    if (tokens == 0) return true;
    if (!L.has_shared8()) return fail(error, "layer has no resident shared FFN");
    const int D = (int)ctx->cfg.d, Fs = (int)ctx->cfg.sharedF;
    if (D % 64 || Fs % 64) return fail(error, "widths must be multiples of 64");
    if (xStride % 2 || ((uintptr_t)x & 3)) return fail(error, "input rows must be 4-byte aligned");
    if (tokens > ctx->cfg.maxTokens) return fail(error, "rows exceed the context's maxTokens");
    // more rows than a block, 16-byte aligned (what the tile copies and stores need): the tensor cores
    if (tokens > (uint32_t)kMaxGemvRows && !((uintptr_t)x & 15) && !((uintptr_t)y & 15) && xStride % 8 == 0 &&
        int8_gemm_fits(D, Fs))
        return launch_shared_int8_gemm(ctx, L, x, xStride, tokens, y, stream, error);
    if (tokens <= (uint32_t)kMaxGemvRows && !((uintptr_t)x & 15) && xStride % 8 == 0 && D <= 8192 && Fs <= 8192)
        return launch_block_int8(ctx, L, x, xStride, tokens, y, stream, error);
    uint16_t *acts = ctx->sharedActs;
    const unsigned tokenBlocks = (tokens + kInt8Rows - 1) / kInt8Rows;
    {
        LaunchScope scope(ctx, stream, "shared_int8_gate_up_act");
        k_int8_rows<true><<<dim3((Fs + 7) / 8, tokenBlocks), 256, 0, stream>>>(
            L.shared8W[0], L.shared8S[0], L.shared8B[0], L.shared8W[1], L.shared8S[1], L.shared8B[1], x, xStride,
            (int)tokens, Fs, D, acts, (uint32_t)Fs);
    }
    {
        LaunchScope scope(ctx, stream, "shared_int8_down");
        k_int8_rows<false><<<dim3((D + 7) / 8, tokenBlocks), 256, 0, stream>>>(
            L.shared8W[2], L.shared8S[2], L.shared8B[2], nullptr, nullptr, nullptr, acts, (uint32_t)Fs, (int)tokens, D,
            Fs, y, (uint32_t)D);
    }
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

// Top-K of logits rows, one warp per row (the rows' logits are in global memory).
__global__ void __launch_bounds__(256)
k_topk_rows(const float *logits, const uint16_t *gain, int T, int E, int K, uint32_t *ids, uint16_t *weights) {
    const int t = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (t >= T) return;
    warp_topk(logits + (size_t)t * E, E, K, gain, ids + (size_t)t * K, weights + (size_t)t * K);
}

bool launch_router_topk(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                        uint32_t tokens, uint32_t *ids, uint16_t *weights, float *logits,
                        cudaStream_t stream, const char **error) {
    if (tokens == 0) return true;
    if (!L.has_router()) return fail(error, "layer has no resident router");
    const int E = (int)L.routerExperts, D = (int)ctx->cfg.d;
    // (16-byte aligned rows for the tile copies; a CTA's rows as fp32 in shared memory)
    if (tokens > kMaxGemvRows && !logits && !((uintptr_t)x & 15) && xStride % 8 == 0 && D % 64 == 0 && D <= 12288)
        return launch_router_select(ctx, L, x, xStride, tokens, ids, weights, stream, error);
    if (L.routerQ && tokens > kMaxGemvRows) {
        float *lg = logits ? logits : ctx->logitsRows;
        if (!launch_router_logits_int8(ctx, L, x, xStride, tokens, lg, RouterTail{}, stream, error)) return false;
        {
            LaunchScope scope(ctx, stream, "topk_rows");
            k_topk_rows<<<(tokens + 7) / 8, 256, 0, stream>>>(lg, L.gain, (int)tokens, E, (int)ctx->cfg.topK, ids,
                                                             weights);
        }
        FF_CUDA_OK(cudaGetLastError(), error);
        return true;
    }
    if (tokens > kMaxGemvRows)
        return launch_router_prefill(ctx, L, x, xStride, tokens, ids, weights, logits, stream, error);
    float *lg = logits ? logits : ctx->logits;
    const RouterTail tail{ids, weights, L.gain, ctx->routerCounts, (int)ctx->cfg.topK};
    if (L.routerQ) return launch_router_logits_int8(ctx, L, x, xStride, tokens, lg, tail, stream, error);
    {
        LaunchScope scope(ctx, stream, "router_logits");
        // Twelve chunks in flight (two CTAs an SM) while the CTAs are at most one wave of them, four (and four an SM) where they
        // are more than three an SM, loads where they are used in between.  us in a graph, 12 / 0 / 4: 160 experts, 16 rows, 4096
        // inputs 8.3 / 7.4 / 8.6, 6144 9.8 / 8.4 / 10.3, scaled 12.6 / 10.7 / 12.5; 256 experts, 9 rows, 6144 inputs 9.4 / 9.6 / 9.5, 13
        // rows 12.8 / 10.0 / 11.1, 16 rows 13.2 / 12.3 / 11.7, scaled 16.1 / 15.5 / 14.1.
        const dim3 grid((E + 7) / 8, tokens);
        const uint32_t perSm = (grid.x * grid.y + (uint32_t)ctx->smCount - 1u) / (uint32_t)ctx->smCount;
        auto kernel = perSm <= 2u ? k_router_logits<12> : perSm == 3u ? k_router_logits<0> : k_router_logits<4>;
        FF_CUDA_OK(launch_pdl(kernel, grid, 256, 0, stream, L.routerW, L.routerScale, L.logitBias, x, xStride, E, D, lg, tail), error);
    }
    return true;
}

// Router top-K (when ids is null) + routed experts (+ shared FFN) for up to 16 rows.
//   decodeCombine: one row; y = bf16(residual' + sum_k w_k v_k), residual' = shared output when
//                  withShared else `residual`.
//   otherwise:     partial rows are written; sharedOut receives the shared FFN rows.
bool launch_block_small(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                        uint32_t tokens, const uint32_t *ids, const uint16_t *weights,
                        bool withShared, bool decodeCombine, const uint16_t *residual,
                        uint16_t *partials, uint16_t *sharedOut, uint16_t *y,
                        cudaStream_t stream, const char **error) {
    if (tokens == 0) return true;
    if (tokens > kMaxGemvRows) return fail(error, "more than 16 rows in a decode/verify block");
    if (decodeCombine && tokens != 1) return fail(error, "decode combine takes exactly one row");
    if (!L.experts) return fail(error, "layer has no resident experts");
    if (withShared && !L.shared) return fail(error, "layer has no resident shared FFN");
    if (decodeCombine)
        return launch_decode_fused(ctx, L, x, ids, weights, withShared, true, residual, y, stream, error);
    if (!ids) {
        if (L.routerExperts != L.expertCount) return fail(error, "router and layer disagree on the expert count");
        if (!launch_router_topk(ctx, L, x, xStride, tokens, ctx->ids, ctx->weights, nullptr, stream, error)) return false;
        ids = ctx->ids;
    }
    return launch_block_int4(ctx, L, x, xStride, tokens, ids, withShared, partials, sharedOut, stream, error);
}

bool launch_reduce(FFContext *ctx, const uint16_t *partials, const uint16_t *weights,
                   const uint16_t *residual, uint16_t *y, uint32_t tokens, cudaStream_t stream,
                   const char **error, const uint32_t *rowIndex) {
    if (tokens == 0) return true;
    const int D = (int)ctx->cfg.d;
    const bool wide = D % 8 == 0 && !((reinterpret_cast<uintptr_t>(partials) | reinterpret_cast<uintptr_t>(y) |
                                        reinterpret_cast<uintptr_t>(residual)) & 15u);
    {
        LaunchScope scope(ctx, stream, "reduce_token_major");
        if (wide) {
            const size_t items = (size_t)tokens * (D / 8);
            const unsigned blocks = (unsigned)((items + 255) / 256);
            const uint32_t K = ctx->cfg.topK;
            auto kernel = blocks <= (unsigned)ctx->smCount * 4 ? (K == 8 ? k_reduce_token_major_x8<8, true> : k_reduce_token_major_x8<8, false>)
                                                               : (K > 3 ? k_reduce_token_major_x8<1, true> : k_reduce_token_major_x8<1, false>);
            FF_CUDA_OK(launch_pdl(kernel, blocks, 256, 0, stream,
                              partials, rowIndex, weights, residual, y, (int)tokens, (int)ctx->cfg.topK, D),
                   error);
        } else {
            dim3 grid((D / 2 + 255) / 256, tokens);
            k_reduce_token_major<<<grid, 256, 0, stream>>>(partials, rowIndex, weights, residual, y, (int)tokens,
                                                           (int)ctx->cfg.topK, D);
        }
    }
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

bool launch_gemv_rows(FFContext *ctx, const FFProjection &p, const uint16_t *x, uint32_t xStride,
                      uint32_t rows, uint16_t *y, uint32_t yStride, cudaStream_t stream,
                      const char **error) {
    if (rows == 0) return true;
    if (rows > kMaxGemvRows) return fail(error, "ff_int4_gemv_rows takes at most 16 input rows");
    if (p.cols % kGroup != 0) return fail(error, "columns must be a multiple of 64");
    if ((reinterpret_cast<uintptr_t>(p.weights) & 15u) || (p.cols / 2) % 16 != 0)
        return fail(error, "packed weights must be 16-byte aligned with 16-byte-multiple rows");
    GemvJob job{};
    job.w0 = static_cast<const uint8_t *>(p.weights);
    job.s0 = static_cast<const uint16_t *>(p.scales);
    job.b0 = static_cast<const uint16_t *>(p.biases);
    job.in = x;
    job.out = y;
    job.rows = p.rows;
    job.cols = p.cols;
    job.inStride = xStride;
    job.outStride = yStride;
    job.n = rows;
    for (uint32_t i = 0; i < kMaxGemvRows; ++i) job.inRow[i] = job.outRow[i] = i < rows ? i : 0u;
    return launch_inline_job<false>(ctx, job, stream, error);
}

// Shared FFN for up to 16 rows without a route plan: gate/up/GeGLU job, then the down job.
bool launch_shared_small(FFContext *ctx, const LayerStore &L, const uint16_t *x, uint32_t xStride,
                         uint32_t tokens, uint16_t *y, cudaStream_t stream, const char **error) {
    const FFConfig &c = ctx->cfg;
    if (tokens == 0) return true;
    if (!L.shared) return fail(error, "layer has no resident shared FFN");
    GemvJob j0{};
    j0.w0 = L.shared + L.sharedOff.gateWOff;
    j0.s0 = reinterpret_cast<const uint16_t *>(L.shared + L.sharedOff.gateSOff);
    j0.b0 = reinterpret_cast<const uint16_t *>(L.shared + L.sharedOff.gateBOff);
    j0.w1 = L.shared + L.sharedOff.upWOff;
    j0.s1 = reinterpret_cast<const uint16_t *>(L.shared + L.sharedOff.upSOff);
    j0.b1 = reinterpret_cast<const uint16_t *>(L.shared + L.sharedOff.upBOff);
    j0.in = x;
    j0.out = ctx->sharedActs;
    j0.rows = c.sharedF;
    j0.cols = c.d;
    j0.inStride = xStride;
    j0.outStride = c.sharedF;
    j0.n = tokens;
    j0.flags = kJobRoundGateUp;
    GemvJob j1{};
    j1.w0 = L.shared + L.sharedOff.downWOff;
    j1.s0 = reinterpret_cast<const uint16_t *>(L.shared + L.sharedOff.downSOff);
    j1.b0 = reinterpret_cast<const uint16_t *>(L.shared + L.sharedOff.downBOff);
    j1.in = ctx->sharedActs;
    j1.out = y;
    j1.rows = c.d;
    j1.cols = c.sharedF;
    j1.inStride = c.sharedF;
    j1.outStride = c.d;
    j1.n = tokens;
    for (uint32_t i = 0; i < kMaxGemvRows; ++i)
        j0.inRow[i] = j0.outRow[i] = j1.inRow[i] = j1.outRow[i] = i < tokens ? i : 0u;
    if (!launch_inline_job<true>(ctx, j0, stream, error)) return false;
    return launch_inline_job<false>(ctx, j1, stream, error);
}

bool launch_dequant_probe(FFContext *ctx, const uint8_t *w, const uint16_t *s, const uint16_t *b,
                          uint32_t rows, uint32_t cols, float *out32, uint16_t *out16,
                          cudaStream_t stream, const char **error) {
    const size_t words = (size_t)rows * cols / 8;
    {
        LaunchScope scope(ctx, stream, "dequant_probe");
        k_dequant_probe<<<(unsigned)((words + 255) / 256), 256, 0, stream>>>(w, s, b, (int)rows,
                                                                             (int)cols, out32, out16);
    }
    FF_CUDA_OK(cudaGetLastError(), error);
    return true;
}

}  // namespace ff

// ---- shared FFN without any allocation -----------------------------------------------------

// Scratch for ff_shared_ffn_noalloc: the GeGLU activations between the gate/up kernel and the
// down kernel, [kNoAllocMaxRows][kNoAllocMaxIntermediate] bf16 = 128 KiB.  It is part of the
// library image, so every GPU that loads the library holds it until the process exits.
constexpr uint32_t kNoAllocMaxRows = 16;
constexpr uint32_t kNoAllocMaxIntermediate = 4096;
constexpr uint32_t kNoAllocMaxWidth = 16384;
static __device__ __align__(256) uint16_t g_noAllocActs[kNoAllocMaxRows * kNoAllocMaxIntermediate];

extern "C" bool ff_shared_ffn_noalloc(const FFProjection *gate, const FFProjection *up,
                                      const FFProjection *down, const uint16_t *x,
                                      uint32_t xStride, uint32_t rows, uint16_t *y,
                                      uint32_t yStride, void *stream, const char **error) {
    using namespace ff;
    if (error) *error = nullptr;
    if (!gate || !up || !down || !x || !y) return fail(error, "null argument");
    if (rows == 0) return true;
    if (rows > kNoAllocMaxRows)
        return fail(error, "ff_shared_ffn_noalloc takes at most " + std::to_string(kNoAllocMaxRows) +
                               " rows, got " + std::to_string(rows));
    const uint32_t d = gate->cols, f = gate->rows;
    if (f > kNoAllocMaxIntermediate)
        return fail(error, "intermediate width " + std::to_string(f) +
                               " exceeds the static scratch's maximum of " +
                               std::to_string(kNoAllocMaxIntermediate));
    if (d > kNoAllocMaxWidth)
        return fail(error, "model width " + std::to_string(d) + " exceeds the maximum of " +
                               std::to_string(kNoAllocMaxWidth) + " (one input row must fit in shared memory)");
    if (up->rows != f || up->cols != d || down->rows != d || down->cols != f)
        return fail(error, "SharedExpert dimension mismatch: gate=(" + std::to_string(gate->rows) + "," +
                               std::to_string(gate->cols) + ") up=(" + std::to_string(up->rows) + "," +
                               std::to_string(up->cols) + ") down=(" + std::to_string(down->rows) + "," +
                               std::to_string(down->cols) + ")");
    if (d % kGroup || f % kGroup || d == 0 || f == 0)
        return fail(error, "widths must be non-zero multiples of the group size 64");
    if (xStride < d || yStride < d || xStride % 2) return fail(error, "row stride is too small or odd");
    if ((reinterpret_cast<uintptr_t>(x) & 3u) || (reinterpret_cast<uintptr_t>(y) & 1u))
        return fail(error, "input rows must be 4-byte aligned and output rows 2-byte aligned");
    const FFProjection *ps[3] = {gate, up, down};
    for (const FFProjection *p : ps)
        if (!p->weights || !p->scales || !p->biases || (reinterpret_cast<uintptr_t>(p->weights) & 15u) ||
            (reinterpret_cast<uintptr_t>(p->scales) & 1u) || (reinterpret_cast<uintptr_t>(p->biases) & 1u))
            return fail(error, "projection pointers must be non-null, the weights 16-byte aligned, scales and "
                               "biases 2-byte aligned");
    // both kernels' staging must fit before anything is enqueued (wide matrices run as passes of
    // fewer rows; kNoAllocMaxWidth and kNoAllocMaxIntermediate guarantee that one row always fits)
    if (gemv_pass_rows(rows, d) == 0 || gemv_pass_rows(rows, f) == 0)
        return fail(error, "one input row does not fit in shared memory");

    // Per-device set-up, done by the first call on each device with that device current: the
    // array's name is only a host-side handle, so its device address is looked up here.
    struct DeviceSetup {
        uint16_t *scratch = nullptr;
        int smCount = 0;
    };
    static DeviceSetup setups[kMaxDevices];
    static std::mutex setupLock;
    int device = 0;
    FF_CUDA_OK(cudaGetDevice(&device), error);
    if (device < 0 || device >= kMaxDevices) return fail(error, "device ordinal out of range");
    DeviceSetup setup;
    {
        std::lock_guard<std::mutex> guard(setupLock);
        if (!setups[device].scratch) {
            void *ptr = nullptr;
            FF_CUDA_OK(cudaGetSymbolAddress(&ptr, g_noAllocActs), error);
            int sms = 0;
            FF_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), error);
            if (!ptr || sms <= 0) return fail(error, "could not set up the static scratch on this device");
            setups[device].smCount = sms;
            setups[device].scratch = static_cast<uint16_t *>(ptr);
        }
        setup = setups[device];
    }

    FFContext local;  // launch bookkeeping only: owns nothing on the device
    local.device = device;
    local.smCount = setup.smCount;
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    GemvJob j0{}, j1{};
    j0.w0 = static_cast<const uint8_t *>(gate->weights);
    j0.s0 = static_cast<const uint16_t *>(gate->scales);
    j0.b0 = static_cast<const uint16_t *>(gate->biases);
    j0.w1 = static_cast<const uint8_t *>(up->weights);
    j0.s1 = static_cast<const uint16_t *>(up->scales);
    j0.b1 = static_cast<const uint16_t *>(up->biases);
    j0.in = x;
    j0.out = setup.scratch;
    j0.rows = f;
    j0.cols = d;
    j0.inStride = xStride;
    j0.outStride = f;
    j0.n = rows;
    j0.flags = kJobRoundGateUp;
    j1.w0 = static_cast<const uint8_t *>(down->weights);
    j1.s0 = static_cast<const uint16_t *>(down->scales);
    j1.b0 = static_cast<const uint16_t *>(down->biases);
    j1.in = setup.scratch;
    j1.out = y;
    j1.rows = d;
    j1.cols = f;
    j1.inStride = f;
    j1.outStride = yStride;
    j1.n = rows;
    for (uint32_t i = 0; i < (uint32_t)kMaxGemvRows; ++i)
        j0.inRow[i] = j0.outRow[i] = j1.inRow[i] = j1.outRow[i] = i < rows ? i : 0u;
    if (!launch_inline_job<true>(&local, j0, s, error)) return false;
    return launch_inline_job<false>(&local, j1, s, error);
}

