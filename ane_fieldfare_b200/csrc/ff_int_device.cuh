// Device helpers for packed INT4 (or INT8) rows against one input row on the integer tensor cores.
//
// mma.sync m16n8k32 u8 x s8 takes the codes as bytes, straight from memory: the low nibbles of a word
// are one AND away, the high ones another (they stay in place and count 16 times, which the input
// makes up for) — two integer instructions for eight codes, where bf16 operands cost eight.  The input
// row enters as integers: per group of 64 values (or per row) x = V 2^-E with |V| < 2^30, V written as four
// signed base-256 digits, one digit per MMA column.  A bf16 value has eight significant bits, so a value
// down to 2^-19 of the largest is exact, a smaller one is off by less than 2^-27 of the largest (odd codes;
// even ones 2^-31), about what a 32-bit floating sum rounds of the largest's product, its scale and its bias
// part; the integer sums themselves are exact.  Error of an expert's outputs against 64 bits, bf16 rounding
// included (2816 inputs, one of them 2^p times the rest, its weight code * scale + bias zero): p = 12 1.7e-3 to
// 1.8e-3, p = 16 2.5e-3 to 2.7e-3, p = 20 1.6e-2 to 1.9e-2 (with fp32 sums on bf16 operands 1.8e-3, 2.7e-3 to
// 4.5e-3, 3.1e-2 to 7.5e-2); 1.65e-3 without the outlier, or where scale and bias of its group are zero.
#pragma once

#include "ff_mma_device.cuh"

namespace ff {

constexpr uint32_t kDigitGroupBytes = 256;  // four digits of 64 values

__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What a group of an input row carries besides its digits.
struct alignas(8) GroupAux {
    float unit;  // 2^-E: the value of the digits' last place
    float sum;   // sum of the group's values
};

// The largest magnitude's bf16 bits among eight values.
__device__ __forceinline__ uint32_t top_exponent(const uint4 &v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) top = max(top, max(w[i] & 0x7FFFu, (w[i] >> 16) & 0x7FFFu));
    return top;
}
__device__ __forceinline__ float sum_of_run(const uint4 &v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = __uint_as_float(w[i] << 16) + __uint_as_float(w[i] & 0xFFFF0000u);
    return (p[0] + p[1]) + (p[2] + p[3]);
}
// 2^E for values up to `top` (bf16 bits): |x| < 2^(e - 126) for exponent field e, E = 156 - e held to what a
// float can carry; `unit` = 2^-E, NaN when there is an infinity or a NaN among them.
struct RowScale {
    float toInt, unit;
};
__device__ __forceinline__ RowScale row_scale(uint32_t top) {
    const int e = (int)(top >> 7), E = min(156 - e, 126);
    return RowScale{__int_as_float((E + 127) << 23), e == 255 ? __int_as_float(0x7FFFFFFF) : __int_as_float((127 - E) << 23)};
}

// Eight consecutive bf16 values `v` (run `run` of a row) as digits.  Layout of a group: digit column c (0 =
// highest) at 64 c; inside, per 16 values [even 0..6 | even 8..14 | odd 1..7 | odd 9..15] — what lane
// (column, t) of the MMA loads as 16 bytes for the low and the high nibbles of its eight packed bytes.
// INT8: values in their own order.
template <bool INT8>
__device__ __forceinline__ void digits_store(int run, const uint4 &v, float scale, uint8_t *digits) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const float scaleOdd = INT8 ? scale : scale * 0.0625f;
    uint32_t U[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        // balanced digits: bytes of V + 0x808080, the lower three less 128
        const float x = __uint_as_float((i & 1) ? w[i >> 1] & 0xFFFF0000u : w[i >> 1] << 16);
        const uint32_t V = (uint32_t)__float2int_rn(x * ((i & 1) ? scaleOdd : scale));
        U[i] = (V + 0x00808080u) ^ 0x00808080u;
    }
    // (INT8: a run is eight bytes, 16 t + 0..3 | 4..7 | 8..11 | 12..15 of a quarter)
    uint8_t *dst = digits + (size_t)(run >> 3) * kDigitGroupBytes + (run & 7) / 2 * 16 + (run & 1) * (INT8 ? 8 : 4);
#pragma unroll
    for (int odd = 0; odd < 2; ++odd) {
        const uint32_t u0 = INT8 ? U[4 * odd] : U[odd], u1 = INT8 ? U[4 * odd + 1] : U[2 + odd],
                       u2 = INT8 ? U[4 * odd + 2] : U[4 + odd], u3 = INT8 ? U[4 * odd + 3] : U[6 + odd];
        const uint32_t l0 = __byte_perm(u0, u1, 0x5140), l1 = __byte_perm(u2, u3, 0x5140);
        const uint32_t h0 = __byte_perm(u0, u1, 0x7362), h1 = __byte_perm(u2, u3, 0x7362);
        uint8_t *at = dst + odd * (INT8 ? 4 : 8);
        *reinterpret_cast<uint32_t *>(at + 192) = __byte_perm(l0, l1, 0x5410);
        *reinterpret_cast<uint32_t *>(at + 128) = __byte_perm(l0, l1, 0x7632);
        *reinterpret_cast<uint32_t *>(at + 64) = __byte_perm(h0, h1, 0x5410);
        *reinterpret_cast<uint32_t *>(at) = __byte_perm(h0, h1, 0x7632);
    }
}

// A run with its group's own scale, and the group's `aux` (runs of a group in eight adjacent lanes; called by
// whole warps, `valid` false for lanes past the row).
template <bool INT8 = false>
__device__ __forceinline__ void digits_put(int run, bool valid, const uint4 &v, uint8_t *digits, GroupAux *aux) {
    uint32_t top = top_exponent(v);
    float sum = sum_of_run(v);
#pragma unroll
    for (int o = 1; o <= 4; o <<= 1) {
        top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    if (!valid) return;
    const RowScale scale = row_scale(top);
    digits_store<INT8>(run, v, scale.toInt, digits);
    if ((run & 7) == 0) *aux = GroupAux{scale.unit, sum};
}

// (shared-memory addresses: the tile function is not inlined, so a pointer would be a generic one)
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// Scales and biases as the kernels read them: u32 scale | bias << 16 per (row, group), the groups of a
// row padded to a multiple of four (ff_load_layer lays them out once, tile by tile).
__host__ __device__ inline uint32_t padded_groups(uint32_t groups) { return (groups + 3u) & ~3u; }
// Groups [begin, end) of part p when `groups` are split into `parts` runs of even length (64-bit reads of
// two groups' scales).
__host__ __device__ inline void even_range(int groups, int parts, int p, int &begin, int &end) {
    const int per = ((groups + parts - 1) / parts + 1) & ~1;
    begin = min(groups, p * per);
    end = min(groups, begin + per);
}

// N consecutive groups of a 16-row tile (N even, or the last ones): lo / hi this lane's eight packed
// bytes of tile rows g and g + 8 (g = lane / 4, t = lane % 4: bytes [8 t, + 8) of the group's 32; next
// group 32 bytes on), dig this lane's 16 digit bytes of MMA column g, sb0 / sb1 the scale | bias words of
// its row(s), aux its input's groups; all shared-memory addresses.
//   PAIR = false: one input, its digits in columns 0..3 (lanes g < 4 load them): lane t = 0 (high digits)
//     and 1 (low) account for both rows, acc[0] and acc[1].
//   PAIR = true: two inputs, columns 0..3 and 4..7: lanes t < 2 account for row g with the first, t >= 2
//     for row g + 8 with the second, acc[0]; aux and sb0 are that row's.
// Shared-memory bandwidth bounds this (512 bytes of codes and 256 or 512 of digits per group), so the
// small operands come two groups at a time.
template <int N, bool PAIR>
__device__ __forceinline__ void groups_int4(uint32_t lo, uint32_t hi, uint32_t dig, uint32_t sb0, uint32_t sb1, uint32_t aux,
                                            bool useDigits, bool lower, float (&acc)[2], float (&accBias)[2]) {
    constexpr int N2 = (N + 1) / 2;
    uint2 wl[N], wh[N], s0[N2], s1[N2];
    uint4 x[N], ax[N2];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        wl[u] = lds64(lo + 32 * u);
        wh[u] = lds64(hi + 32 * u);
        x[u] = make_uint4(0, 0, 0, 0);
        if (PAIR || useDigits) x[u] = lds128(dig + kDigitGroupBytes * u);
    }
#pragma unroll
    for (int u = 0; u < N2; ++u) {
        ax[u] = lds128(aux + 16 * u);
        s0[u] = lds64(sb0 + 8 * u);
        if (!PAIR) s1[u] = lds64(sb1 + 8 * u);
    }
    int d[N][4];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        d[u][0] = d[u][1] = d[u][2] = d[u][3] = 0;
        mma_u8s8(d[u], wl[u].x & 0x0F0F0F0Fu, wh[u].x & 0x0F0F0F0Fu, wl[u].y & 0x0F0F0F0Fu, wh[u].y & 0x0F0F0F0Fu, x[u].x, x[u].y);
    }
#pragma unroll
    for (int u = 0; u < N; ++u)
        mma_u8s8(d[u], wl[u].x & 0xF0F0F0F0u, wh[u].x & 0xF0F0F0F0u, wl[u].y & 0xF0F0F0F0u, wh[u].y & 0xF0F0F0F0u, x[u].z, x[u].w);
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const float unit = __uint_as_float((u & 1) ? ax[u >> 1].z : ax[u >> 1].x), sum = __uint_as_float((u & 1) ? ax[u >> 1].w : ax[u >> 1].y);
        const uint32_t w0 = (u & 1) ? s0[u >> 1].y : s0[u >> 1].x;
        const int v0 = PAIR ? (lower ? d[u][0] : d[u][2]) * 256 + (lower ? d[u][1] : d[u][3]) : d[u][0] * 256 + d[u][1];
        acc[0] = fmaf(__uint_as_float(w0 << 16) * unit, (float)v0, acc[0]);
        accBias[0] = fmaf(__uint_as_float(w0 & 0xFFFF0000u), sum, accBias[0]);
        if (!PAIR) {
            const uint32_t w1 = (u & 1) ? s1[u >> 1].y : s1[u >> 1].x;
            acc[1] = fmaf(__uint_as_float(w1 << 16) * unit, (float)(d[u][2] * 256 + d[u][3]), acc[1]);
            accBias[1] = fmaf(__uint_as_float(w1 & 0xFFFF0000u), sum, accBias[1]);
        }
    }
}

// `n` consecutive groups of a 16-row tile, in ascending order.  PAIR = false: x = row g, y = row g + 8 in
// lanes t = 0; PAIR = true: x = row g in lanes t = 0, row g + 8 in lanes t = 2 (other lanes hold parts).
template <bool PAIR>
static __device__ __noinline__ float2 tile_int4(uint32_t lo, uint32_t hi, uint32_t dig, uint32_t sb0, uint32_t sb1, uint32_t aux, int n) {
    const bool lower = (threadIdx.x & 3) < 2, useDigits = (threadIdx.x & 31) < 16;
    float acc[2] = {0.0f, 0.0f}, accBias[2] = {0.0f, 0.0f};
#pragma unroll 1
    for (; n >= 4; n -= 4) {
        groups_int4<4, PAIR>(lo, hi, dig, sb0, sb1, aux, useDigits, lower, acc, accBias);
        lo += 128;
        hi += 128;
        dig += 4 * kDigitGroupBytes;
        sb0 += 16;
        sb1 += 16;
        aux += 32;
    }
    // the rest in one batch, so that its latencies overlap
    if (n == 3) groups_int4<3, PAIR>(lo, hi, dig, sb0, sb1, aux, useDigits, lower, acc, accBias);
    else if (n == 2) groups_int4<2, PAIR>(lo, hi, dig, sb0, sb1, aux, useDigits, lower, acc, accBias);
    else if (n == 1) groups_int4<1, PAIR>(lo, hi, dig, sb0, sb1, aux, useDigits, lower, acc, accBias);
    const float x = fmaf(acc[0], 65536.0f, __shfl_xor_sync(0xFFFFFFFFu, acc[0], 1)) + accBias[0];
    const float y = PAIR ? 0.0f : fmaf(acc[1], 65536.0f, __shfl_xor_sync(0xFFFFFFFFu, acc[1], 1)) + accBias[1];
    return make_float2(x, y);
}

}  // namespace ff
