// What the products of f32 activations on tcgen05 share (k_mm_plain.cu: f16 / bf16 weights, k_mm_q6.cu: Q6_K): the split of an activation
// into three terms of a 16-bit type or six digits, and the walk over a CTA's stretch of the (tile, step) sequence.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "tc_common.cuh"

namespace tlb {

namespace plain {

using namespace tc;
constexpr int KB = 64;                  // weights of a row per box: one 128-byte swizzled line
constexpr int CONV_WARPS = 8;

__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {   // K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)64 << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// A value and what is left of it: pairs of terms as the weights' type, packed
template <bool BF16>
__device__ __forceinline__ uint32_t take_term(float &a, float &b) {
    float2 back;
    uint32_t bits;
    if (BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        bits = *reinterpret_cast<const uint32_t *>(&h);
        back = __bfloat1622float2(h);
    } else {
        const __half2 h = __floats2half2_rn(a, b);
        bits = *reinterpret_cast<const uint32_t *>(&h);
        back = __half22float2(h);
    }
    // an infinite or undefined activation stays what it is in the first term and adds nothing in the others
    a = fabsf(back.x) < __int_as_float(0x7f800000) ? a - back.x : 0.f;
    b = fabsf(back.y) < __int_as_float(0x7f800000) ? b - back.y : 0.f;
    return bits;
}

// A value of magnitude at most 2^26 in signed digits of nine bits: digit t, at 2^(18 - 9t), and what is left of it, both exact (the digit and the rest have
// no bits that the 24 of the value do not span)
constexpr int DIGITS = 6;
template <int T>
__device__ __forceinline__ uint32_t take_digit(float &a, float &b) {
    constexpr float MAGIC = 12582912.f;   // 1.5 * 2^23: adding it rounds to a whole number
    constexpr float UP = T <= 2 ? (float)(1 << (T <= 2 ? 18 - 9 * T : 0)) : 1.f / (float)(1 << (T > 2 ? 9 * T - 18 : 0)), DOWN = 1.f / UP;
    const float da = __fadd_rn(__fmaf_rn(a, DOWN, MAGIC), -MAGIC), db = __fadd_rn(__fmaf_rn(b, DOWN, MAGIC), -MAGIC);
    a = __fmaf_rn(da, -UP, a);
    b = __fmaf_rn(db, -UP, b);
    const __half2 h = __floats2half2_rn(da, db);
    return *reinterpret_cast<const uint32_t *>(&h);
}

}  // namespace plain

struct PlainParams {
    const float *x;        // activations: column n at x + n * ldx
    float *out;            // [N][ldy]
    float *partial;        // [CTA][first / last segment][N][128]
    int64_t K, M, ldx, ldy;
    int N, n_mma, acc_stride, steps, tiles, stages, tmem_cols;
    uint32_t idesc;
    int *err;
};

// where a CTA's stretch of the tiles x steps sequence begins
__device__ __forceinline__ int64_t plain_begin(int64_t c, int64_t total, int ctas) { return c * total / ctas; }

namespace plain {

// A segment is the part of the stretch that lies in one tile, a chunk up to CS steps of a segment. Every role walks the
// same chunks: body(chunk number, first step, end, whether a segment begins / ends with it).
template <int CS, class F>
__device__ __forceinline__ void walk(int steps, int g0, int g1, int tile_first, F &&body) {
    int c = 0, tile_end = (tile_first + 1) * steps;
    for (int g = g0; g < g1; tile_end += steps) {
        const int seg = g, seg_end = min(g1, tile_end);
        for (; g < seg_end; c++) {
            const int e = min(seg_end, g + CS);
            body(c, g, e, g == seg, e == seg_end);
            g = e;
        }
    }
}

// One of eight splitting warps: U columns of a chunk (CS steps of KS values) at a time, a lane holds V consecutive values of each; the
// loads of the next group (or of the next chunk's first) go out before this one is worked on, because a round trip to L2 takes
// as long as splitting three columns. AS_DIGITS: not three terms but six digits (the factor puts the largest magnitude into [2^25, 2^26]); values
// that these do not hold to the last bit (not finite, all below 2^-95, or with bits 2^53 below the largest) have the factor NaN.
template <bool BF16, int NC, int KS, int CS, bool AS_DIGITS>
__device__ __forceinline__ void split_columns(const PlainParams &p, uint8_t *smem, int b_tile, int b_chunk, float (&inv)[4][NC], uint64_t (&bar_b)[2], uint64_t (&bar_bfree)[2], int w,
                                              int lane, int g0, int g1, int tile_first, volatile int *fail) {
    constexpr int V = CS * KS / 32, U = NC <= 24 ? NC / CONV_WARPS : NC / CONV_WARPS / 2;
    const int box = lane * V / KB, piece = lane * V % KB / 8, half = lane * V % 8;
    // where a lane's values of the chunk [g, e) are: column n at k + n * ldx
    struct At { int g, e, tile_end; int64_t k; };
    auto chunk = [&](int g, int tile_end) {
        At at{g, min(min(g1, tile_end), g + CS), tile_end, (int64_t)(g - tile_end + p.steps) * KS + lane * V};
        return at;
    };
    auto load = [&](float (&v)[U][V], const At &at, int col) {
        const bool live = at.g < g1 && at.k < p.K && box < KS / KB * (at.e - at.g);
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int i = 0; i < V; i += 4) {
                const bool in = live && col + u * CONV_WARPS < p.N;
                const float4 f = in ? *reinterpret_cast<const float4 *>(p.x + (int64_t)(col + u * CONV_WARPS) * p.ldx + at.k + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[u][i] = f.x; v[u][i + 1] = f.y; v[u][i + 2] = f.z; v[u][i + 3] = f.w;
            }
    };
    int c = 0, n0 = w;
    At at = chunk(g0, (tile_first + 1) * p.steps);
    float nx[U][V];
    load(nx, at, n0);
    while (at.g < g1) {
        const int buf = c & 1;
        float v[U][V];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int i = 0; i < V; i++) v[u][i] = nx[u][i];
        const bool last = n0 + U * CONV_WARPS >= p.N;
        const At to = last ? chunk(at.e, at.e == at.tile_end ? at.tile_end + p.steps : at.tile_end) : at;
        load(nx, to, last ? w : n0 + U * CONV_WARPS);
        if (n0 == w && c >= 2) mbar_wait_nap(&bar_bfree[buf], (uint32_t)(((c >> 1) & 1) ^ 1), fail, 0);
        uint8_t *tile = smem + buf * b_chunk + box * b_tile + half * 2;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int n = n0 + u * CONV_WARPS;
            if (n >= p.N) break;
            bool lost = false;
            float factor = 1.f;
            if (!BF16) {
                uint32_t m = 0;
#pragma unroll
                for (int i = 0; i < V; i++) m = max(m, __float_as_uint(v[u][i]) & 0x7fffffffu);
                m = __reduce_max_sync(0xffffffffu, m);
                const bool zero = m == 0;
                m >>= 23;
                // 2^(14 - exponent), kept within what f32 holds on both sides; 1 where nothing finite is to be scaled
                const int ex = m == 0 || m == 255 ? 0 : max(-112, min(120, (AS_DIGITS ? 152 : 141) - (int)m));
                const float sc = __uint_as_float((uint32_t)(127 + ex) << 23);
#pragma unroll
                for (int i = 0; i < V; i++) {
                    const float f = v[u][i] * sc;
                    lost |= f == 0.f && v[u][i] != 0.f;
                    v[u][i] = f;
                }
                lost |= m == 255 || (m < 32 && !zero);
                factor = __uint_as_float((uint32_t)(127 - ex) << 23);
            }
#pragma unroll
            for (int t = 0; t < (AS_DIGITS ? DIGITS : 3); t++) {
                auto take = [&](float &a, float &b) {
                    if constexpr (AS_DIGITS)
                        return t == 0 ? take_digit<0>(a, b) : t == 1 ? take_digit<1>(a, b) : t == 2 ? take_digit<2>(a, b) : t == 3 ? take_digit<3>(a, b) : t == 4 ? take_digit<4>(a, b) : take_digit<5>(a, b);
                    else return take_term<BF16>(a, b);
                };
                const int row = t * p.N + n;
                uint8_t *o = tile + row * 128 + ((piece ^ (row & 7)) << 4);
                if (V == 8) *reinterpret_cast<uint4 *>(o) = make_uint4(take(v[u][0], v[u][1]), take(v[u][2], v[u][3]), take(v[u][4 % V], v[u][5 % V]), take(v[u][6 % V], v[u][7 % V]));
                else *reinterpret_cast<uint2 *>(o) = make_uint2(take(v[u][0], v[u][1]), take(v[u][2], v[u][3]));
            }
            if constexpr (AS_DIGITS) {
#pragma unroll
                for (int i = 0; i < V; i++) lost |= v[u][i] != 0.f;
                if (__any_sync(0xffffffffu, lost)) factor = __uint_as_float(0x7fc00000u);
            }
            if (!BF16 && lane == 0) inv[c & 3][n] = factor;
        }
        if (last) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> async-proxy (MMA) reads
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_b[buf]);
            c++;
            n0 = w;
        } else {
            n0 += U * CONV_WARPS;
        }
        at = to;
    }
}

}  // namespace plain

}  // namespace tlb
