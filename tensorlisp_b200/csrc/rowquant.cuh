// Row sources and the Q8_K block quantizer shared by the row-producing kernels (k_fused.cu), the few-column mul_mat (k_gemv.cu)
// and the attention epilogue (k_attn.cu).
#pragma once
#include <cuda_fp16.h>

#include "kernels.h"

namespace tlb {

__device__ __forceinline__ int nearest_int_f(float v) {
    float t = __fadd_rn(v, 12582912.f);
    return (__float_as_int(t) & 0x007fffff) - 0x00400000;
}


// The f32 value at (column n, element k) before any normalisation: a, a + b, act(a) * b or f16 a.
// PLAIN: the caller knows the mode to be RQ_PLAIN or RQ_NORM (eight exponentials and divisions at every place that loads a row are most of
// a kernel's code, and a kernel of a few microseconds waits for its code).
template <bool PLAIN = false>
__device__ __forceinline__ void rq_load8(const RowQuantArgs &p, int n, int64_t k0, float (&x)[8]) {
    if (!PLAIN && p.mode == RQ_GLU) {
        const float4 g0 = *reinterpret_cast<const float4 *>(p.a + n * p.lda + k0), g1 = *reinterpret_cast<const float4 *>(p.a + n * p.lda + k0 + 4);
        const float4 u0 = *reinterpret_cast<const float4 *>(p.b + n * p.ldb + k0), u1 = *reinterpret_cast<const float4 *>(p.b + n * p.ldb + k0 + 4);
        const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
        for (int e = 0; e < 8; e++) x[e] = __fmul_rn(__fdiv_rn(g[e], __fadd_rn(1.0f, expf(-g[e]))), u[e]);   // SiLU(g)*u
    } else if (!PLAIN && p.mode == RQ_F16) {
        const uint4 h = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __half *>(p.a) + n * p.lda + k0);
        const __half2 *h2 = reinterpret_cast<const __half2 *>(&h);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float2 f = __half22float2(h2[e]);
            x[2 * e] = f.x;
            x[2 * e + 1] = f.y;
        }
    } else {
        const float4 a0 = *reinterpret_cast<const float4 *>(p.a + n * p.lda + k0), a1 = *reinterpret_cast<const float4 *>(p.a + n * p.lda + k0 + 4);
        x[0] = a0.x; x[1] = a0.y; x[2] = a0.z; x[3] = a0.w; x[4] = a1.x; x[5] = a1.y; x[6] = a1.z; x[7] = a1.w;
        if (p.b) {   // residual add: x = a + b
            const float4 b0 = *reinterpret_cast<const float4 *>(p.b + n * p.ldb + k0), b1 = *reinterpret_cast<const float4 *>(p.b + n * p.ldb + k0 + 4);
            x[0] = __fadd_rn(x[0], b0.x); x[1] = __fadd_rn(x[1], b0.y); x[2] = __fadd_rn(x[2], b0.z); x[3] = __fadd_rn(x[3], b0.w);
            x[4] = __fadd_rn(x[4], b1.x); x[5] = __fadd_rn(x[5], b1.y); x[6] = __fadd_rn(x[6], b1.z); x[7] = __fadd_rn(x[7], b1.w);
        }
    }
}

// Codes and scale of one 256-value block held by a warp (lane l: values l*8 .. l*8+7; quantize_row_q8_K_ref, ggml-quants.c:2768-2805)
__device__ __forceinline__ void rq_q8k(int lane, const float (&v)[8], int (&q)[8], float &d) {
    float amax = 0.f, mx = 0.f;
    int idx = 512;
#pragma unroll
    for (int e = 0; e < 8; e++)
        if (fabsf(v[e]) > amax) { amax = fabsf(v[e]); mx = v[e]; idx = lane * 8 + e; }
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, amax, s), om = __shfl_xor_sync(0xffffffffu, mx, s);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, s);
        if (oa > amax || (oa == amax && oi < idx)) { amax = oa; mx = om; idx = oi; }
    }
    d = 0.f;
    if (amax == 0.f) {
#pragma unroll
        for (int e = 0; e < 8; e++) q[e] = 0;
    } else {
        const float iscale = __fdiv_rn(-127.f, mx);
#pragma unroll
        for (int e = 0; e < 8; e++) q[e] = min(127, nearest_int_f(__fmul_rn(iscale, v[e])));
        d = __fdiv_rn(1.f, iscale);
    }
}

// Q8_K quantization of one 256-value block held by a warp (lane l: values l*8 .. l*8+7), its optional f32
// copy, and its slice of the tensor-core operand blob
__device__ __forceinline__ void rq_quant_block(const RowQuantArgs &p, int n, int sb, int nblk, int lane, float (&v)[8]) {
    char *ob = (char *)p.out;
    const int64_t K = p.K;
    const int64_t k0 = (int64_t)sb * 256 + lane * 8;
    int8_t *qs = (int8_t *)(ob + p.qs_off);
    float *ds = (float *)(ob + p.d_off);
    int16_t *bsums = (int16_t *)(ob + p.bsum_off);
    if (p.y_out) {
        *reinterpret_cast<float4 *>(p.y_out + n * p.ld_y + k0) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(p.y_out + n * p.ld_y + k0 + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    int q[8];
    float d;
    rq_q8k(lane, v, q, d);
    int s8 = 0;
#pragma unroll
    for (int e = 0; e < 8; e++) s8 += q[e];
    const int s16 = s8 + __shfl_xor_sync(0xffffffffu, s8, 1);
    uint2 packed;
    packed.x = (uint32_t)(q[0] & 0xff) | ((uint32_t)(q[1] & 0xff) << 8) | ((uint32_t)(q[2] & 0xff) << 16) | ((uint32_t)(q[3] & 0xff) << 24);
    packed.y = (uint32_t)(q[4] & 0xff) | ((uint32_t)(q[5] & 0xff) << 8) | ((uint32_t)(q[6] & 0xff) << 16) | ((uint32_t)(q[7] & 0xff) << 24);
    if (!p.operand_only) {
        *reinterpret_cast<uint2 *>(qs + (size_t)n * K + k0) = packed;
        if ((lane & 1) == 0) bsums[(size_t)n * (K / 16) + sb * 16 + (lane >> 1)] = (int16_t)s16;
        if (lane == 0) ds[(size_t)n * (K / 256) + sb] = d;
    }
    if (p.npad == MM_FOLD_NPAD) {
        // operand of the folded-scale prompt GEMM: f16(code x scale) in natural order
        const int64_t kk = (int64_t)sb * 256 + lane * 8;
        uint8_t *o = (uint8_t *)ob + p.blob_off + mm_fold_at(n, kk, mm_fold_groups(p.N));
        uint32_t h[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const __half2 t = __floats2half2_rn(__fmul_rn((float)q[2 * e], d), __fmul_rn((float)q[2 * e + 1], d));
            h[e] = *reinterpret_cast<const uint32_t *>(&t);
        }
        *reinterpret_cast<uint4 *>(o) = make_uint4(h[0], h[1], h[2], h[3]);
    } else if (p.npad > 0) {
        // tensor-core operand: this lane's 8 codes are K chunk `lane` of column n, in the order
        // (0, 2, 1, 3, 4, 6, 5, 7) in which the weight nibbles come out of a 32-bit word
        const int ch = n / p.npad, nl = n % p.npad;   // blobs: [chunk of npad columns][block]
        uint8_t *o = (uint8_t *)ob + p.blob_off + ((size_t)ch * nblk + sb) * p.blob_bytes;
        __half2 h[4];
        h[0] = __floats2half2_rn((float)q[0], (float)q[2]);
        h[1] = __floats2half2_rn((float)q[1], (float)q[3]);
        h[2] = __floats2half2_rn((float)q[4], (float)q[6]);
        h[3] = __floats2half2_rn((float)q[5], (float)q[7]);
        *reinterpret_cast<uint4 *>(o + (size_t)(nl / 8) * 4096 + lane * 128 + (nl % 8) * 16) = *reinterpret_cast<const uint4 *>(h);
        if ((lane & 1) == 0)
            *reinterpret_cast<__half *>(o + (size_t)p.npad * 512 + (size_t)(nl / 8) * 256 + (lane >> 4) * 128 + (nl % 8) * 16 + ((lane >> 1) & 7) * 2) = __float2half_rn((float)s16);
        if (lane == 0) reinterpret_cast<float *>(o + (size_t)p.npad * 544)[nl] = d;
    }
}

}  // namespace tlb
