// MUL_MAT of every shape and weight type that no specialised kernel takes (reference: crates/kernels/src/cuda/lower.rs:543-571
// and native/mm.cu, whose semantics are y[m,n] = sum_k dq(W[k,m]) x[k,n]): strided or broadcast batches, rows that are not
// whole super-blocks, plain weights with odd rows. Q8_0, Q4_0 and Q4_K weights take quantized activations like the
// reference's CPU backend (ggml-cpu.c:1272-1357), the others the f32 values.
#include <cuda_fp16.h>
#include <cuda_bf16.h>

#include "kernels.h"
#include "dequant.cuh"

namespace tlb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    return v;
}

// ---------------------------------------------------------------- generic strided / batched product
// One warp per output element; lanes walk the row's blocks. Handles every shape the streaming
// kernel does not (K not a multiple of 256, strided or broadcast batches, plain weight types).
__device__ __forceinline__ void scale_min_k4(int j, const uint8_t *q, int &d, int &m) {
    if (j < 4) {
        d = q[j] & 63;
        m = q[j + 4] & 63;
    } else {
        d = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4);
        m = (q[j + 4] >> 4) | ((q[j] >> 6) << 4);
    }
}

__global__ void __launch_bounds__(128) k_mm_generic(MMGeneric p, const uint8_t *__restrict__ W, const uint8_t *__restrict__ X,
                                                     uint8_t *__restrict__ Y) {
    const int lane = threadIdx.x & 31;
    const int64_t m = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int64_t M = p.y.ne[0], N = p.y.ne[1], K = p.w.ne[0];
    if (m >= M) return;
    const int64_t n = blockIdx.y % N, i2 = (blockIdx.y / N) % p.y.ne[2], i3 = blockIdx.z;
    const uint8_t *wrow = W + m * p.w.nb[1] + (i2 / p.r2) * p.w.nb[2] + (i3 / p.r3) * p.w.nb[3];
    float f = 0.f;
    if (p.wtype == TLB_TYPE_F32 || p.wtype == TLB_TYPE_F16 || p.wtype == TLB_TYPE_BF16) {
        const uint8_t *xcol = X + n * p.x.nb[1] + i2 * p.x.nb[2] + i3 * p.x.nb[3];
        for (int64_t k = lane; k < K; k += 32) {
            float wv;
            if (p.wtype == TLB_TYPE_F32) wv = reinterpret_cast<const float *>(wrow)[k];
            else if (p.wtype == TLB_TYPE_F16) wv = __half2float(reinterpret_cast<const __half *>(wrow)[k]);
            else wv = __bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(wrow)[k]);
            f += wv * *reinterpret_cast<const float *>(xcol + k * p.x.nb[0]);
        }
    } else if (p.wtype != TLB_TYPE_Q8_0 && p.wtype != TLB_TYPE_Q4_0 && p.wtype != TLB_TYPE_Q4_K) {
        // the other block types: decoded weights times the f32 activations, the reference executor's own arithmetic
        // for every type (crates/kernels/src/cuda/native/mm.cu:16-42)
        const uint8_t *xcol = X + n * p.x.nb[1] + i2 * p.x.nb[2] + i3 * p.x.nb[3];
        for (int64_t k = lane; k < K; k += 32) f += dq_elem(wrow, p.wtype, k) * *reinterpret_cast<const float *>(xcol + k * p.x.nb[0]);
    } else {
        const int64_t col = n + N * (i2 + p.y.ne[2] * i3);  // column of the quantized activation block
        const char *ab = (const char *)p.act;
        const int8_t *aq = (const int8_t *)(ab + p.a.qs_off) + col * K;
        const float *ad = (const float *)(ab + p.a.d_off);
        if (p.wtype == TLB_TYPE_Q8_0) {
            for (int64_t b = lane; b < K / 32; b += 32) {
                const uint8_t *blk = wrow + b * 34;
                const float d = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t *>(blk)));
                const int8_t *qs = reinterpret_cast<const int8_t *>(blk + 2);
                int s = 0;
                for (int j = 0; j < 32; j++) s += (int)qs[j] * (int)aq[b * 32 + j];
                f += (float)s * (d * ad[col * (K / 32) + b]);
            }
        } else if (p.wtype == TLB_TYPE_Q4_0) {
            for (int64_t b = lane; b < K / 32; b += 32) {
                const uint8_t *blk = wrow + b * 18;
                const float d = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t *>(blk)));
                int s = 0;
                for (int j = 0; j < 16; j++) {
                    s += ((int)(blk[2 + j] & 0x0F) - 8) * (int)aq[b * 32 + j];
                    s += ((int)(blk[2 + j] >> 4) - 8) * (int)aq[b * 32 + j + 16];
                }
                f += (float)s * d * ad[col * (K / 32) + b];
            }
        } else {  // Q4_K, one (super-block, sub-block) per lane step
            const int16_t *bs = (const int16_t *)(ab + p.a.bsum_off) + col * (K / 16);
            for (int64_t u = lane; u < K / 32; u += 32) {
                const int64_t sb = u >> 3;
                const int j = (int)(u & 7);
                const uint8_t *blk = wrow + sb * 144;
                const float d = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t *>(blk)));
                const float dmin = __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t *>(blk + 2)));
                int sc, mn;
                scale_min_k4(j, blk + 4, sc, mn);
                const uint8_t *q = blk + 16 + (j >> 1) * 32;
                const int shift = (j & 1) * 4;
                int s = 0;
                for (int l = 0; l < 32; l++) s += (int)((q[l] >> shift) & 0xF) * (int)aq[sb * 256 + j * 32 + l];
                const int bsum = (int)bs[sb * 16 + 2 * j] + (int)bs[sb * 16 + 2 * j + 1];
                f += ad[col * (K / 256) + sb] * (d * (float)(sc * s) - dmin * (float)(mn * bsum));
            }
        }
    }
    f = warp_sum(f);
    if (lane == 0) *reinterpret_cast<float *>(Y + m * p.y.nb[0] + n * p.y.nb[1] + i2 * p.y.nb[2] + i3 * p.y.nb[3]) = f;
}

cudaError_t launch_mm_generic(const MMGeneric &p, const void *W, const void *X, void *Y, cudaStream_t st) {
    const int64_t M = p.y.ne[0], N = p.y.ne[1];
    if (M == 0 || N == 0) return cudaSuccess;
    dim3 grid((unsigned)((M + 3) / 4), (unsigned)(N * p.y.ne[2]), (unsigned)p.y.ne[3]);
    k_mm_generic<<<grid, 128, 0, st>>>(p, (const uint8_t *)W, (const uint8_t *)X, (uint8_t *)Y);
    return cudaGetLastError();
}

}  // namespace tlb
