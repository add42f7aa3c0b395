// MUL_MAT with Q8_0, Q4_0 or Q4_K weights and up to eight activation columns (token generation for one or a few users; k_gemv_f32.cu
// has Q6_K, few_column_faster the line to the tcgen05 kernels):
// every weight byte is read once, everything else hides behind that or is fixed cost.
//
// Arithmetic follows the reference's CPU backend (ggml-cpu.c:1272-1357): activations become int8 blocks, every output is an
// integer dot product per block scaled in f32 (ggml-cpu/quants.c:451-479 for Q8_0, :225-260 for Q4_0, :696-770 for Q4_K); only
// the order of the f32 additions differs.
//
// One kernel does what used to be three to six launches: the producer of the activation (residual add + RMS norm, gate, f16
// cast), its quantizer, up to three matrices that read it, and SiLU(gate) * up behind a gate / up pair. At one column a
// launch and its ramp cost 4 to 5 us, a layer matrix of 9 to 33 MB streams in 2 to 5 us, and a row of activations is a few KB: so
// every CTA produces and quantizes one or two rows for itself, while its first weights are already on their way (more
// columns are quantized by a launch in front, which has all SMs for it).
//
// The integer pipe bounds the unpacking: it takes an instruction every other cycle, dp4a and the masks of the nibbles alike
// (dp4a version: 8 us for the 33 MB of a [14336 x 4096] Q4_K matrix, of which the stream needs 5). So the dot products go to
// the integer matrix instruction: m16n8k32 takes 16 rows x 32 codes against up to eight columns in 8 cycles of a pipe of its own,
// straight from registers.
//
// Layout of the work: one CTA per SM takes a contiguous range of rows (whole groups of eight), so all finish together whatever
// the row count. A producer thread copies tiles of 16 rows x up to 2048 weights through a ring; a copy's box is a little wider than
// the tile, so that the rows' distance in shared memory keeps eight of them on different banks (what it brings of the next
// tile comes from L2 again). Each of eight warps takes 256 weights of the tile's 16 rows; the sums over a row's tiles stay in
// registers, the eight warps' parts meet in shared memory once at the end. Registers and shared memory are sized
// for two CTAs per SM: the next launch's CTA starts beside this one (programmatic dependent launch) and fills its ring while
// this one drains.
#include <algorithm>
#include <cuda_fp16.h>

#include "kernels.h"
#include "pdl.cuh"
#include "rowquant.cuh"
#include "tc_common.cuh"

namespace tlb {

cudaError_t tc_encode_2d_bytes(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows);

namespace gemv {

using namespace tc;   // mbarriers and copies

constexpr int WARPS = 8;                      // consumers
constexpr int THREADS = 32 * (WARPS + 1);     // and the producer
constexpr int MAX_STAGES = 16;
constexpr int MAX_COLS = (int)GEMV_MAX_COLS;
constexpr int PART_BYTES = 8 * 1024;          // partial sums before they are added up

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory"); }
// 16 rows x 32 codes times 32 codes x 8 columns; A as unsigned or signed bytes. (The zero addend is an operand of its own, so that
// it costs no register moves.)
template <bool U8>
__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    if (U8)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(0));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(0));
}
// two 16-bit values times bytes 0, 1 (lo) or 2, 3 (hi) of b
__device__ __forceinline__ int dp2a_lo(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp2a.lo.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int dp2a_hi(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp2a.hi.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

struct Maps {
    CUtensorMap m[3];
};
struct Params {
    float *y[3];            // [column][ldy[j]]; with glu only y[0]
    int64_t ldy[3];
    int M[3];
    int n_mats, glu;        // glu: matrices 0 and 1 are gate and up of equal size, y[0] = SiLU(gate) * up
    int K, unit_bytes;                 // a unit: 256 weights of a row
    int units, seg_units, segs;        // of a row; of a tile; tiles per row group
    int groups;                        // row groups of 16 in a tile (more than one where a row has less than eight units)
    int sets, stages_per_set, stage_stride, row_stride;   // a set of warps takes whole row groups and has a ring of its own
    int epoch;                         // row groups (per set and tile slot) between two additions of the parts
    int act_stride, d_off, bsum_off;   // per column in shared memory: codes | d | sums
    int n0, nc;                        // columns of this pass
    RowQuantArgs act;                  // where the activation rows come from; RQ_READY: an ActLayout block
    const uint8_t *ready;
    int *err;
};

// ---------------------------------------------------------------- activations into shared memory
// Codes of a column lie in the order in which a lane's 8 bytes feed the matrix instruction. Q4_K: their own (a lane takes 8
// consecutive nibble bytes of a row). Q8_0 / Q4_0: of 32 codes, bytes 4t .. 4t + 3 and 16 + 4t .. 16 + 4t + 3 side by side.
template <int TYPE>
__device__ __forceinline__ void put_codes(const Params &p, uint8_t *act, int k0, uint2 codes) {   // eight codes from k0 on
    if (TYPE == TLB_TYPE_Q4_K) {
        *reinterpret_cast<uint2 *>(act + k0) = codes;
    } else {
        uint8_t *o = act + (k0 & ~31) + ((k0 & 8) >> 2) * 8 + ((k0 & 16) >> 2);
        *reinterpret_cast<uint32_t *>(o) = codes.x;
        *reinterpret_cast<uint32_t *>(o + 8) = codes.y;
    }
}

// B blocks of 256 values, WARPS blocks apart (a lane has eight of each), into the codes, scales and sums of a column. One block is a
// chain of about 700 cycles (reductions, two divisions), so every step is taken for all B before the next one.
template <int TYPE, int B>
__device__ __forceinline__ void store_blocks(const Params &p, uint8_t *act, int sb0, int nblk, int lane, const float (&v)[B][8]) {
    float *d_out = reinterpret_cast<float *>(act + p.d_off);
    float amax[B], mul[B], d[B];
    if (TYPE == TLB_TYPE_Q4_K) {   // quantize_row_q8_K_ref (ggml-quants.c:2768-2805), as in rq_quant_block
        // the first value of the largest magnitude (a magnitude's bits order like the magnitude). Its sign is plain unless both
        // signs reach it
        float hi[B], lo[B];
#pragma unroll
        for (int h = 0; h < B; h++) {
            hi[h] = fmaxf(fmaxf(fmaxf(v[h][0], v[h][1]), fmaxf(v[h][2], v[h][3])), fmaxf(fmaxf(v[h][4], v[h][5]), fmaxf(v[h][6], v[h][7])));
            lo[h] = fminf(fminf(fminf(v[h][0], v[h][1]), fminf(v[h][2], v[h][3])), fminf(fminf(v[h][4], v[h][5]), fminf(v[h][6], v[h][7])));
            amax[h] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(hi[h]), fabsf(lo[h])))));
        }
#pragma unroll
        for (int h = 0; h < B; h++) {
            const uint32_t pos = __ballot_sync(0xffffffffu, hi[h] == amax[h]), neg = __ballot_sync(0xffffffffu, lo[h] == -amax[h]);
            float mx = neg == 0 ? amax[h] : -amax[h];
            if (pos != 0 && neg != 0) {
                float first = 0.f;
#pragma unroll
                for (int e = 7; e >= 0; e--)
                    if (fabsf(v[h][e]) == amax[h]) first = v[h][e];
                mx = __shfl_sync(0xffffffffu, first, __ffs(pos | neg) - 1);
            }
            mul[h] = amax[h] != 0.f ? __fdiv_rn(-127.f, mx) : 0.f;
        }
#pragma unroll
        for (int h = 0; h < B; h++) d[h] = amax[h] != 0.f ? __fdiv_rn(1.f, mul[h]) : 0.f;
    } else {                       // quantize_row_q8_0_ref (ggml-quants.c:276-299)
#pragma unroll
        for (int h = 0; h < B; h++) {
            amax[h] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; e++) amax[h] = fmaxf(amax[h], fabsf(v[h][e]));
            amax[h] = fmaxf(amax[h], __shfl_xor_sync(0xffffffffu, amax[h], 1));
            amax[h] = fmaxf(amax[h], __shfl_xor_sync(0xffffffffu, amax[h], 2));
            d[h] = __fdiv_rn(amax[h], 127.f);
        }
#pragma unroll
        for (int h = 0; h < B; h++) mul[h] = d[h] != 0.f ? __fdiv_rn(1.0f, d[h]) : 0.0f;
    }
#pragma unroll
    for (int h = 0; h < B; h++) {
        const int sb = sb0 + h * WARPS;
        int q[8], s8 = 0;
#pragma unroll
        for (int e = 0; e < 8; e++) {
            q[e] = TYPE == TLB_TYPE_Q4_K ? min(127, nearest_int_f(__fmul_rn(mul[h], v[h][e]))) : (int)roundf(__fmul_rn(v[h][e], mul[h]));
            s8 += q[e];
        }
        if (TYPE == TLB_TYPE_Q4_K) {
            s8 += __shfl_xor_sync(0xffffffffu, s8, 1);
            s8 += __shfl_xor_sync(0xffffffffu, s8, 2);   // a sub-block: at most 32 x 127
        }
        if (sb >= nblk) break;
        if (TYPE == TLB_TYPE_Q4_K) {
            if ((lane & 3) == 0) reinterpret_cast<int16_t *>(act + p.bsum_off)[sb * 8 + (lane >> 2)] = (int16_t)s8;
            if (lane == 0) d_out[sb] = d[h];
        } else if ((lane & 3) == 0) {
            d_out[sb * 8 + (lane >> 2)] = __half2float(__float2half_rn(d[h]));
        }
        uint2 packed;
        packed.x = (uint32_t)(q[0] & 0xff) | ((uint32_t)(q[1] & 0xff) << 8) | ((uint32_t)(q[2] & 0xff) << 16) | ((uint32_t)(q[3] & 0xff) << 24);
        packed.y = (uint32_t)(q[4] & 0xff) | ((uint32_t)(q[5] & 0xff) << 8) | ((uint32_t)(q[6] & 0xff) << 16) | ((uint32_t)(q[7] & 0xff) << 24);
        put_codes<TYPE>(p, act, sb * 256 + lane * 8, packed);
    }
}

// The rows of this pass. RQ_READY: codes, scales and sums another launch has left in an ActLayout block. Otherwise they are
// produced and quantized here: sums of squares in the order of k_row_quant_q8k (256 threads, stretches of 2048), so that rows from
// here and from the row quantizers agree in every bit. (k_norm, for a norm that is not folded, adds in another order: its scale may
// differ by an ulp.)
template <int TYPE>
__device__ __forceinline__ void load_activations(const Params &p, uint8_t *act, float *red) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const RowQuantArgs &a = p.act;
    const int nblk = p.K / 256;
    if (a.mode == RQ_READY) {
        griddep_wait();
        const int8_t *qs = reinterpret_cast<const int8_t *>(p.ready + a.qs_off);
        const float *ds = reinterpret_cast<const float *>(p.ready + a.d_off);
        const int16_t *bs = reinterpret_cast<const int16_t *>(p.ready + a.bsum_off);
        const int nd = TYPE == TLB_TYPE_Q4_K ? nblk : p.K / 32;
        for (int n = 0; n < p.nc; n++) {
            uint8_t *o = act + (size_t)n * p.act_stride;
            const int8_t *q = qs + (int64_t)(p.n0 + n) * p.K;
#pragma unroll 4
            for (int k = tid * 16; k < p.K; k += WARPS * 32 * 16) {
                const uint4 v = *reinterpret_cast<const uint4 *>(q + k);
                put_codes<TYPE>(p, o, k, make_uint2(v.x, v.y));
                put_codes<TYPE>(p, o, k + 8, make_uint2(v.z, v.w));
            }
            for (int i = tid; i < nd; i += WARPS * 32) reinterpret_cast<float *>(o + p.d_off)[i] = ds[(int64_t)(p.n0 + n) * nd + i];
            if (TYPE == TLB_TYPE_Q4_K)
                for (int i = tid; i < p.K / 32; i += WARPS * 32) {
                    const int16_t *b = bs + (int64_t)(p.n0 + n) * (p.K / 16) + 2 * i;
                    reinterpret_cast<int16_t *>(o + p.bsum_off)[i] = (int16_t)(b[0] + b[1]);
                }
        }
        consumers_sync();
        return;
    }
    constexpr int Q = 2, B = 2;   // turns ahead, blocks of a turn
    auto block_at = [&](int turn, int h) { return turn * (B * WARPS) + h * WARPS + warp; };
    if (a.mode == RQ_NORM)        // not written by the kernel in front, and in HBM as a rule
        for (int k = tid * 32; k < (int)a.wn; k += WARPS * 32 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.w + k));
    // n = -1 is a rehearsal on zeros, one turn long, while the kernel in front is still running: the code runs once per launch and
    // is bound by fetching it otherwise (about 1000 cycles of the 1760 before the first block was reached). Behind a norm only, where
    // the code is longest and a whole layer's part runs in front: a batch-1 decode step 2394 -> 2309 us; a product right behind
    // another one would wait for its own rehearsal (1 us).
    float scale = 1.f;
#pragma unroll 1
    for (int n = a.mode == RQ_NORM ? -1 : 0; n < p.nc; n++) {
        const bool real = n >= 0;
        if (n == 0) griddep_wait();
        uint8_t *const out = act + (size_t)max(n, 0) * p.act_stride;
        const int n_in = p.n0 + max(n, 0), blocks = real ? nblk : min(nblk, B * WARPS);
        float nx[Q][B][8] = {};
        if (real) {
#pragma unroll
            for (int i = 0; i < Q * B; i++)
                if (block_at(i / B, i % B) < nblk) rq_load8(a, n_in, (int64_t)block_at(i / B, i % B) * 256 + lane * 8, nx[i / B][i % B]);
        }
        if (a.mode == RQ_NORM) {
            float ss = 0.f;
            if (nblk <= Q * B * WARPS) {   // (no values: zeros, which add nothing)
#pragma unroll
                for (int i = 0; i < Q * B; i++)
#pragma unroll
                    for (int e = 0; e < 8; e++) ss = __fadd_rn(ss, __fmul_rn(nx[i / B][i % B][e], nx[i / B][i % B][e]));
            } else if (real) {
#pragma unroll 2
                for (int64_t k0 = (int64_t)tid * 8; k0 < p.K; k0 += 2048) {
                    float x[8];
                    rq_load8(a, n_in, k0, x);
#pragma unroll
                    for (int e = 0; e < 8; e++) ss = __fadd_rn(ss, __fmul_rn(x[e], x[e]));
                }
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, s));
            if (lane == 0) red[(n & 1) * WARPS + warp] = ss;
            consumers_sync();
            float tot = 0.f;
#pragma unroll
            for (int i = 0; i < WARPS; i++) tot = __fadd_rn(tot, red[(n & 1) * WARPS + i]);
            scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(tot, (float)p.K), a.eps)));
        }
        // Two blocks per warp and turn in a loop that is not unrolled (four side by side: 2.5 us for a row of 4096, most of it
        // instruction fetch). What a turn waits for otherwise is L2, about 1000 cycles away: the next two turns are on their way.
#pragma unroll 1
        for (int turn = 0; block_at(turn, 0) < blocks; turn++) {
            float v[B][8];
#pragma unroll
            for (int h = 0; h < B; h++) {
                const int sb = block_at(turn, h);
                const int64_t k0 = (int64_t)sb * 256 + lane * 8;
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    v[h][e] = nx[0][h][e];
#pragma unroll
                    for (int i = 0; i + 1 < Q; i++) nx[i][h][e] = nx[i + 1][h][e];
                }
                if (real && block_at(turn + Q, h) < nblk) rq_load8(a, n_in, (int64_t)block_at(turn + Q, h) * 256 + lane * 8, nx[Q - 1][h]);
                if (sb >= nblk) continue;
                if (real && blockIdx.x == 0 && a.mode != RQ_GLU && a.mode != RQ_F16 && a.b && a.sum_out) {   // the sum is the new residual stream
                    *reinterpret_cast<float4 *>(a.sum_out + n_in * a.ld_sum + k0) = make_float4(v[h][0], v[h][1], v[h][2], v[h][3]);
                    *reinterpret_cast<float4 *>(a.sum_out + n_in * a.ld_sum + k0 + 4) = make_float4(v[h][4], v[h][5], v[h][6], v[h][7]);
                }
                if (real && a.mode == RQ_NORM) {
                    const int wi = a.wn == p.K ? (int)k0 : (int)((uint32_t)k0 % (uint32_t)a.wn);   // (norm weights come in whole groups of eight: fuse_gemv)
                    const float4 w0 = *reinterpret_cast<const float4 *>(a.w + wi), w1 = *reinterpret_cast<const float4 *>(a.w + wi + 4);
                    const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                    for (int e = 0; e < 8; e++) v[h][e] = __fmul_rn(__fmul_rn(v[h][e], scale), w[e]);
                }
            }
            store_blocks<TYPE, B>(p, out, block_at(turn, 0), blocks, lane, v);
        }
    }
    consumers_sync();
}

// ---------------------------------------------------------------- 256 weights of 16 rows
// Lane (g, t) = (lane / 4, lane % 4) brings bytes of rows g and g + 8 and of column g, and gets the sums of those rows with
// columns 2t and 2t + 1: f[0], f[1] of row g, f[2], f[3] of row g + 8. ONE: a single column, f[0] and f[2] of lanes with t = 0.
// w: row g of the tile, this warp's unit; w8: row g + 8.
// b: this lane's codes of the unit; where there is no column g, a stretch of zeros.
template <bool ONE>
__device__ __forceinline__ void unit_q4_K(const Params &p, const uint8_t *w, const uint8_t *w8, const uint8_t *b, int unit, const uint8_t *act, float (&f)[4]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    const uint4 h0 = *reinterpret_cast<const uint4 *>(w), h1 = *reinterpret_cast<const uint4 *>(w8);
    uint2 q0[4], q1[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        q0[c] = *reinterpret_cast<const uint2 *>(w + 16 + c * 32 + t * 8);
        q1[c] = *reinterpret_cast<const uint2 *>(w8 + 16 + c * 32 + t * 8);
    }
    // 6-bit scales and mins of the eight sub-blocks (get_scale_min_k4, ggml-quants.c:880-887), a byte each
    const uint32_t sc[2][2] = {{h0.y & 0x3f3f3f3fu, (h0.w & 0x0f0f0f0fu) | ((h0.y >> 2) & 0x30303030u)}, {h1.y & 0x3f3f3f3fu, (h1.w & 0x0f0f0f0fu) | ((h1.y >> 2) & 0x30303030u)}};
    const uint32_t mn[2][2] = {{h0.z & 0x3f3f3f3fu, ((h0.w >> 4) & 0x0f0f0f0fu) | ((h0.z >> 2) & 0x30303030u)}, {h1.z & 0x3f3f3f3fu, ((h1.w >> 4) & 0x0f0f0f0fu) | ((h1.z >> 2) & 0x30303030u)}};
    int lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};   // hi: of the high nibbles in place, 16 x their value
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint2 bl = *reinterpret_cast<const uint2 *>(b + c * 64), bh = *reinterpret_cast<const uint2 *>(b + c * 64 + 32);
        int d[4];
        imma<true>(d, q0[c].x & 0x0f0f0f0fu, q1[c].x & 0x0f0f0f0fu, q0[c].y & 0x0f0f0f0fu, q1[c].y & 0x0f0f0f0fu, bl);
        const int s0 = (int)__byte_perm(sc[0][c >> 1], 0, 0x4440 + (c & 1) * 2), s1 = (int)__byte_perm(sc[1][c >> 1], 0, 0x4440 + (c & 1) * 2);
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (!ONE || !(i & 1)) lo[i] += (i < 2 ? s0 : s1) * d[i];
        imma<true>(d, q0[c].x & 0xf0f0f0f0u, q1[c].x & 0xf0f0f0f0u, q0[c].y & 0xf0f0f0f0u, q1[c].y & 0xf0f0f0f0u, bh);
        const int u0 = (int)__byte_perm(sc[0][c >> 1], 0, 0x4441 + (c & 1) * 2), u1 = (int)__byte_perm(sc[1][c >> 1], 0, 0x4441 + (c & 1) * 2);
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (!ONE || !(i & 1)) hi[i] += (i < 2 ? u0 : u1) * d[i];
    }
    const float2 dm0 = __half22float2(*reinterpret_cast<const __half2 *>(&h0.x)), dm1 = __half22float2(*reinterpret_cast<const __half2 *>(&h1.x));
#pragma unroll
    for (int n = 0; n < (ONE ? 1 : 2); n++) {
        const uint8_t *a = act + (ONE ? 0 : min(2 * t + n, p.nc - 1) * p.act_stride);
        const uint4 bs = *reinterpret_cast<const uint4 *>(a + p.bsum_off + unit * 16);   // sums of the eight sub-blocks
        const float yd = reinterpret_cast<const float *>(a + p.d_off)[unit];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int m = dp2a_hi(bs.w, mn[r][1], dp2a_lo(bs.z, mn[r][1], dp2a_hi(bs.y, mn[r][0], dp2a_lo(bs.x, mn[r][0], 0))));
            const float2 dm = r ? dm1 : dm0;
            f[2 * r + n] = fmaf(yd, dm.x * (float)(lo[2 * r + n] + (hi[2 * r + n] >> 4)) - dm.y * (float)m, f[2 * r + n]);
        }
    }
}

// Eight blocks of 34 (Q8_0) or 18 (Q4_0) bytes: blocks start on 2-byte boundaries, every other one's codes on a word.
template <int TYPE, bool ONE>
__device__ __forceinline__ void unit_q_0(const Params &p, const uint8_t *w, const uint8_t *w8, const uint8_t *b, int unit, const uint8_t *act, float (&f)[4]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    const uint8_t *a0 = act + (ONE ? 0 : min(2 * t, p.nc - 1) * p.act_stride) + p.d_off + unit * 32, *a1 = act + min(2 * t + 1, p.nc - 1) * p.act_stride + p.d_off + unit * 32;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        constexpr int BB = TYPE == TLB_TYPE_Q8_0 ? 34 : 18;
        const uint32_t *s[2] = {reinterpret_cast<const uint32_t *>(w + (k * BB & ~3)), reinterpret_cast<const uint32_t *>(w8 + (k * BB & ~3))};
        const bool odd = k & 1;
        uint32_t qa[2], qb[2];   // codes 4t .. and 16 + 4t .. of rows g and g + 8
        float dw[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint32_t head = s[r][0];
            dw[r] = __half2float(__ushort_as_half((unsigned short)(odd ? head >> 16 : head & 0xffffu)));
            const uint32_t x0 = odd ? s[r][1 + t] : __funnelshift_r(s[r][t], s[r][t + 1], 16);
            if (TYPE == TLB_TYPE_Q8_0) {
                qa[r] = x0;
                qb[r] = odd ? s[r][5 + t] : __funnelshift_r(s[r][t + 4], s[r][t + 5], 16);
            } else {   // 16 x (q - 8) as signed bytes
                qa[r] = ((x0 << 4) & 0xf0f0f0f0u) ^ 0x80808080u;
                qb[r] = (x0 & 0xf0f0f0f0u) ^ 0x80808080u;
                dw[r] *= 0.0625f;
            }
        }
        int d[4];
        imma<false>(d, qa[0], qa[1], qb[0], qb[1], *reinterpret_cast<const uint2 *>(b + k * 32));
        const float y0 = reinterpret_cast<const float *>(a0)[k], y1 = ONE ? 0.f : reinterpret_cast<const float *>(a1)[k];
        f[0] = fmaf((float)d[0], dw[0] * y0, f[0]);
        f[2] = fmaf((float)d[2], dw[1] * y0, f[2]);
        if (!ONE) {
            f[1] = fmaf((float)d[1], dw[0] * y1, f[1]);
            f[3] = fmaf((float)d[3], dw[1] * y1, f[3]);
        }
    }
}

// ---------------------------------------------------------------- the kernel
// This CTA's rows of each matrix: a contiguous range of the groups of eight laid end to end (of gate and up: the same rows), in
// row groups of 16. Group i: matrix, first row, rows (0: none; the last one of a range may have eight or less).
struct Rows {
    int lo[3], hi[3], groups[3], total;
    __device__ __forceinline__ Rows(const Params &p) {
        int all = 0;
        const int nm = p.glu ? 1 : p.n_mats;
        for (int j = 0; j < nm; j++) all += (p.M[j] + 7) / 8;
        const int r0 = (int)((int64_t)all * blockIdx.x / gridDim.x), r1 = (int)((int64_t)all * (blockIdx.x + 1) / gridDim.x);
        int base = 0;
        total = 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int m = j < nm ? (p.M[j] + 7) / 8 : 0;
            const int l = min(max(r0 - base, 0), m), h = min(max(r1 - base, 0), m);
            lo[j] = l * 8;
            hi[j] = min(h * 8, j < nm ? p.M[j] : 0);
            groups[j] = (h - l + 1) / 2;
            base += m;
            total += groups[j];
        }
        if (p.glu) {
            lo[1] = lo[0];
            hi[1] = hi[0];
            total *= 2;
        }
    }
    __device__ __forceinline__ int at(const Params &p, int i, int &mat, int &row0) const {
        if (i >= total) return 0;
        if (p.glu) {
            mat = i & 1;
            i >>= 1;
        } else {
            mat = 0;
            if (i >= groups[0]) {
                i -= groups[0];
                mat = 1;
                if (i >= groups[1]) {
                    i -= groups[1];
                    mat = 2;
                }
            }
        }
        row0 = (mat == 0 ? lo[0] : (mat == 1 ? lo[1] : lo[2])) + i * 16;
        return min(16, (mat == 0 ? hi[0] : (mat == 1 ? hi[1] : hi[2])) - row0);
    }
};

template <int TYPE, bool ONE>
__global__ void __launch_bounds__(THREADS, 2) k_gemv(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES];
    __shared__ float red[2 * WARPS];
    __shared__ __align__(16) uint8_t zeros[256];
    griddep_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t *act = smem + p.sets * p.stages_per_set * p.stage_stride;
    float *part = reinterpret_cast<float *>(act + p.nc * p.act_stride);
    const Rows rows(p);
    const int lanes_per_set = p.groups * p.seg_units;   // warps of a set
    if (tid < 64) reinterpret_cast<uint32_t *>(zeros)[tid] = 0;
    if (tid == 0) {
        for (int s = 0; s < p.sets * p.stages_per_set; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], (uint32_t)lanes_per_set);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // Tile slot i of a set: row groups (set + i / segs * sets) * groups .. + groups, segment i % segs
    const int slots = (rows.total + p.groups - 1) / p.groups;

    if (warp == WARPS) {
        // ---- producer: the weights do not depend on the kernel in front. (A wait for a free stage and the start of a copy are
        // about 350 cycles; working out the rows of every tile anew made it 1500, twice what an SM's share of HBM allows.)
        if (lane != 0) return;
        int s = 0, turn = 0;
        uint32_t ph = 0;
        bool ok = true;
        const uint32_t bytes = (uint32_t)p.stage_stride;
        for (int slot0 = 0; slot0 < slots && ok; slot0 += p.sets)
            for (int x = 0, seg = 0; seg < p.segs && ok; seg++, turn++, x += p.seg_units * p.unit_bytes / 8) {   // x in 8-byte elements
                for (int set = 0; set < p.sets && slot0 + set < slots; set++) {
                    const int st = set * p.stages_per_set + s;
                    if (turn >= p.stages_per_set && !(ok = mbar_wait_limit(&empty[st], ph ^ 1u))) break;
                    mbar_expect_tx(&full[st], bytes);
                    // a box is 16 rows whatever is left of the range: rows past it are another CTA's, or zeros past the matrix
                    for (int gr = 0; gr < p.groups; gr++) {
                        int mat = 0, row0 = 0;
                        rows.at(p, min((slot0 + set) * p.groups + gr, rows.total - 1), mat, row0);
                        const CUtensorMap *m = mat == 0 ? &maps.m[0] : (mat == 1 ? &maps.m[1] : &maps.m[2]);
                        tma_2d(smem + st * p.stage_stride + gr * 16 * p.row_stride, m, x, row0, &full[st]);
                    }
                }
                if (++s == p.stages_per_set) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        if (!ok) {
            // the consumers stopped releasing stages: record it, then wait (bounded) for the copies still in flight
            report_error(p.err, 1);
            for (int st = 0; st < p.sets * p.stages_per_set; st++)
                if (mbar_wait_limit(&full[st], 0, 1u << 12)) mbar_wait_limit(&full[st], 1, 1u << 12);   // one of the two phases has passed
        }
        return;
    }

    // ---- consumers
    load_activations<TYPE>(p, act, red);   // (waits for the kernel in front)
    const int set = warp / lanes_per_set, in_set = warp % lanes_per_set, gr = in_set / p.seg_units, u = in_set % p.seg_units;
    const bool works = set < p.sets;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true, ready = false;
    const int g = lane >> 2, t = lane & 3;
    const uint8_t *b0 = g < p.nc ? act + g * p.act_stride + u * 256 + t * 8 : zeros + t * 8;
    const int b_seg = g < p.nc ? p.seg_units * 256 : 0;
    for (int e0 = 0; e0 < slots; e0 += p.epoch * p.sets) {
        const int e1 = min(slots, e0 + p.epoch * p.sets);
        if (works)
            for (int slot = e0 + set; slot < e1; slot += p.sets) {
                float f[4] = {0.f, 0.f, 0.f, 0.f};
                for (int seg = 0; seg < p.segs; seg++) {
                    const int st = set * p.stages_per_set + s;
                    if (ok && !ready && !mbar_wait_limit(&full[st], ph)) {
                        if (lane == 0) report_error(p.err, 1);
                        ok = false;   // this warp stops releasing stages; the producer's bounded wait ends the copies
                    }
                    if (++s == p.stages_per_set) {
                        s = 0;
                        ph ^= 1u;
                    }
                    // a probe takes 100 to 300 cycles to answer: the next stage's goes out before this one's weights are worked on
                    ready = mbar_test(su32(&full[set * p.stages_per_set + s]), ph);
                    const int unit = seg * p.seg_units + u;
                    if (unit < p.units) {
                        // rows past a matrix's end hold what the stage held before; their sums are not used
                        const uint8_t *w = smem + st * p.stage_stride + (gr * 16 + g) * p.row_stride + u * p.unit_bytes;
                        if (TYPE == TLB_TYPE_Q4_K) unit_q4_K<ONE>(p, w, w + 8 * p.row_stride, b0 + seg * b_seg, unit, act, f);
                        else unit_q_0<TYPE, ONE>(p, w, w + 8 * p.row_stride, b0 + seg * b_seg, unit, act, f);
                    }
                    __syncwarp();
                    if (lane == 0 && ok) mbar_arrive(&empty[st]);
                }
                // part [slot of the epoch][group][unit warp][column][row]
                float *o = part + ((size_t)((slot - e0) * p.groups + gr) * p.seg_units + u) * p.nc * 16;
                if (ONE) {
                    if (t == 0) {
                        o[g] = f[0];
                        o[g + 8] = f[2];
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (2 * t + (i & 1) < p.nc) o[(2 * t + (i & 1)) * 16 + g + (i >> 1) * 8] = f[i];
                }
            }
        consumers_sync();
        // ---- the rows of this stretch: their parts in order
        const int n_vals = (e1 - e0) * p.groups * p.nc * 16;
        for (int i = tid; i < n_vals; i += WARPS * 32) {
            const int r = i & 15, n = (i >> 4) % p.nc, gi = (i >> 4) / p.nc;   // row, column, group of the epoch
            int mat, row0;
            if (r >= rows.at(p, e0 * p.groups + gi, mat, row0) || (p.glu && mat == 1)) continue;
            const float *q = part + ((size_t)gi * p.seg_units * p.nc + n) * 16 + r;
            float v = 0.f;
            for (int x = 0; x < p.seg_units; x++) v += q[x * p.nc * 16];
            if (p.glu) {   // SiLU(gate) * up, as k_row_quant_q8k in its RQ_GLU mode
                q += p.seg_units * p.nc * 16;
                float up = 0.f;
                for (int x = 0; x < p.seg_units; x++) up += q[x * p.nc * 16];
                v = __fmul_rn(__fdiv_rn(v, __fadd_rn(1.0f, expf(-v))), up);
            }
            float *y = mat == 0 ? p.y[0] : (mat == 1 ? p.y[1] : p.y[2]);
            const int64_t ld = mat == 0 ? p.ldy[0] : (mat == 1 ? p.ldy[1] : p.ldy[2]);
            y[(p.n0 + n) * ld + row0 + r] = v;
        }
        if (e1 < slots) consumers_sync();
    }
}

}  // namespace gemv

// ---------------------------------------------------------------- host side
using gemv::k_gemv;

constexpr int GEMV_SMEM_ONE = 224 * 1024;        // one CTA per SM
constexpr int GEMV_SMEM_TWO = 112 * 1024 - 512;  // two

// fills the geometry of a launch of nc columns; false when a row of activations leaves no room for two tiles
static bool gemv_geometry(gemv::Params &p, uint32_t type, int64_t K, int nc, size_t &smem) {
    auto pad = [](int64_t n, int mod) {   // the next size that is `mod` bytes past a multiple of 128
        int64_t r = (n + 15) / 16 * 16;
        while (r % 128 != mod) r += 16;
        return (int)r;
    };
    p.K = (int)K;
    p.nc = nc;
    p.unit_bytes = (int)tlb_row_size(type, 256);
    p.units = (int)(K / 256);
    // a tile's row segment: eight units, or four where a unit is 272 bytes (16 rows x 8 of those leave no room for a ring)
    const int most = type == TLB_TYPE_Q8_0 ? 4 : 8;
    p.segs = (p.units + most - 1) / most;
    p.seg_units = (p.units + p.segs - 1) / p.segs;
    p.groups = p.segs == 1 ? std::max(1, gemv::WARPS / p.seg_units) : 1;
    while (p.groups > 1 && 16 * p.groups * p.seg_units * p.unit_bytes > 24 * 1024) p.groups--;
    p.sets = gemv::WARPS / (p.groups * p.seg_units);
    // rows g = 0..7 of a tile (and columns of activations) must fall on different banks: 8-byte reads of four lanes (Q4_K,
    // codes), or 4-byte reads (34- and 18-byte blocks)
    p.row_stride = pad((int64_t)p.seg_units * p.unit_bytes, type == TLB_TYPE_Q4_K ? 32 : 16);
    p.stage_stride = 16 * p.groups * p.row_stride;
    p.d_off = (int)((K + 15) / 16 * 16);
    p.bsum_off = p.d_off + (int)((type == TLB_TYPE_Q4_K ? K / 256 * 4 : K / 32 * 4) + 15) / 16 * 16;
    p.act_stride = pad(p.bsum_off + (type == TLB_TYPE_Q4_K ? K / 32 * 2 : 0), 32);
    const int group_part = p.sets * p.groups * p.seg_units * nc * 64;   // of one row group of every set and slot
    p.epoch = std::max(1, gemv::PART_BYTES / group_part);
    if (p.epoch * p.sets * p.groups % 2) p.epoch++;                     // gate and up of a row stay together
    const int fixed = nc * p.act_stride + p.epoch * group_part;
    const int budget = fixed + std::max(3, 2 * p.sets) * p.stage_stride <= GEMV_SMEM_TWO ? GEMV_SMEM_TWO : GEMV_SMEM_ONE;
    p.stages_per_set = std::min(gemv::MAX_STAGES / p.sets, (budget - fixed) / (p.sets * p.stage_stride));
    smem = (size_t)std::max(p.stages_per_set, 0) * p.sets * p.stage_stride + fixed;
    return p.stages_per_set >= 2;
}

bool gemv_supported(uint32_t type, int64_t K, int64_t M, int64_t N) {
    if (type == TLB_TYPE_Q6_K) return gemv_f32_supported(type, K, M, N);
    if (type != TLB_TYPE_Q4_K && type != TLB_TYPE_Q8_0 && type != TLB_TYPE_Q4_0) return false;
    if (K % 256 != 0 || K < 256 || K > (1 << 20) || M < 1 || M > (1 << 28) || N < 1 || !tc_available()) return false;
    gemv::Params p{};
    size_t smem;
    return gemv_geometry(p, type, K, 1, smem);
}

void gemv_configure() {
    auto set = [](auto *k) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMV_SMEM_ONE); };
    set(k_gemv<TLB_TYPE_Q4_K, true>);
    set(k_gemv<TLB_TYPE_Q4_K, false>);
    set(k_gemv<TLB_TYPE_Q8_0, true>);
    set(k_gemv<TLB_TYPE_Q8_0, false>);
    set(k_gemv<TLB_TYPE_Q4_0, true>);
    set(k_gemv<TLB_TYPE_Q4_0, false>);
    gemv_f32_configure();
}

cudaError_t launch_gemv(const GemvArgs &g, int sm_count, int *err, cudaStream_t st) {
    if (g.type == TLB_TYPE_Q6_K) return launch_gemv_f32(g, sm_count, err, st);
    gemv::Params p{};
    gemv::Maps maps;
    int64_t rows_total = 0;
    p.n_mats = g.n_mats;
    p.glu = g.glu;
    for (int j = 0; j < g.n_mats; j++) {
        p.M[j] = (int)g.M[j];
        rows_total += g.M[j];
        if (j == 0 || !g.glu) {
            p.y[j] = g.y[j];
            p.ldy[j] = g.ldy[j];
        }
    }
    p.act = g.act;
    p.ready = (const uint8_t *)g.ready;
    p.err = err;
    for (int64_t n0 = 0; n0 < g.N;) {
        size_t smem = 0;
        int nc = (int)std::min<int64_t>(gemv::MAX_COLS, g.N - n0);
        while (nc > 1 && !gemv_geometry(p, g.type, g.K, nc, smem)) nc--;
        if (!gemv_geometry(p, g.type, g.K, nc, smem)) return cudaErrorInvalidValue;
        p.n0 = (int)n0;
        // A CTA per SM leaves room for the next launch's CTA beside it, which then has its ring full when this one ends. Long streams
        // gain more from two CTAs of their own (measured [128256 x 4096]: Q4_K 66 -> 55 us, Q8_0 102 -> 88): from 48 tiles per SM on.
        const int64_t tiles = (rows_total + 15) / 16 * p.segs / p.groups / sm_count;
        const dim3 grid((unsigned)(tiles >= 48 && smem <= (size_t)GEMV_SMEM_TWO ? 2 * sm_count : sm_count)), block(gemv::THREADS);
        cudaError_t e = cudaSuccess;
        for (int j = 0; j < 3 && e == cudaSuccess; j++)
            e = tc_encode_2d_bytes(&maps.m[j], g.W[j < g.n_mats ? j : 0], tlb_row_size(g.type, g.K), (uint64_t)g.M[j < g.n_mats ? j : 0], (uint32_t)p.row_stride, 16);
        if (e != cudaSuccess) return e;
        switch (g.type) {
            case TLB_TYPE_Q4_K: e = nc == 1 ? launch_pdl_if(g.early, k_gemv<TLB_TYPE_Q4_K, true>, grid, block, smem, st, maps, p) : launch_pdl_if(g.early, k_gemv<TLB_TYPE_Q4_K, false>, grid, block, smem, st, maps, p); break;
            case TLB_TYPE_Q8_0: e = nc == 1 ? launch_pdl_if(g.early, k_gemv<TLB_TYPE_Q8_0, true>, grid, block, smem, st, maps, p) : launch_pdl_if(g.early, k_gemv<TLB_TYPE_Q8_0, false>, grid, block, smem, st, maps, p); break;
            case TLB_TYPE_Q4_0: e = nc == 1 ? launch_pdl_if(g.early, k_gemv<TLB_TYPE_Q4_0, true>, grid, block, smem, st, maps, p) : launch_pdl_if(g.early, k_gemv<TLB_TYPE_Q4_0, false>, grid, block, smem, st, maps, p); break;
            default: return cudaErrorInvalidValue;
        }
        if (e != cudaSuccess) return e;
        n0 += nc;
    }
    return cudaSuccess;
}

}  // namespace tlb
