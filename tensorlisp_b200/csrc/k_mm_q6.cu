// MUL_MAT with Q6_K weights and more than a few f32 activation columns on tcgen05 (reference: crates/kernels/src/cuda/native/mm.cu:16-42,
// decoded weights times f32 activations, summed in f32).
//
// A weight is d * sc * (q - 32) with an 8-bit scale sc per 16 weights and d per 256. sc is cut into two digits of four bits, 16 s1 + s0, both in
// [-8, 8]: (q - 32) * s1 and (q - 32) * s0 are whole numbers of at most 2^8. 256 activations of a column are six digits of nine bits at the scale of
// their largest (mm_terms.cuh), which hold every f32 down to 2^-29 of it to its last bit; a super-block with a smaller value, or one that is not finite, is
// summed value by value. (Three digits, 26 bits, lost a large activation's neighbours where its weight is zero: 7.4e-5 of a row's norm beside 1e4, 0.68 beside
// 1e8.) Products of a weight's and an activation's digit, and the sums of 256 of them, stay within 2^24: exact in the f32 accumulators of
// kind::f16, which otherwise truncate (terms of f16 values in their place: 3.3e-7 relative error against f64). So each super-block has two
// accumulators of six columns per activation; d and the scale come in as the sums leave tensor memory.
//
// Layout: one CTA per SM, a stretch of the (row tile of 128, super-block) sequence each (stream-K as in k_mm_plain.cu). Rows are 210 bytes per
// super-block, so their pieces lie on 2-byte boundaries; eight rows together are a multiple of 16 bytes, so eight tensor copies, one per row of
// the eight, bring a tile's super-block, 240 bytes from the boundary of 16 below it (by words or 16 bytes through registers of the SM's own
// copies, 256 or 64 instructions: 2.7 and 1.7 us per super-block). Eight warps unpack, two and a half instructions per weight, and store the two
// digits into tensor memory, 128 weights of 128 rows at a time in two buffers; eight split activations, four add up, one issues MMAs.
//
// Relative error against f64, k_gemv_f32.cu and here, 5 to 40 columns: 9.9e-8 / 4.3e-8 at [300 x 4096], 9.8e-8 / 5.1e-8 at [20000 x 4096], 1.1e-7 / 5.1e-8 at [20000 x
// 14336]; activations over five decades 8.3 to 10e-8 / 7.6 to 10e-8 at [20000 x 4096], 0.94 to 1.0e-7 / 7.1 to 8.7e-8 at [20000 x 14336].
//
// Measured, passes of four columns of k_gemv_f32.cu and here, a launch timed alone, cold: [32000 x 4096] x 8 136 -> 74 us, x 16 260 -> 140, x 64 1003 -> 530;
// [4096 x 14336] x 16 240 -> 81, x 64 929 -> 292; [1500 x 2048] x 5 20 -> 18 (three digits and passes of 21 columns: 67, 85, 302, 50, 164, 17). What bounds it:
// issue slots. A pass of one column takes 66 us at [32000 x 4096], copies alone 44, unpacking adds 13; splitting and adding grow with columns times
// digits, so that ten columns in one pass (113 us) gain little on two passes of five.
#include <algorithm>
#include <cstdlib>
#include <cuda_fp16.h>

#include "kernels.h"
#include "dequant.cuh"
#include "mm_terms.cuh"
#include "pdl.cuh"

namespace tlb {

cudaError_t tc_encode_2d_bytes(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows);

namespace q6tc {

using namespace plain;
constexpr int BLOCK = 210;
constexpr int KS = 256;                          // weights of a step (and chunk): a super-block
constexpr int BOXES = KS / KB;
constexpr int ROW_UNITS = 14;                    // 16-byte units that hold a super-block starting on any 2-byte boundary
constexpr int ROW_STRIDE = 240;                  // 15 units: a warp's reads of one word of 32 rows meet each bank four times, the least on 16-byte boundaries
constexpr int COPY_BYTES = ROWS / 8 * ROW_STRIDE;   // of one copy: every eighth row of a tile
constexpr int LEFT = 8 * COPY_BYTES;             // behind them the up to seven rows that are left at the end of the matrix
constexpr int RAW_STAGE = (LEFT + 7 * ROW_STRIDE + 127) / 128 * 128;
constexpr int MAX_STAGES = 6;
constexpr int MAX_COLS = 8;                      // columns per pass, and what the adding warps hold in registers
constexpr int CONV_WARP0 = 6, DEC_WARP0 = 14, DEC_WARPS = 8;
constexpr int THREADS = 32 * (DEC_WARP0 + DEC_WARPS);
// dynamic shared memory beside the static arrays
constexpr int SMEM_ROOM = 227 * 1024 - 3 * 1024;
constexpr uint32_t A_COL0 = 256, A_HALF = 128;   // tensor memory: accumulators in [0, 256), then per half of a super-block 64 columns of either digit

struct Params : PlainParams {
    const uint8_t *W;
    int64_t row_bytes;
};

__device__ __forceinline__ void cp16_some(uint32_t dst, const uint8_t *src, int bytes) {   // the rest is zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_arrive(uint64_t *bar) {   // when this thread's copies so far have landed
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(su32(bar)) : "memory");
}

// Four words of a row from word w0 on; sh: 16 where the super-block starts in the middle of a word
__device__ __forceinline__ void words(const uint32_t *row, int w0, uint32_t sh, uint32_t (&o)[4]) {
    uint32_t prev = row[w0];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t next = row[w0 + j + 1];
        o[j] = __funnelshift_r(prev, next, sh);
        prev = next;
    }
}

// 64 weights of a row, its 16 of either 32 of half h, as two digits (s0, then s1): columns 16k + 8 part .. of a half's buffer. sc: the
// half's eight scales, the part's from the lowest byte on
__device__ __forceinline__ void unpack(const uint32_t *row, uint32_t sh, int h, uint32_t sc_lo, uint32_t sc_hi, int part, uint32_t dst) {
    uint32_t qa[4], qb[4], qh[4];
    words(row, 16 * h + 4 * part, sh, qa);
    words(row, 16 * h + 8 + 4 * part, sh, qb);
    words(row, 32 + 8 * h + 4 * part, sh, qh);
    dst += (uint32_t)(8 * part);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int s = (int)(int8_t)((k < 2 ? sc_lo : sc_hi) >> (16 * (k & 1))), s0 = ((s + 8) & 15) - 8;
        // digit * (q - 32) from 1024 + q in one multiply-add: 1056 times a digit is exact in f16
        const __half2 off = __half2half2(__ushort_as_half((unsigned short)0xe420));   // -1056
        const __half2 hi = __half2half2(__int2half_rn((s - s0) >> 4)), lo = __half2half2(__int2half_rn(s0)), hi_off = __hmul2(hi, off), lo_off = __hmul2(lo, off);
        uint32_t vl[8], vh[8];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t low = k < 2 ? (k == 0 ? qa[j] : qb[j]) & 0x0f0f0f0fu : ((k == 2 ? qa[j] : qb[j]) >> 4) & 0x0f0f0f0fu;
            const uint32_t q = low | ((k == 0 ? qh[j] << 4 : (k == 1 ? qh[j] << 2 : (k == 2 ? qh[j] : qh[j] >> 2))) & 0x30303030u);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t b = __byte_perm(q, 0x64646464u, i ? 0x4342 : 0x4140);   // 1024 + q as f16
                const __half2 v = *reinterpret_cast<const __half2 *>(&b), l = __hfma2(v, lo, lo_off), g = __hfma2(v, hi, hi_off);
                vl[2 * j + i] = *reinterpret_cast<const uint32_t *>(&l);
                vh[2 * j + i] = *reinterpret_cast<const uint32_t *>(&g);
            }
        }
        tmem_st8(dst + (uint32_t)(16 * k), vl);
        tmem_st8(dst + (uint32_t)(64 + 16 * k), vh);
    }
}

__global__ void __launch_bounds__(THREADS, 1) k_mm_q6(const __grid_constant__ CUtensorMap wmap, Params p) {
    constexpr int NC = MAX_COLS;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
    __shared__ uint64_t bar_raw[MAX_STAGES], bar_rawfree[MAX_STAGES], bar_b[2], bar_bfree[2], bar_acc[2], bar_accfree[2], bar_a[2], bar_afree[2];
    __shared__ float inv[4][NC];      // per chunk in flight and column: what its sums are multiplied by (NaN: they are taken value by value)
    __shared__ float dsm[4][ROWS];    // and per row
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_fail;
    volatile int *fail = &s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b_tile = p.n_mma * KB * 2, b_chunk = BOXES * b_tile;
    uint8_t *raw = smem + 2 * b_chunk;
    if (tid == 0) {
        for (int i = 0; i < p.stages; i++) {
            mbar_init(&bar_raw[i], 1 + 32);
            mbar_init(&bar_rawfree[i], DEC_WARPS);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar_b[i], CONV_WARPS);
            mbar_init(&bar_bfree[i], 1);
            mbar_init(&bar_acc[i], 1);
            mbar_init(&bar_accfree[i], 4);
            mbar_init(&bar_a[i], DEC_WARPS);
            mbar_init(&bar_afree[i], 1);
        }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&tmem_base_s, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    griddep_launch();
    const int64_t total = (int64_t)p.tiles * p.steps;   // below 2^31 (mm_q6_supported)
    const int g0 = (int)plain_begin(blockIdx.x, total, gridDim.x), g1 = (int)plain_begin(blockIdx.x + 1, total, gridDim.x);
    const int tile_first = g0 / p.steps;

    // Lane L of tensor memory has row 8 (L % 16) + L / 16 of the tile: the order in which the copies leave them.
    const int whole = (int)min((int64_t)ROWS / 8, p.M / 8 - (int64_t)(p.tiles - 1) * (ROWS / 8)) * 8;   // rows of the last tile that are copied in eights

    if (warp == 0) {
        // ---- copies; the weights do not depend on the kernel in front
        const uint8_t *end = p.W + p.M * p.row_bytes;
        int tile = tile_first, step = g0 - tile * p.steps, s = 0;
        uint32_t ph = 0;
        for (int g = g0; g < g1; g++) {
            if (g - g0 >= p.stages) mbar_wait_nap(&bar_rawfree[s], ph ^ 1u, fail, 0);
            uint8_t *dst = raw + (size_t)s * RAW_STAGE;
            if (lane == 0) mbar_expect_tx(&bar_raw[s], 8 * COPY_BYTES);
            __syncwarp();
            if (lane < 8) tma_2d(dst + lane * COPY_BYTES, &wmap, ((lane * (int)p.row_bytes + step * BLOCK) & ~15) / 8, tile * (ROWS / 8), &bar_raw[s]);
            if (tile == p.tiles - 1) {
                const int rows = (int)(p.M - (int64_t)tile * ROWS);
                for (int r = whole + (lane >> 4); r < rows; r += 2) {
                    const uint8_t *a = p.W + ((int64_t)tile * ROWS + r) * p.row_bytes + (int64_t)step * BLOCK;
                    const uint8_t *src = (const uint8_t *)((uintptr_t)a & ~(uintptr_t)15) + (lane & 15) * 16;
                    // what the last one has beyond the matrix is zero-filled
                    if ((lane & 15) < ROW_UNITS) cp16_some(su32(dst + LEFT + (r - whole) * ROW_STRIDE + (lane & 15) * 16), src < end ? src : p.W, (int)max((int64_t)0, min((int64_t)16, (int64_t)(end - src))));
                }
            }
            cp_arrive(&bar_raw[s]);
            if (++step == p.steps) {
                step = 0;
                tile++;
            }
            if (++s == p.stages) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        walk<1>(p.steps, g0, g1, tile_first, [&](int c, int, int, bool, bool) {
            const int buf = c & 1;
            const uint32_t ph = (uint32_t)((c >> 1) & 1);
            if (c >= 2) mbar_wait_nap(&bar_accfree[buf], ph ^ 1u, fail, 0);
            mbar_wait_nap(&bar_b[buf], ph, fail, 0);
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                mbar_wait_nap(&bar_a[h], (uint32_t)(c & 1), fail, 0);
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (int t = 0; t < 2; t++)
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const uint64_t bd = desc_sw128(su32(smem + buf * b_chunk + (2 * h + b) * b_tile));
#pragma unroll
                            for (int k = 0; k < KB / 16; k++)
                                umma_f16_ta(tmem + (uint32_t)((2 * buf + t) * p.acc_stride), tmem + A_COL0 + (uint32_t)h * A_HALF + (uint32_t)(t * 64 + (b * 4 + k) * 8), bd + 2 * k, p.idesc,
                                            (h || b || k) ? 1u : 0u);
                        }
                    umma_commit(&bar_afree[h]);
                    if (h) {
                        umma_commit(&bar_bfree[buf]);
                        umma_commit(&bar_acc[buf]);
                    }
                }
                __syncwarp();
            }
        });
    } else if (warp < CONV_WARP0) {
        // ---- adding warps: warp % 4 fixes the 32 rows a warp may read
        griddep_wait();
        const int q = warp & 3, r = 8 * (lane & 15) + 2 * q + (lane >> 4);
        float sum[NC], rest[NC];   // what the additions of super-blocks round away is kept: without it 16 of them end up to 1.2e-7 from f64
        walk<1>(p.steps, g0, g1, tile_first, [&](int c, int g, int e, bool begins, bool ends) {
            const int buf = c & 1, tile = g / p.steps;
            const int64_t row = (int64_t)tile * ROWS + r;
            if (begins) {
#pragma unroll
                for (int n = 0; n < NC; n++) sum[n] = rest[n] = 0.f;
            }
            mbar_wait_nap(&bar_acc[buf], (uint32_t)((c >> 1) & 1), fail, 32);
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)(2 * buf * p.acc_stride) + ((uint32_t)(q * 32) << 16);
            const float d = dsm[c & 3][q * 32 + lane];
            const bool d_finite = fabsf(d) < __int_as_float(0x7f800000);
            float total[NC];
#pragma unroll
            for (int t = DIGITS - 1; t >= 0; t -= 3) {   // the smallest digit first, three in flight
                float lo[3][NC], hi[3][NC];
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    tmem_ld8(acc + (uint32_t)((t - u) * p.N), lo[u]);
                    tmem_ld8(acc + (uint32_t)(p.acc_stride + (t - u) * p.N), hi[u]);
                }
                tmem_ld_wait();
#pragma unroll
                for (int u = 0; u < 3; u++)
#pragma unroll
                    for (int n = 0; n < NC; n++) {
                        const float v = fmaf(16.f, hi[u][n], lo[u][n]);
                        total[n] = t - u == DIGITS - 1 ? v : fmaf(total[n], 1.f / 512.f, v);
                    }
            }
#pragma unroll
            for (int n = 0; n < NC; n++) {
                const float f = inv[c & 3][n];
                float v = __fmul_rn(total[n] * 262144.f * d, f);
                if (!d_finite || f != f) {
                    v = 0.f;
                    if (n < p.N && row < p.M) {
                        const int step = g - tile * p.steps;
                        for (int slot = 0; slot < 4; slot++)
                            v += q6_K_slot_sum(p.W + row * p.row_bytes + (int64_t)step * BLOCK, p.x + (int64_t)n * p.ldx + (int64_t)step * KS, slot);
                    }
                }
                const float s = __fadd_rn(sum[n], v), w = __fsub_rn(s, sum[n]);
                rest[n] += __fadd_rn(__fsub_rn(sum[n], __fsub_rn(s, w)), __fsub_rn(v, w));
                sum[n] = s;
            }
            __syncwarp();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_accfree[buf]);
            if (!ends) return;
            const int t0 = tile * p.steps, t1 = t0 + p.steps, seg = max(g0, t0);
            const bool whole = seg == t0 && e == t1;
            float *o = whole ? p.out + row : p.partial + ((size_t)blockIdx.x * 2 + (seg == g0 ? 0 : 1)) * p.N * ROWS + r;
            const size_t ldo = whole ? (size_t)p.ldy : ROWS;
            if (whole && row >= p.M) return;
#pragma unroll
            for (int n = 0; n < NC; n++)
                if (n < p.N) o[(size_t)n * ldo] = sum[n] + (fabsf(sum[n]) < __int_as_float(0x7f800000) ? rest[n] : 0.f);
        });
    } else if (warp < DEC_WARP0) {
        griddep_wait();
        split_columns<false, NC, KS, 1, true>(p, smem, b_tile, b_chunk, inv, bar_b, bar_bfree, warp - CONV_WARP0, lane, g0, g1, tile_first, fail);
    } else {
        // ---- unpacking warps: warp % 4 fixes the rows, two warps take 16 of every 32 weights each
        const int part = (warp - DEC_WARP0) >> 2, slot = (warp & 3) * 32 + lane, r = 8 * (slot & 15) + (slot >> 4);
        const uint32_t a_lane = tmem + A_COL0 + ((uint32_t)((warp & 3) * 32) << 16);
        int s = 0, tile = tile_first, step = g0 - tile * p.steps;
        uint32_t ph = 0;
        for (int c = 0; c < g1 - g0; c++) {
            const uint32_t off = (uint32_t)(((uint64_t)tile * ROWS + r) * p.row_bytes + (uint64_t)step * BLOCK) & 15u;   // p.W is on a multiple of 16
            const uint32_t sh = (off & 2u) * 8;
            mbar_wait_nap(&bar_raw[s], ph, fail, 0);
            const uint8_t *place = raw + (size_t)s * RAW_STAGE + (tile == p.tiles - 1 && r >= whole ? LEFT + min(r - whole, 6) * ROW_STRIDE : slot * ROW_STRIDE);
            const uint32_t *rrow = reinterpret_cast<const uint32_t *>(place + (off & 12u));
            uint32_t scales[4];
            words(rrow, 48, sh, scales);
            if (part == 0) dsm[c & 3][slot] = __half2float(__ushort_as_half((unsigned short)(rrow[52] >> sh)));
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                if (c >= 1) {
                    mbar_wait_nap(&bar_afree[h], (uint32_t)((c - 1) & 1), fail, 0);   // the MMAs that read this buffer are done
                    tc_fence_after();
                }
                unpack(rrow, sh, h, (h ? scales[2] : scales[0]) >> (8 * part), (h ? scales[3] : scales[1]) >> (8 * part), part, a_lane + (uint32_t)h * A_HALF);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_a[h]);
            }
            if (lane == 0) mbar_arrive(&bar_rawfree[s]);
            if (++step == p.steps) {
                step = 0;
                tile++;
            }
            if (++s == p.stages) {
                s = 0;
                ph ^= 1u;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
    if (tid == 0 && s_fail) report_error(p.err, 2);
}

}  // namespace q6tc

// ---------------------------------------------------------------- host side
void mm_q6_configure() { cudaFuncSetAttribute(q6tc::k_mm_q6, cudaFuncAttributeMaxDynamicSharedMemorySize, q6tc::SMEM_ROOM); }

// From three columns on, where k_gemv_q6.cu takes fewer. us of a launch, cold, here / k_gemv_f32.cu, three and four columns: [32000 x 4096] 70 / 100 and
// 72 / 74, [4096 x 4096] 27.1 / 25.5 and 25.2 / 22.4, [4096 x 14336] 44 / 64 and 42 / 67, [3000 x 2816] 23.5 / 22.4 and 21.2 / 21.4, [2000 x 8448] 29 / 32
// and 28 / 42; two columns lose everywhere (67 / 57, 27 / 18, 44 / 39).
//
// Small matrices, whose passes of four columns cost k_gemv_f32.cu less than half a pass of eight here. In a row of launches, us, there / here: [1500 x 2048] x 3
// 7.9 / 10.0, x 4 7.3 / 9.9, x 5 11.7 / 10.0, x 12 17.8 / 19.9, x 16 23.4 / 19.8; [1024 x 4096] x 4 7.2 / 12.8, x 8 12.7 / 13.9, x 12 18.7 / 25.4, x 16 24.3 /
// 25.5; [4096 x 4096] x 3 16.5 / 17.9, x 4 13.1 / 18.3, x 5 22.9 / 19.8, x 8 23.6 / 20.7, x 12 35.2 / 37.7, x 16 46.9 / 38.4; [30000 x 512] x 5 29 / 16; [32000 x 4096]
// x 3 93 / 62, x 4 66 / 64. Both are a constant and a part that grows with the weights (here also with the parts of a tile's sum); rows of more than
// 4096 weights have passes of two columns there.
static bool decode_faster(int64_t K, int64_t M, int64_t N) {
    if (K > 4096 || getenv("TLB_Q6_DIGITS")) return false;
    const double x = (double)(K * M) * 1e-6;
    const double pass1 = 4.0 + 0.33 * x, pass2 = 4.2 + 0.352 * x, pass4 = 5.2 + 0.461 * x;
    const int64_t rest = N % 4, passes = N / 4 + (rest + 1) / 2;
    const double there = (double)(N / 4) * pass4 + (rest & 1 ? pass1 : 0) + (rest & 2 ? pass2 : 0) - 1.5 * (double)(passes - 1) - (rest == 3 ? 1.5 : 0);
    return there < (double)((N + q6tc::MAX_COLS - 1) / q6tc::MAX_COLS) * (6.3 + 0.31 * (double)(K / q6tc::KS) + 0.41 * x);
}
bool mm_q6_supported(uint32_t type, int64_t K, int64_t M, int64_t N) {
    return type == TLB_TYPE_Q6_K && K % q6tc::KS == 0 && K >= q6tc::KS && M >= 8 && N > 2 && N > gemv_q6_columns(K, M) && !decode_faster(K, M, N) && N <= (1 << 20) && K <= (1 << 20) &&
           (M + tc::ROWS - 1) / tc::ROWS * (K / q6tc::KS) < (1ll << 31) && tc_available();
}

PlainPlan mm_q6_plan(int64_t K, int64_t M, int64_t N, int sm_count) {
    PlainPlan t{};
    t.passes = (int)((N + q6tc::MAX_COLS - 1) / q6tc::MAX_COLS);
    t.cols = (int)((N + t.passes - 1) / t.passes);
    t.passes = (int)((N + t.cols - 1) / t.cols);
    t.steps = (int)(K / q6tc::KS);
    t.tiles = (int)((M + tc::ROWS - 1) / tc::ROWS);
    t.ctas = (int)std::min<int64_t>(sm_count, (int64_t)t.steps * t.tiles);
    t.bytes = t.tiles % t.ctas ? (uint64_t)t.ctas * 2 * t.cols * tc::ROWS * 4 : 0;   // parts of cut tiles
    return t;
}

cudaError_t launch_mm_q6(const PlainPlan &t, const void *W, int64_t K, int64_t M, int64_t N, const float *x, int64_t ldx, float *y, int64_t ldy, void *scratch, int *err, cudaStream_t st,
                         bool early) {
    // eight rows in one (their length is a multiple of 16 bytes), in bytes
    CUtensorMap map;
    cudaError_t e = tc_encode_2d_bytes(&map, W, (uint64_t)(K / q6tc::KS) * q6tc::BLOCK * 8, (uint64_t)M / 8, q6tc::ROW_STRIDE, tc::ROWS / 8);
    for (int pass = 0; pass < t.passes && e == cudaSuccess; pass++) {
        const int64_t n0 = (int64_t)pass * t.cols;
        q6tc::Params p{};
        const int n = p.N = (int)std::min<int64_t>(t.cols, N - n0);
        p.n_mma = (plain::DIGITS * n + 15) / 16 * 16;
        p.acc_stride = 64;   // the adding warps read eight columns at a time: past the last digit's end what they read is not used
        p.x = x + n0 * ldx;
        p.out = y + n0 * ldy;
        p.partial = (float *)scratch;
        p.K = K;
        p.M = M;
        p.ldx = ldx;
        p.ldy = ldy;
        p.steps = t.steps;
        p.tiles = t.tiles;
        p.idesc = (1u << 4) | ((uint32_t)(p.n_mma >> 3) << 17) | ((uint32_t)(tc::ROWS >> 4) << 24);
        p.err = err;
        p.W = (const uint8_t *)W;
        p.row_bytes = K / q6tc::KS * q6tc::BLOCK;
        const int b_bytes = 2 * q6tc::BOXES * p.n_mma * plain::KB * 2;
        p.stages = std::min(q6tc::MAX_STAGES, (q6tc::SMEM_ROOM - 1024 - b_bytes) / q6tc::RAW_STAGE);
        const size_t smem = (size_t)b_bytes + (size_t)p.stages * q6tc::RAW_STAGE + 1024;
        e = launch_pdl_if(early, q6tc::k_mm_q6, dim3((unsigned)t.ctas), dim3(q6tc::THREADS), smem, st, map, p);
        if (e == cudaSuccess) e = launch_mm_plain_fixup(t, n, p.partial, p.out, M, ldy, st);
    }
    return e;
}

}  // namespace tlb
