// MUL_MAT with Q6_K weights and more than a few f32 activation columns on tcgen05 (reference: crates/kernels/src/cuda/native/mm.cu:16-42,
// decoded weights times f32 activations, summed in f32).
//
// A weight is d * sc * (q - 32) with an 8-bit scale sc per 16 weights and d per 256. sc is cut into two digits of four bits, 16 s1 + s0, both in
// [-8, 8]: (q - 32) * s1 and (q - 32) * s0 are whole numbers of at most 2^8. 256 activations of a column are 26-bit whole numbers at the scale of
// their largest, three digits of nine bits (mm_terms.cuh). Products of a weight's and an activation's digit, and the sums of 256 of them, stay within
// 2^24: exact in the f32 accumulators of kind::f16, which otherwise truncate (terms of f16 values in their place: 3.3e-7 relative error against
// f64). So each super-block has two accumulators of three columns per activation; d and the scale come in as the sums leave tensor memory.
//
// Layout: one CTA per SM, a stretch of the (row tile of 128, super-block) sequence each (stream-K as in k_mm_plain.cu). Rows are 210 bytes per
// super-block, so their pieces lie on 2-byte boundaries; eight rows together are a multiple of 16 bytes, so eight tensor copies, one per row of
// the eight, bring a tile's super-block, 240 bytes from the boundary of 16 below it (by words or 16 bytes through registers of the SM's own
// copies, 256 or 64 instructions: 2.7 and 1.7 us per super-block). Eight warps unpack, two and a half instructions per weight, and store the two
// digits into tensor memory, 128 weights of 128 rows at a time in two buffers; eight split activations, four add up, one issues MMAs.
//
// Relative error against f64, N(0, 1) activations, decoded weights in f32 (as before) and here: 1.0e-7 / 4.5e-8 at [300 x 4096], 9.9e-8 / 7.3e-8 at
// [20000 x 4096], 1.1e-7 / 8.6e-8 at [20000 x 14336]; activations over five decades 1.0e-7 / 1.2e-7.
//
// Measured, passes of four columns (k_gemv_q6.cu) and here, a launch timed alone, cold: [32000 x 4096] x 8 93 -> 66 us, x 16 174 -> 83, x 64 664 ->
// 301; [4096 x 14336] x 16 206 -> 50, x 64 792 -> 164; [1500 x 2048] x 5 20 -> 17. Up to four columns it loses: 51 us there at [32000 x 4096] x 4, 62
// here. What bounds it: issue slots (59% busy at 16 columns, a sixth of the stalls instruction fetch); copies alone take 44 us of the 83, unpacking
// adds 13, splitting and adding 11, the MMAs 7.
#include <algorithm>
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
constexpr int MAX_COLS = 21;                     // columns per pass: four accumulators of 64 columns (two super-blocks)
constexpr int CONV_WARP0 = 6, DEC_WARP0 = 14, DEC_WARPS = 8;
constexpr int THREADS = 32 * (DEC_WARP0 + DEC_WARPS);
constexpr int RUN = 8;
// dynamic shared memory beside the static arrays of k_mm_q6<nc>
constexpr int smem_room(int nc) { return 227 * 1024 - 3 * 1024 - nc * ROWS * 4; }
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

// NC: columns the adding warps hold in registers, a multiple of 8 and at least N
template <int NC>
__global__ void __launch_bounds__(THREADS, 1) k_mm_q6(const __grid_constant__ CUtensorMap wmap, Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
    __shared__ uint64_t bar_raw[MAX_STAGES], bar_rawfree[MAX_STAGES], bar_b[2], bar_bfree[2], bar_acc[2], bar_accfree[2], bar_a[2], bar_afree[2];
    __shared__ float inv[4][NC];      // per chunk in flight and column: what its sums are multiplied by (NaN: they are taken value by value)
    __shared__ float dsm[4][ROWS];    // and per row
    __shared__ float outer[NC][ROWS]; // sums of RUN super-blocks each: 56 added up one by one end 1.2e-7 from f64
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
        float sum[NC];
        int run = 0;
        bool flushed = false;
        walk<1>(p.steps, g0, g1, tile_first, [&](int c, int g, int e, bool begins, bool ends) {
            const int buf = c & 1, tile = g / p.steps;
            const int64_t row = (int64_t)tile * ROWS + r;
            if (begins) {
#pragma unroll
                for (int n = 0; n < NC; n++) sum[n] = 0.f;
                run = 0;
                flushed = false;
            }
            mbar_wait_nap(&bar_acc[buf], (uint32_t)((c >> 1) & 1), fail, 32);
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)(2 * buf * p.acc_stride) + ((uint32_t)(q * 32) << 16);
            const float d = dsm[c & 3][q * 32 + lane];
            const bool d_finite = fabsf(d) < __int_as_float(0x7f800000);
#pragma unroll
            for (int n0 = 0; n0 < NC; n0 += 8) {
                if (n0 >= p.N) break;
                float total[8];
#pragma unroll
                for (int t = 2; t >= 0; t--) {   // the smallest digit first
                    float lo[8], hi[8];
                    tmem_ld8(acc + (uint32_t)(t * p.N + n0), lo);
                    tmem_ld8(acc + (uint32_t)(p.acc_stride + t * p.N + n0), hi);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float v = fmaf(16.f, hi[j], lo[j]);
                        total[j] = t == 2 ? v : fmaf(v, t == 1 ? 512.f : 262144.f, total[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float f = inv[c & 3][n0 + j];
                    float v = total[j] * d * f;
                    if (!d_finite || f != f) {
                        v = 0.f;
                        if (n0 + j < p.N && row < p.M) {
                            const int step = g - tile * p.steps;
                            for (int slot = 0; slot < 4; slot++) v += q6_K_slot_sum(p.W + row * p.row_bytes + (int64_t)step * BLOCK, p.x + (int64_t)(n0 + j) * p.ldx + (int64_t)step * KS, slot);
                        }
                    }
                    sum[n0 + j] += v;
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_accfree[buf]);
            if (++run == RUN || (ends && flushed)) {
                run = 0;
#pragma unroll
                for (int n = 0; n < NC; n++) {
                    if (n >= p.N) break;
                    float &o = outer[n][q * 32 + lane];   // this thread's own
                    const float v = flushed ? o + sum[n] : sum[n];
                    o = v;
                    sum[n] = ends ? v : 0.f;
                }
                flushed = true;
            }
            if (!ends) return;
            const int t0 = tile * p.steps, t1 = t0 + p.steps, seg = max(g0, t0);
            const bool whole = seg == t0 && e == t1;
            float *o = whole ? p.out + row : p.partial + ((size_t)blockIdx.x * 2 + (seg == g0 ? 0 : 1)) * p.N * ROWS + r;
            const size_t ldo = whole ? (size_t)p.ldy : ROWS;
            if (whole && row >= p.M) return;
#pragma unroll
            for (int n = 0; n < NC; n++)
                if (n < p.N) o[(size_t)n * ldo] = sum[n];
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
void mm_q6_configure() {
    auto set = [](auto *k, int nc) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, q6tc::smem_room(nc)); };
    set(q6tc::k_mm_q6<8>, 8);
    set(q6tc::k_mm_q6<16>, 16);
    set(q6tc::k_mm_q6<24>, 24);
}

bool mm_q6_supported(uint32_t type, int64_t K, int64_t M, int64_t N) {
    return type == TLB_TYPE_Q6_K && K % q6tc::KS == 0 && K >= q6tc::KS && M >= 8 && N > MM_Q6_FEW && N <= (1 << 20) && K <= (1 << 20) && (M + tc::ROWS - 1) / tc::ROWS * (K / q6tc::KS) < (1ll << 31) &&
           tc_available();
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
        p.n_mma = (3 * n + 15) / 16 * 16;
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
        const int nc = (n + 7) / 8 * 8;
        p.stages = std::min(q6tc::MAX_STAGES, (q6tc::smem_room(nc) - 1024 - b_bytes) / q6tc::RAW_STAGE);
        const size_t smem = (size_t)b_bytes + (size_t)p.stages * q6tc::RAW_STAGE + 1024;
        auto go = [&](auto *k) { return launch_pdl_if(early, k, dim3((unsigned)t.ctas), dim3(q6tc::THREADS), smem, st, map, p); };
        e = nc == 8 ? go(q6tc::k_mm_q6<8>) : (nc == 16 ? go(q6tc::k_mm_q6<16>) : go(q6tc::k_mm_q6<24>));
        if (e == cudaSuccess) e = launch_mm_plain_fixup(t, n, p.partial, p.out, M, ldy, st);
    }
    return e;
}

}  // namespace tlb
