// MUL_MAT with f16 / bf16 weight matrices on tcgen05 (reference: crates/kernels/src/cuda/native/mm.cu:16-42, whose
// arithmetic is weight times f32 activation, summed in f32).
//
// The weights go to the tensor cores as they are. An f32 activation is split into three terms of the weights' type whose
// sum it is: bf16 terms cover its 24 bits exactly, f16 terms do so after the values of a chunk (128 or 256 of a column) have
// been scaled by a power of two that brings the largest magnitude to [2^14, 2^15): 33 bits below that, down to the f16
// subnormals. The terms are further columns of the same product, so one pass over the weights serves them all. The tensor core
// truncates when it adds to an f32 accumulator (2.9e-6 relative error over 4096 terms); so an accumulator holds one chunk only,
// and the chunks are added up in registers (2.1e-7, as with f32 multiply-adds throughout).
//
// What bounds it: reading the weights once (HBM) up to about 64 columns. A step of 128 weights of 128 rows is 32 KB, for
// which an SM's share of the measured copy bandwidth is about 1400 cycles; its eight MMAs take 360 cycles at up to 64
// columns (21 activations) and 770 at 192. One CTA per SM, 14 warps that meet through mbarriers: one issues the TMA copies of
// the weights, eight split the activations of the next chunk into swizzled B tiles (in the kernel, because a launch of
// their own costs more than all of it up to 16 columns), one issues the MMAs, four add up. The (tile, step) sequence is cut
// into equal stretches over the CTAs whatever the tile count (stream-K), because the 112 tiles of a layer matrix would leave a
// quarter of the SMs idle; a tile cut by a boundary leaves its parts in scratch and k_mm_plain_fixup adds them in order.
// [14336 x 4096] f16 x 8 columns (117 MB): 313 us with a warp per output element, 27 us here (4.4 TB/s); 16 columns 31, 33 columns 51.
#include <algorithm>
#include <cuda_bf16.h>

#include "kernels.h"
#include "pdl.cuh"
#include "tc_common.cuh"
#include "mm_terms.cuh"

namespace tlb {

cudaError_t tc_encode_2d_sw128(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t cols, uint64_t rows, uint32_t box_cols, uint32_t box_rows, bool bf16);

namespace plain {

using namespace tc;
constexpr int KS = 2 * KB;              // and per step. A thread that waits for a barrier and starts a copy needs about 420
                                        // cycles for the pair, so a step of one 16 KB box would leave no slack (34 -> 29 us)
constexpr int A_BOX = ROWS * KB * 2, A_STAGE = 2 * A_BOX;
constexpr int MAX_COLS = 80;            // activation columns per pass: three terms each, 240 MMA columns
constexpr int CONV_WARP0 = 6;
constexpr int THREADS = 32 * (CONV_WARP0 + CONV_WARPS);   // TMA, MMA, four adding and eight splitting warps
constexpr int SMEM = 208 * 1024;
constexpr int MAX_STAGES = 6;

// steps per chunk: what an accumulator sums up, what a split chunk of activations covers. Two chunks of B tiles must leave
// room for the weights in flight.
__host__ __device__ constexpr int chunk_steps(int nc) { return nc <= 24 ? 2 : 1; }

}  // namespace plain

// NC: columns the adding warps hold in registers, a multiple of 8 and at least N
template <bool BF16, int NC>
__global__ void __launch_bounds__(plain::THREADS, 1) k_mm_plain(const __grid_constant__ CUtensorMap wmap, PlainParams p) {
    using namespace plain;
    constexpr int CS = chunk_steps(NC);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
    __shared__ uint64_t bar_full[MAX_STAGES], bar_free[MAX_STAGES], bar_b[2], bar_bfree[2], bar_acc[2], bar_accfree[2];
    __shared__ float inv[4][NC];   // per chunk in flight and column: what its sums are multiplied by
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_fail;
    volatile int *fail = &s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b_tile = p.n_mma * KB * 2, b_chunk = 2 * CS * b_tile;   // a B tile per box of 64
    uint8_t *a_ring = smem + 2 * b_chunk;
    if (tid == 0) {
        for (int i = 0; i < p.stages; i++) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_free[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar_b[i], CONV_WARPS);
            mbar_init(&bar_bfree[i], 1);
            mbar_init(&bar_acc[i], 1);
            mbar_init(&bar_accfree[i], 4);
        }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&tmem_base_s, (uint32_t)p.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    griddep_launch();
    const int64_t total = (int64_t)p.tiles * p.steps;   // below 2^31 (mm_plain_supported)
    const int g0 = (int)plain_begin(blockIdx.x, total, gridDim.x), g1 = (int)plain_begin(blockIdx.x + 1, total, gridDim.x);
    const int tile_first = g0 / p.steps;
    auto walk = [&](auto &&body) { plain::walk<CS>(p.steps, g0, g1, tile_first, body); };

    if (warp == 0) {
        if (lane == 0) {   // the weights do not depend on the kernel in front
            int tile = tile_first, step = g0 - tile * p.steps, s = 0;
            uint32_t ph = 0;
            for (int g = g0; g < g1; g++) {
                if (g - g0 >= p.stages) mbar_wait_nap(&bar_free[s], ph ^ 1u, fail, 0);
                mbar_expect_tx(&bar_full[s], A_STAGE);
#pragma unroll
                for (int b = 0; b < 2; b++)   // a box wholly past the row's end reads as zeros
                    tma_2d(a_ring + (size_t)s * A_STAGE + b * A_BOX, &wmap, step * KS + b * KB, tile * ROWS, &bar_full[s]);
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
    } else if (warp == 1) {
        const bool leader = elect_one();
        int s = 0;
        uint32_t sph = 0;
        walk([&](int c, int g, int e, bool, bool) {
            const int buf = c & 1;
            const uint32_t ph = (uint32_t)((c >> 1) & 1);
            if (c >= 2) mbar_wait_nap(&bar_accfree[buf], ph ^ 1u, fail, 0);
            mbar_wait_nap(&bar_b[buf], ph, fail, 0);
            tc_fence_after();
            for (int h = g; h < e; h++) {
                mbar_wait_nap(&bar_full[s], sph, fail, 0);
                tc_fence_after();
                if (leader) {
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        const uint64_t ad = desc_sw128(su32(a_ring + (size_t)s * A_STAGE + b * A_BOX)), bd = desc_sw128(su32(smem + buf * b_chunk + ((h - g) * 2 + b) * b_tile));
#pragma unroll
                        for (int k = 0; k < KB / 16; k++)
                            umma_f16(tmem + (uint32_t)(buf * p.acc_stride), ad + 2 * k, bd + 2 * k, p.idesc, (h > g || b || k) ? 1u : 0u);
                    }
                    umma_commit(&bar_free[s]);
                    if (h == e - 1) {
                        umma_commit(&bar_bfree[buf]);
                        umma_commit(&bar_acc[buf]);
                    }
                }
                __syncwarp();
                if (++s == p.stages) {
                    s = 0;
                    sph ^= 1u;
                }
            }
        });
    } else if (warp < CONV_WARP0) {
        // ---- adding warps: warp % 4 fixes the 32 rows a warp may read
        griddep_wait();
        const int q = warp & 3, r = q * 32 + lane;
        float sum[NC];
        walk([&](int c, int g, int e, bool begins, bool ends) {
            const int buf = c & 1;
            if (begins) {
#pragma unroll
                for (int n = 0; n < NC; n++) sum[n] = 0.f;
            }
            mbar_wait_nap(&bar_acc[buf], (uint32_t)((c >> 1) & 1), fail, 32);
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)(buf * p.acc_stride) + ((uint32_t)(q * 32) << 16);
#pragma unroll
            for (int n0 = 0; n0 < NC; n0 += 8) {
                if (n0 >= p.N) break;
                float t0[8], t1[8], t2[8];
                tmem_ld8(acc + (uint32_t)n0, t0);
                tmem_ld8(acc + (uint32_t)(p.N + n0), t1);
                tmem_ld8(acc + (uint32_t)(2 * p.N + n0), t2);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 8; j++) sum[n0 + j] += (t0[j] + (t1[j] + t2[j])) * (BF16 ? 1.f : inv[c & 3][n0 + j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_accfree[buf]);
            if (!ends) return;
            const int tile = g / p.steps, t0 = tile * p.steps, t1 = t0 + p.steps, seg = max(g0, t0);
            const bool whole = seg == t0 && e == t1;
            const int64_t row = (int64_t)tile * ROWS + r;
            float *o = whole ? p.out + row : p.partial + ((size_t)blockIdx.x * 2 + (seg == g0 ? 0 : 1)) * p.N * ROWS + r;
            const size_t ldo = whole ? (size_t)p.ldy : ROWS;
            if (whole && row >= p.M) return;
#pragma unroll
            for (int n = 0; n < NC; n++)
                if (n < p.N) o[(size_t)n * ldo] = sum[n];
        });
    } else {
        griddep_wait();
        split_columns<BF16, NC, KS, CS, false>(p, smem, b_tile, b_chunk, inv, bar_b, bar_bfree, warp - CONV_WARP0, lane, g0, g1, tile_first, fail);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, (uint32_t)p.tmem_cols);
    if (tid == 0 && s_fail) report_error(p.err, 2);
}

// a tile cut by CTA boundaries: its parts, in step order
__global__ void __launch_bounds__(256) k_mm_plain_fixup(const float *__restrict__ partial, float *__restrict__ out, int64_t M, int64_t ldy, int N, int steps, int tiles, int ctas) {
    griddep_launch();
    griddep_wait();
    const int64_t total = (int64_t)tiles * steps, t0 = (int64_t)blockIdx.x * steps, t1 = t0 + steps;
    // the CTA that has step g: begin(c) <= g < begin(c + 1)
    auto owner = [&](int64_t g) {
        int64_t c = g * ctas / total;
        while (plain_begin(c + 1, total, ctas) <= g) c++;
        while (plain_begin(c, total, ctas) > g) c--;
        return (int)c;
    };
    const int c0 = owner(t0), c1 = owner(t1 - 1);
    if (c0 == c1) return;
    const int i = blockIdx.y * 256 + threadIdx.x, n = i / tc::ROWS, r = i % tc::ROWS;
    const int64_t row = (int64_t)blockIdx.x * tc::ROWS + r;
    if (n >= N || row >= M) return;
    // A tile of a matrix of few rows has up to a part per step: what an addition rounds off is carried along (56 parts: 1.4e-7 from f64
    // without). Not in a sum that is no longer finite.
    float s = 0.f, rest = 0.f;
    for (int c = c0; c <= c1; c++) {
        const bool first = plain_begin(c, total, ctas) >= t0;   // this tile is where the CTA's stretch begins
        const float v = partial[((size_t)c * 2 + (first ? 0 : 1)) * N * tc::ROWS + (size_t)n * tc::ROWS + r];
        const float sum = __fadd_rn(s, v), got = __fsub_rn(sum, s);
        rest = __fadd_rn(rest, __fadd_rn(__fsub_rn(s, __fsub_rn(sum, got)), __fsub_rn(v, got)));
        s = sum;
    }
    out[(size_t)n * ldy + row] = fabsf(s) < __int_as_float(0x7f800000) ? s + rest : s;
}

// ---------------------------------------------------------------- host side
template <bool BF16, int NC>
static void plain_attr() { cudaFuncSetAttribute(k_mm_plain<BF16, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, plain::SMEM + 1024); }
template <bool BF16>
static void plain_attrs() { plain_attr<BF16, 8>(); plain_attr<BF16, 16>(); plain_attr<BF16, 24>(); plain_attr<BF16, 48>(); plain_attr<BF16, 80>(); }
void mm_plain_configure() {
    plain_attrs<false>();
    plain_attrs<true>();
}

// Rows of 16-byte multiples on both sides; anything else (odd row lengths, batches) stays with the generic kernel.
bool mm_plain_supported(uint32_t type, int64_t K, int64_t M, int64_t N, uint64_t w_row_bytes) {
    return (type == TLB_TYPE_F16 || type == TLB_TYPE_BF16) && K >= plain::KB && K % 8 == 0 && w_row_bytes % 16 == 0 && M >= 1 && N >= 1 && N <= (1 << 20) &&
           (M + tc::ROWS - 1) / tc::ROWS * ((K + plain::KS - 1) / plain::KS) < (1ll << 31) && tc_available();
}

PlainPlan mm_plain_plan(int64_t K, int64_t M, int64_t N, int sm_count) {
    PlainPlan t{};
    t.passes = (int)((N + plain::MAX_COLS - 1) / plain::MAX_COLS);
    t.cols = (int)((N + t.passes - 1) / t.passes);
    t.passes = (int)((N + t.cols - 1) / t.cols);
    t.steps = (int)((K + plain::KS - 1) / plain::KS);
    t.tiles = (int)((M + tc::ROWS - 1) / tc::ROWS);
    // at least two steps per CTA: below that the start of a CTA costs more than its share of the stream
    t.ctas = (int)std::max<int64_t>(1, std::min<int64_t>(sm_count, (int64_t)t.steps * t.tiles / 2));
    t.bytes = t.tiles % t.ctas ? (uint64_t)t.ctas * 2 * t.cols * tc::ROWS * 4 : 0;   // parts of cut tiles
    return t;
}

cudaError_t launch_mm_plain_fixup(const PlainPlan &t, int n, const float *partial, float *y, int64_t M, int64_t ldy, cudaStream_t st) {
    if (t.tiles % t.ctas == 0) return cudaSuccess;
    return launch_pdl(k_mm_plain_fixup, dim3((unsigned)t.tiles, (unsigned)((n * tc::ROWS + 255) / 256)), dim3(256), 0, st, partial, y, M, ldy, n, t.steps, t.tiles, t.ctas);
}

template <bool BF16>
static cudaError_t launch_plain_pass(const PlainPlan &t, const CUtensorMap &map, PlainParams p, cudaStream_t st, bool early) {
    const int nc = p.N <= 8 ? 8 : (p.N <= 16 ? 16 : (p.N <= 24 ? 24 : (p.N <= 48 ? 48 : 80)));
    const int b_bytes = 2 * plain::chunk_steps(nc) * p.n_mma * plain::KS * 2;
    p.stages = std::min(plain::MAX_STAGES, (plain::SMEM - b_bytes) / plain::A_STAGE);
    const size_t smem = (size_t)b_bytes + (size_t)p.stages * plain::A_STAGE + 1024;
    const dim3 grid((unsigned)t.ctas), block(plain::THREADS);
    switch (nc) {
        case 8: return launch_pdl_if(early, k_mm_plain<BF16, 8>, grid, block, smem, st, map, p);
        case 16: return launch_pdl_if(early, k_mm_plain<BF16, 16>, grid, block, smem, st, map, p);
        case 24: return launch_pdl_if(early, k_mm_plain<BF16, 24>, grid, block, smem, st, map, p);
        case 48: return launch_pdl_if(early, k_mm_plain<BF16, 48>, grid, block, smem, st, map, p);
        default: return launch_pdl_if(early, k_mm_plain<BF16, 80>, grid, block, smem, st, map, p);
    }
}

cudaError_t launch_mm_plain(const PlainPlan &t, bool bf16, const void *W, uint64_t w_row_bytes, int64_t K, int64_t M, int64_t N, const float *x, int64_t ldx, float *y, int64_t ldy,
                            void *scratch, int *err, cudaStream_t st, bool early) {
    CUtensorMap map;
    cudaError_t e = tc_encode_2d_sw128(&map, W, w_row_bytes, (uint64_t)K, (uint64_t)M, plain::KB, tc::ROWS, bf16);
    for (int pass = 0; pass < t.passes && e == cudaSuccess; pass++) {
        const int64_t n0 = (int64_t)pass * t.cols;
        PlainParams p{};
        const int n = p.N = (int)std::min<int64_t>(t.cols, N - n0);
        p.n_mma = (3 * n + 15) / 16 * 16;
        p.acc_stride = 16;   // the adding warps read eight columns at a time, past the last term's end
        while (p.acc_stride < p.n_mma || p.acc_stride < 2 * n + (n + 7) / 8 * 8) p.acc_stride *= 2;
        p.tmem_cols = 2 * p.acc_stride;
        p.x = x + n0 * ldx;
        p.out = y + n0 * ldy;
        p.partial = (float *)scratch;
        p.K = K;
        p.M = M;
        p.ldx = ldx;
        p.ldy = ldy;
        p.steps = t.steps;
        p.tiles = t.tiles;
        p.idesc = (1u << 4) | (bf16 ? (1u << 7) | (1u << 10) : 0u) | ((uint32_t)(p.n_mma >> 3) << 17) | ((uint32_t)(tc::ROWS >> 4) << 24);
        p.err = err;
        e = bf16 ? launch_plain_pass<true>(t, map, p, st, early) : launch_plain_pass<false>(t, map, p, st, early);
        if (e == cudaSuccess) e = launch_mm_plain_fixup(t, n, p.partial, p.out, M, ldy, st);
    }
    return e;
}

}  // namespace tlb
