// Batched MUL_MAT (more than eight activation columns) with Q8_0 or Q4_0 weights on the 5th-generation tensor cores:
// the output projection of a decode step (vocab x d_model, Q8_0) is the largest matrix of the model.
//
// Arithmetic (same integers as the reference's ggml-cpu path, vendor/ggml/src/ggml-cpu/quants.c:451-479):
// per 32-element block b, output row r and activation column c
//     D_b = sum_k q[r,k] * q8[k,c]            (int8 x int8 -> int32, exact)
//     y  += (float)D_b * (d_w[r,b] * d_a[c,b])
// tcgen05.mma kind::i8 computes D_b for 128 rows x N columns in one instruction (K = 32 = one block),
// each block into its own TMEM accumulator; the epilogue warps apply the two f32 scales.
//
// Data movement: TMA brings a 128-row x 272-byte box (8 blocks of 34 bytes per row) of raw weights and
// one packed activation blob per 256 elements of K into shared memory. The weight codes need no
// arithmetic at all: sixteen warps strip the 2-byte scales, realign the codes and store them into
// tensor memory (tcgen05.st), where the MMA reads its A operand; B (the int8 activations, K-major core
// matrices) stays in shared memory. Eight warps drain the accumulators, one warp issues the MMAs,
// one the TMA copies; they meet only through mbarriers, every wait is bounded.
//
// Q4_0 has the same blocks in 18 bytes (a box is 144 bytes wide, 9 x 16: its 128-bit reads are conflict-free too) and the same
// activations; the realigning warps turn a nibble into the code less 8 on the way, three instructions for four weights. In passes of
// eight columns of the few-column kernel every eight cost another stream of the weights: [4096 x 4096] x 16 columns 27.6 -> 15.4 us,
// [32000 x 4096] x 64 254 -> 97 (a launch timed alone, cold, about 8 us of which are not the kernel's).
#include <algorithm>
#include <cstdlib>
#include <cuda.h>
#include <cuda_fp16.h>

#include "kernels.h"
#include "tc_common.cuh"
#include "pdl.cuh"

namespace tlb {

namespace tc8 {
constexpr int ROWS = 128;
constexpr int THREADS = 832;   // TMA warp + 8 epilogue warps + 16 realigning warps + MMA warp
constexpr int EPI_WARP0 = 1, DEQ_WARP0 = 9, MMA_WARP = 25;
constexpr int STAGE_BLOCKS = 8;                       // Q8_0 blocks of a row per pipeline stage (256 elements of K)
constexpr int ROW_CHUNK = STAGE_BLOCKS * 34;          // 272 bytes: 17 x 16, so 128-bit reads at row stride are conflict-free
constexpr int RAW_BYTES = ROWS * ROW_CHUNK;
__host__ __device__ constexpr int row_chunk(bool q4) { return STAGE_BLOCKS * (q4 ? 18 : 34); }   // bytes of a row per stage
__host__ __device__ constexpr int raw_bytes(bool q4) { return ROWS * row_chunk(q4); }
constexpr uint32_t TMEM_COLS = 512;                   // accumulators in [0, 256), the A ring in [256, 512)
constexpr uint32_t A_COL0 = 256;
constexpr int A_RING = 4;                             // stages of A (8 blocks x 8 columns of 4 int8) and of weight scales
}  // namespace tc8

// Bytes of one packed activation blob (256 elements of K, NPAD columns):
//   B    int8 [NPAD x 256]  K-major core matrices (8 columns x 16 bytes), lbo 128, sbo 2048     NPAD*256
//   d_a  f32  [8][NPAD]     activation scale per block and column                              NPAD*32
static inline __host__ __device__ int tc8_blob_bytes(int npad) { return npad * 288; }

__global__ void __launch_bounds__(256) k_act_pack_q80(const int8_t *qs, const float *ds, int64_t K, int N,
                                                       int npad, uint8_t *__restrict__ out) {
    griddep_launch();
    griddep_wait();
    // grid (stage, chunk of npad columns); blobs are laid out [chunk][stage]
    const int st = blockIdx.x;
    uint8_t *o = out + ((size_t)blockIdx.y * gridDim.x + st) * tc8_blob_bytes(npad);
    qs += (size_t)blockIdx.y * npad * K;
    ds += (size_t)blockIdx.y * npad * (K / 32);
    N = min(npad, N - (int)blockIdx.y * npad);
    for (int u = threadIdx.x; u < npad * 16; u += blockDim.x) {
        const int n = u / 16, kc = u % 16;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (n < N) v = *reinterpret_cast<const uint4 *>(qs + (size_t)n * K + (size_t)st * 256 + kc * 16);
        *reinterpret_cast<uint4 *>(o + (size_t)(n / 8) * 2048 + kc * 128 + (n % 8) * 16) = v;
    }
    float *od = reinterpret_cast<float *>(o + (size_t)npad * 256);
    for (int u = threadIdx.x; u < npad * 8; u += blockDim.x) {
        const int b = u / npad, n = u % npad;
        od[u] = n < N ? ds[(size_t)n * (K / 32) + (size_t)st * 8 + b] : 0.f;
    }
}

struct Tc8Params {
    const uint8_t *act;
    float *out;
    int64_t M;
    int N, npad, nst, st_per_split, n_split;
    int64_t ldy;
    int *err;
};

namespace tc8 {
__device__ __forceinline__ void umma_i8_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16i(uint32_t taddr, int (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                   "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8i(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}

// The two blocks (2G, 2G+1) of a row's 272-byte chunk are bytes [68G, 68G+68) = 17 words that start G
// words into a 16-byte unit; five aligned 128-bit reads cover them for every G. Block 2G has its scale
// in the low half of the first word and its codes 2 bytes in; block 2G+1 has its scale in the high half
// of word 8 and its codes word-aligned after it.
template <int G>
__device__ __forceinline__ void split_blocks(const uint8_t *row, uint32_t (&qa)[8], uint32_t (&qb)[8], float &da, float &db) {
    constexpr int U0 = (68 * G) / 16;      // first 16-byte unit
    constexpr int W0 = (68 * G) / 4 - 4 * U0;   // word of the chunk start inside it (= G)
    uint32_t w[20];
#pragma unroll
    for (int u = 0; u < 5; u++) {
        // for G = 3 the fifth unit is bytes 256..271: the last one of the row
        const uint4 v = *reinterpret_cast<const uint4 *>(row + (U0 + u) * 16);
        w[4 * u] = v.x; w[4 * u + 1] = v.y; w[4 * u + 2] = v.z; w[4 * u + 3] = v.w;
    }
    da = __half2float(__ushort_as_half((unsigned short)(w[W0] & 0xffffu)));
#pragma unroll
    for (int j = 0; j < 8; j++) qa[j] = __funnelshift_r(w[W0 + j], w[W0 + j + 1], 16);
    db = __half2float(__ushort_as_half((unsigned short)(w[W0 + 8] >> 16)));
#pragma unroll
    for (int j = 0; j < 8; j++) qb[j] = w[W0 + 9 + j];
}

// The same for a row's 144-byte chunk of Q4_0 blocks: bytes [36G, 36G + 36) = 9 words in three units. A word of codes has elements
// 4j .. 4j + 3 in its low nibbles and 16 + 4j .. in its high ones; nibble - 8 as a signed byte is ((nibble | 0x80) - 8) ^ 0x80.
__device__ __forceinline__ void nibbles_signed(uint32_t w, uint32_t &lo, uint32_t &hi) {
    lo = (((w & 0x0f0f0f0fu) | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
    hi = ((((w >> 4) & 0x0f0f0f0fu) | 0x80808080u) - 0x08080808u) ^ 0x80808080u;
}
template <int G>
__device__ __forceinline__ void split_blocks4(const uint8_t *row, uint32_t (&qa)[8], uint32_t (&qb)[8], float &da, float &db) {
    constexpr int U0 = (36 * G) / 16, W0 = (36 * G) / 4 - 4 * U0;
    uint32_t w[12];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const uint4 v = *reinterpret_cast<const uint4 *>(row + (U0 + u) * 16);
        w[4 * u] = v.x; w[4 * u + 1] = v.y; w[4 * u + 2] = v.z; w[4 * u + 3] = v.w;
    }
    da = __half2float(__ushort_as_half((unsigned short)(w[W0] & 0xffffu)));
    db = __half2float(__ushort_as_half((unsigned short)(w[W0 + 4] >> 16)));
#pragma unroll
    for (int j = 0; j < 4; j++) {
        nibbles_signed(__funnelshift_r(w[W0 + j], w[W0 + j + 1], 16), qa[j], qa[4 + j]);
        nibbles_signed(w[W0 + 5 + j], qb[j], qb[4 + j]);
    }
}
template <bool Q4, int G>
__device__ __forceinline__ void row_blocks(const uint8_t *row, uint32_t (&qa)[8], uint32_t (&qb)[8], float &da, float &db) {
    if constexpr (Q4) split_blocks4<G>(row, qa, qb, da, db);
    else split_blocks<G>(row, qa, qb, da, db);
}
}  // namespace tc8

template <bool Q4, int NPAD, int RAW_STAGES, int ACT_STAGES>
__global__ void __launch_bounds__(tc8::THREADS, 1) k_mmq_tc_q80(const __grid_constant__ CUtensorMap wmap, Tc8Params p) {
    using namespace tc;
    using namespace tc8;
    constexpr int ROWS = tc8::ROWS;
    constexpr int BLOB = NPAD * 288, ROW_CHUNK = tc8::row_chunk(Q4), RAW_BYTES = tc8::raw_bytes(Q4);
    // int8 x int8 -> int32, K-major A and B: c_format s32 (2) at bit 4, a/b format signed 8-bit (1) at bits 7 and 10
    constexpr uint32_t IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NPAD >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
    constexpr int GCOLS = 4 * NPAD;   // accumulator columns of one group of four blocks
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
    uint8_t *raw = smem;                                              // RAW_STAGES x RAW_BYTES
    uint8_t *actb = raw + RAW_STAGES * RAW_BYTES;                // ACT_STAGES x BLOB
    float *dw = reinterpret_cast<float *>(actb + ACT_STAGES * BLOB);  // [A_RING][8][ROWS] weight scales
    __shared__ uint64_t bar_raw[RAW_STAGES], bar_rawfree[RAW_STAGES], bar_act[ACT_STAGES], bar_actfree[ACT_STAGES];
    __shared__ uint64_t bar_aready[tc8::A_RING], bar_afree[tc8::A_RING], bar_dwfree[tc8::A_RING], bar_mma[2], bar_epi[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_fail;
    volatile int *fail = &s_fail;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row_tile = blockIdx.x, split = blockIdx.y;
    const int st0 = split * p.st_per_split;
    const int nst = min(p.st_per_split, p.nst - st0);
    if (tid == 0) {
        for (int i = 0; i < RAW_STAGES; i++) {
            mbar_init(&bar_raw[i], 1);
            mbar_init(&bar_rawfree[i], 16);
        }
        for (int i = 0; i < ACT_STAGES; i++) {
            mbar_init(&bar_act[i], 1);
            mbar_init(&bar_actfree[i], 256);
        }
        for (int i = 0; i < tc8::A_RING; i++) {
            mbar_init(&bar_aready[i], 16);
            mbar_init(&bar_afree[i], 1);
            mbar_init(&bar_dwfree[i], 256);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar_mma[i], 1);
            mbar_init(&bar_epi[i], 256);
        }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(&tmem_base_s, tc8::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    auto load_raw = [&](int i) {
        const int s = i % RAW_STAGES;
        mbar_expect_tx(&bar_raw[s], RAW_BYTES);
        tma_2d(raw + s * RAW_BYTES, &wmap, (st0 + i) * (ROW_CHUNK / 2), row_tile * ROWS, &bar_raw[s]);   // x in 16-bit elements
    };
    auto load_act = [&](int i) {
        const int s = i % ACT_STAGES;
        mbar_expect_tx(&bar_act[s], BLOB);
        bulk_g2s(actb + s * BLOB, p.act + (size_t)(st0 + i) * BLOB, BLOB, &bar_act[s]);
    };
    // weights first, then the dependency wait, then activations (see k_mmq_tc.cu)
    griddep_launch();
    if (tid == 0)
        for (int i = 0; i < nst && i < RAW_STAGES; i++) load_raw(i);
    griddep_wait();
    if (tid == 0)
        for (int i = 0; i < nst && i < ACT_STAGES; i++) load_act(i);

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            for (int i = 0; i < nst; i++) {
                if (i + RAW_STAGES < nst) {
                    mbar_wait_relaxed(&bar_rawfree[i % RAW_STAGES], (uint32_t)((i / RAW_STAGES) & 1), fail);
                    load_raw(i + RAW_STAGES);
                }
                if (i >= 1 && i - 1 + ACT_STAGES < nst) {
                    mbar_wait_relaxed(&bar_actfree[(i - 1) % ACT_STAGES], (uint32_t)(((i - 1) / ACT_STAGES) & 1), fail);
                    load_act(i - 1 + ACT_STAGES);
                }
            }
        }
    } else if (warp == tc8::MMA_WARP) {
        // ---- MMA issuer: the whole warp runs the loop (converged), one elected lane issues
        const bool leader = elect_one();
        for (int i = 0; i < nst; i++) {
            const int as = i % ACT_STAGES, slot = i % tc8::A_RING;
            const uint64_t b_desc0 = smem_desc(su32(actb + as * BLOB), 128, 2048);
            mbar_wait(&bar_act[as], (uint32_t)((i / ACT_STAGES) & 1), fail);
            mbar_wait(&bar_aready[slot], (uint32_t)((i / tc8::A_RING) & 1), fail);
            tc_fence_after();
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                const int G = 2 * i + hh, gb = G & 1;
                if (G >= 2) {
                    mbar_wait(&bar_epi[gb], (uint32_t)(((G - 2) >> 1) & 1), fail);   // accumulator group gb drained
                    tc_fence_after();
                }
                if (leader) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const int blk = 4 * hh + j;
                        umma_i8_ta(tmem_base + (uint32_t)(gb * GCOLS + j * NPAD), tmem_base + tc8::A_COL0 + (uint32_t)(slot * 64 + blk * 8),
                                   b_desc0 + (uint64_t)(blk * (256 >> 4)), IDESC);
                    }
                    umma_commit(&bar_mma[gb]);
                    if (hh == 1) umma_commit(&bar_afree[slot]);
                }
                __syncwarp();
            }
        }
    } else if (warp < tc8::DEQ_WARP0) {
        // ---- epilogue: two warps per TMEM lane quadrant split the columns
        const int q = warp & 3;
        const int row_in_tile = q * 32 + lane;
        constexpr int CW = NPAD / 2;
        const int col0 = ((warp - tc8::EPI_WARP0) >> 2) * CW;
        float yacc[CW];
#pragma unroll
        for (int c = 0; c < CW; c++) yacc[c] = 0.f;
        for (int i = 0; i < nst; i++) {
            const int as = i % ACT_STAGES, slot = i % tc8::A_RING;
            const float *da = reinterpret_cast<const float *>(actb + as * BLOB + NPAD * 256) + col0;   // [8][NPAD]
            const float *dwr = dw + (size_t)slot * 8 * ROWS + row_in_tile;
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                const int G = 2 * i + hh, gb = G & 1;
                mbar_wait_relaxed(&bar_mma[gb], (uint32_t)((G >> 1) & 1), fail);
                tc_fence_after();
                const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(gb * GCOLS + col0);
#pragma unroll
                for (int jp = 0; jp < 4; jp += 2) {
                    int D0[CW], D1[CW];
                    if constexpr (CW == 8) {
                        tmem_ld8i(lane_addr + jp * NPAD, *reinterpret_cast<int(*)[8]>(&D0[0]));
                        tmem_ld8i(lane_addr + (jp + 1) * NPAD, *reinterpret_cast<int(*)[8]>(&D1[0]));
                    } else {
                        tmem_ld16i(lane_addr + jp * NPAD, *reinterpret_cast<int(*)[16]>(&D0[0]));
                        tmem_ld16i(lane_addr + (jp + 1) * NPAD, *reinterpret_cast<int(*)[16]>(&D1[0]));
                    }
                    tmem_ld_wait();
                    if (jp == 2) {
                        tc_fence_before();
                        mbar_arrive(&bar_epi[gb]);   // accumulator group gb may be overwritten
                    }
                    const int b0 = 4 * hh + jp;
                    const float w0 = dwr[b0 * ROWS], w1 = dwr[(b0 + 1) * ROWS];
#pragma unroll
                    for (int c = 0; c < CW; c++) {
                        yacc[c] += (float)D0[c] * (w0 * da[b0 * NPAD + c]);
                        yacc[c] += (float)D1[c] * (w1 * da[(b0 + 1) * NPAD + c]);
                    }
                }
            }
            mbar_arrive(&bar_dwfree[slot]);
            mbar_arrive(&bar_actfree[as]);
        }
        const int64_t row = (int64_t)row_tile * ROWS + row_in_tile;
        if (row < p.M) {
            float *o = p.out + (size_t)split * p.N * p.ldy + row;
#pragma unroll
            for (int c = 0; c < CW; c++)
                if (col0 + c < p.N) o[(size_t)(col0 + c) * p.ldy] = yacc[c];
        }
    } else {
        // ---- realigning warps: lane quadrant = warp % 4 fixes the rows; per quadrant four warps take two blocks each
        const int g = (warp - tc8::DEQ_WARP0) >> 2;
        const int r = (warp & 3) * 32 + lane;
        const uint32_t a_lane = tmem_base + tc8::A_COL0 + ((uint32_t)((warp & 3) * 32) << 16);
        for (int i = 0; i < nst; i++) {
            const int rs = i % RAW_STAGES, slot = i % tc8::A_RING;
            mbar_wait(&bar_raw[rs], (uint32_t)((i / RAW_STAGES) & 1), fail);
            const uint8_t *rrow = raw + rs * RAW_BYTES + r * ROW_CHUNK;
            uint32_t qa[8], qb[8];
            float da, db;
            switch (g) {   // warp-uniform
                case 0: row_blocks<Q4, 0>(rrow, qa, qb, da, db); break;
                case 1: row_blocks<Q4, 1>(rrow, qa, qb, da, db); break;
                case 2: row_blocks<Q4, 2>(rrow, qa, qb, da, db); break;
                default: row_blocks<Q4, 3>(rrow, qa, qb, da, db); break;
            }
            if (i >= tc8::A_RING) {
                // the MMAs that read this ring slot are done, and the epilogue has read its scales
                mbar_wait(&bar_afree[slot], (uint32_t)(((i / tc8::A_RING) - 1) & 1), fail);
                mbar_wait(&bar_dwfree[slot], (uint32_t)(((i / tc8::A_RING) - 1) & 1), fail);
                tc_fence_after();
            }
            tmem_st8(a_lane + (uint32_t)(slot * 64 + (2 * g) * 8), qa);
            tmem_st8(a_lane + (uint32_t)(slot * 64 + (2 * g + 1) * 8), qb);
            float *dws = dw + (size_t)slot * 8 * ROWS + r;
            dws[(2 * g) * ROWS] = da;
            dws[(2 * g + 1) * ROWS] = db;
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bar_aready[slot]);
                mbar_arrive(&bar_rawfree[rs]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, tc8::TMEM_COLS);
    if (tid == 0 && s_fail) report_error(p.err, 2);
}

// ---------------------------------------------------------------- many activation columns (prompt pass)
// Same arithmetic, a 128-row x 128-column output tile per CTA (grid: row tiles x column tiles, row tiles
// fastest so that the CTAs in flight share a few activation blobs and sweep the weights through L2).
// One MMA (128 x 128 x 32) per block into one of two accumulators; every block's accumulator has to come back
// out of tensor memory (64 KB per block and tile) and costs an int->float conversion, a scale product and an
// FMA per element. That drain bounds this kernel, not the MMA (measured: 490 us of 790 with the arithmetic
// left out, tensor pipe 7% busy), so sixteen warps drain (lane quadrant x 32-column slice, sums in registers,
// two f32 lanes per instruction), four realign the weight codes, one issues MMAs, one TMA copies; the warps
// that mostly wait nap between probes.
namespace tc8w {
constexpr int NW = 128;                                  // activation columns per tile
constexpr int EPI_WARPS = 16, DEQ_WARPS = 4;
constexpr int EPI_WARP0 = 1, DEQ_WARP0 = EPI_WARP0 + EPI_WARPS, MMA_WARP = DEQ_WARP0 + DEQ_WARPS;
constexpr int THREADS = (MMA_WARP + 1) * 32;             // 704
constexpr int RAW_STAGES = 2, ACT_STAGES = 3;
constexpr int N_ACC = 3;                                 // accumulators of NW columns in tensor memory columns [0, 384)
constexpr uint32_t A_COL0 = N_ACC * NW;                  // the A ring behind them: 2 stages x 64 columns
constexpr int A_RING = 2;
constexpr int BLOB = NW * 288;
constexpr int CW = NW / (EPI_WARPS / 4);                 // 32 columns per draining warp
// two f32 lanes per instruction (each lane rounds as the scalar instruction does)
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// y += float(D) * (w * s) for 16 columns
__device__ __forceinline__ void drain16(uint64_t *y, const int (&D)[16], uint64_t ww, const ulonglong2 *s) {
#pragma unroll
    for (int c4 = 0; c4 < 4; c4++) {
        const ulonglong2 sv = s[c4];
        y[2 * c4] = fma2(pack2((float)D[4 * c4], (float)D[4 * c4 + 1]), mul2(ww, sv.x), y[2 * c4]);
        y[2 * c4 + 1] = fma2(pack2((float)D[4 * c4 + 2], (float)D[4 * c4 + 3]), mul2(ww, sv.y), y[2 * c4 + 1]);
    }
}
}  // namespace tc8w

template <bool Q4>
__global__ void __launch_bounds__(tc8w::THREADS, 1) k_mmq_tc_q80_wide(const __grid_constant__ CUtensorMap wmap, Tc8Params p) {
    using namespace tc;
    using namespace tc8w;
    constexpr int ROWS = tc8::ROWS, ROW_CHUNK = tc8::row_chunk(Q4), RAW_BYTES = tc8::raw_bytes(Q4);
    constexpr int A_RING = tc8w::A_RING;
    constexpr uint32_t IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NW >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
    uint8_t *raw = smem;                                              // RAW_STAGES x RAW_BYTES
    uint8_t *actb = raw + RAW_STAGES * RAW_BYTES;                // ACT_STAGES x BLOB
    float *dw = reinterpret_cast<float *>(actb + ACT_STAGES * BLOB);  // [A_RING][8][ROWS] weight scales
    __shared__ uint64_t bar_raw[RAW_STAGES], bar_rawfree[RAW_STAGES], bar_act[ACT_STAGES], bar_actfree[ACT_STAGES];
    __shared__ uint64_t bar_aready[A_RING], bar_afree[A_RING], bar_dwfree[A_RING], bar_mma[N_ACC], bar_epi[N_ACC];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_fail;
    volatile int *fail = &s_fail;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row_tile = blockIdx.x, col_tile = blockIdx.y;
    const int nst = p.nst;
    const uint8_t *act = p.act + (size_t)col_tile * nst * BLOB;
    if (tid == 0) {
        for (int i = 0; i < RAW_STAGES; i++) {
            mbar_init(&bar_raw[i], 1);
            mbar_init(&bar_rawfree[i], DEQ_WARPS);
        }
        for (int i = 0; i < ACT_STAGES; i++) {
            mbar_init(&bar_act[i], 1);
            mbar_init(&bar_actfree[i], EPI_WARPS);
        }
        for (int i = 0; i < A_RING; i++) {
            mbar_init(&bar_aready[i], DEQ_WARPS);
            mbar_init(&bar_afree[i], 1);
            mbar_init(&bar_dwfree[i], EPI_WARPS);
        }
        for (int i = 0; i < N_ACC; i++) {
            mbar_init(&bar_mma[i], 1);
            mbar_init(&bar_epi[i], EPI_WARPS);   // one arrival per draining warp
        }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(&tmem_base_s, tc8::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;

    auto load_raw = [&](int i) {
        const int s = i % RAW_STAGES;
        mbar_expect_tx(&bar_raw[s], RAW_BYTES);
        tma_2d(raw + s * RAW_BYTES, &wmap, i * (ROW_CHUNK / 2), row_tile * ROWS, &bar_raw[s]);   // x in 16-bit elements
    };
    auto load_act = [&](int i) {
        const int s = i % ACT_STAGES;
        mbar_expect_tx(&bar_act[s], BLOB);
        bulk_g2s(actb + s * BLOB, act + (size_t)i * BLOB, BLOB, &bar_act[s]);
    };
    griddep_launch();
    if (tid == 0)
        for (int i = 0; i < nst && i < RAW_STAGES; i++) load_raw(i);
    griddep_wait();
    if (tid == 0)
        for (int i = 0; i < nst && i < ACT_STAGES; i++) load_act(i);

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            for (int i = 0; i < nst; i++) {
                if (i + RAW_STAGES < nst) {
                    mbar_wait_relaxed(&bar_rawfree[i % RAW_STAGES], (uint32_t)((i / RAW_STAGES) & 1), fail);
                    load_raw(i + RAW_STAGES);
                }
                if (i + ACT_STAGES < nst) {
                    mbar_wait_relaxed(&bar_actfree[i % ACT_STAGES], (uint32_t)((i / ACT_STAGES) & 1), fail);
                    load_act(i + ACT_STAGES);
                }
            }
        }
    } else if (warp == tc8w::MMA_WARP) {
        // ---- MMA issuer: the whole warp runs the loop (converged), one elected lane issues
        const bool leader = elect_one();
        int gb = 0;            // accumulator of block G = 8 * i + blk: G % N_ACC, in its (G / N_ACC)-th use
        uint32_t use = 0;
        for (int i = 0; i < nst; i++) {
            const int as = i % ACT_STAGES, slot = i % A_RING;
            const uint64_t b_desc0 = smem_desc(su32(actb + as * BLOB), 128, 2048);
            mbar_wait_nap(&bar_act[as], (uint32_t)((i / ACT_STAGES) & 1), fail, 32);
            mbar_wait_nap(&bar_aready[slot], (uint32_t)((i / A_RING) & 1), fail, 32);
            tc_fence_after();
#pragma unroll 1
            for (int blk = 0; blk < 8; blk++) {
                if (use > 0) {
                    mbar_wait_nap(&bar_epi[gb], (use - 1) & 1, fail, 32);   // accumulator gb drained
                    tc_fence_after();
                }
                if (leader) {
                    tc8::umma_i8_ta(tmem_base + (uint32_t)(gb * NW), tmem_base + tc8w::A_COL0 + (uint32_t)(slot * 64 + blk * 8),
                                    b_desc0 + (uint64_t)(blk * (256 >> 4)), IDESC);
                    umma_commit(&bar_mma[gb]);
                    if (blk == 7) umma_commit(&bar_afree[slot]);
                }
                __syncwarp();
                if (++gb == N_ACC) {
                    gb = 0;
                    use++;
                }
            }
        }
    } else if (warp < tc8w::DEQ_WARP0) {
        // ---- draining warps: TMEM lane quadrant warp % 4, column slice (warp - 1) / 4
        const int q = warp & 3;
        const int row_in_tile = q * 32 + lane;
        const int col0 = ((warp - tc8w::EPI_WARP0) >> 2) * CW;
        static_assert(CW == 32, "the draining loop below takes two 16-column loads per block");
        uint64_t yacc[CW / 2];
#pragma unroll
        for (int c = 0; c < CW / 2; c++) yacc[c] = 0ull;   // two +0.0f
        const uint32_t lane_addr0 = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)col0;
        int gb = 0;
        uint32_t use = 0;
        for (int i = 0; i < nst; i++) {
            const int as = i % ACT_STAGES, slot = i % A_RING;
            const float *da = reinterpret_cast<const float *>(actb + as * BLOB + NW * 256) + col0;   // [8][NW]
            const float *dwr = dw + (size_t)slot * 8 * ROWS + row_in_tile;
#pragma unroll 1
            for (int blk = 0; blk < 8; blk++) {
                mbar_wait_relaxed(&bar_mma[gb], use & 1, fail);
                tc_fence_after();
                const float w = dwr[blk * ROWS];
                const uint64_t ww = pack2(w, w);
                const ulonglong2 *dab = reinterpret_cast<const ulonglong2 *>(da + blk * NW);
                // the second load is in flight while the first half is added up
                int D0[16], D1[16];
                tc8::tmem_ld16i(lane_addr0 + (uint32_t)(gb * NW), D0);
                tmem_ld_wait();
                tc8::tmem_ld16i(lane_addr0 + (uint32_t)(gb * NW + 16), D1);
                drain16(yacc, D0, ww, dab);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_epi[gb]);   // accumulator gb may be overwritten
                drain16(yacc + 8, D1, ww, dab + 4);
                if (++gb == N_ACC) {
                    gb = 0;
                    use++;
                }
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bar_dwfree[slot]);
                mbar_arrive(&bar_actfree[as]);
            }
        }
        const int64_t row = (int64_t)row_tile * ROWS + row_in_tile;
        const int ncol = min(NW, p.N - col_tile * NW);
        if (row < p.M) {
            float *o = p.out + (size_t)col_tile * NW * p.ldy + row;
#pragma unroll
            for (int c = 0; c < CW / 2; c++) {
                float lo, hi;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(yacc[c]));
                if (col0 + 2 * c < ncol) o[(size_t)(col0 + 2 * c) * p.ldy] = lo;
                if (col0 + 2 * c + 1 < ncol) o[(size_t)(col0 + 2 * c + 1) * p.ldy] = hi;
            }
        }
    } else {
        // ---- realigning warps: lane quadrant = warp % 4 fixes the rows, every warp takes all eight blocks of its rows
        const int r = (warp & 3) * 32 + lane;
        const uint32_t a_lane = tmem_base + tc8w::A_COL0 + ((uint32_t)((warp & 3) * 32) << 16);
        for (int i = 0; i < nst; i++) {
            const int rs = i % RAW_STAGES, slot = i % A_RING;
            mbar_wait_nap(&bar_raw[rs], (uint32_t)((i / RAW_STAGES) & 1), fail, 128);
            if (i >= A_RING) {
                // the MMAs that read this ring slot are done, and the draining warps have read its scales
                mbar_wait_nap(&bar_afree[slot], (uint32_t)(((i / A_RING) - 1) & 1), fail, 128);
                mbar_wait_nap(&bar_dwfree[slot], (uint32_t)(((i / A_RING) - 1) & 1), fail, 128);
                tc_fence_after();
            }
            const uint8_t *rrow = raw + rs * RAW_BYTES + r * ROW_CHUNK;
            float *dws = dw + (size_t)slot * 8 * ROWS + r;
#pragma unroll
            for (int g = 0; g < 4; g++) {
                uint32_t qa[8], qb[8];
                float da, db;
                if (g == 0) tc8::row_blocks<Q4, 0>(rrow, qa, qb, da, db);
                else if (g == 1) tc8::row_blocks<Q4, 1>(rrow, qa, qb, da, db);
                else if (g == 2) tc8::row_blocks<Q4, 2>(rrow, qa, qb, da, db);
                else tc8::row_blocks<Q4, 3>(rrow, qa, qb, da, db);
                tmem_st8(a_lane + (uint32_t)(slot * 64 + (2 * g) * 8), qa);
                tmem_st8(a_lane + (uint32_t)(slot * 64 + (2 * g + 1) * 8), qb);
                dws[(2 * g) * ROWS] = da;
                dws[(2 * g + 1) * ROWS] = db;
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&bar_aready[slot]);
                mbar_arrive(&bar_rawfree[rs]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, tc8::TMEM_COLS);
    if (tid == 0 && s_fail) report_error(p.err, 2);
}

// ---------------------------------------------------------------- many activation columns, one accumulator (prompt pass)
// The kernel above pays for the reference's arithmetic with one accumulator round trip per 32-element block. This one
// folds both scales into the operands instead and lets the tensor core add up the whole of K:
//     A[r,k] = f16(d_w[r,b] * q[r,k])        (HMUL2 of the exact code by the block's f16 scale: one rounding)
//     B[k,c] = f16(d_a[c,b] * q8[k,c])       (by the activation packer, from the same Q8_0 quantization of the activations
//                                             that the reference makes: one rounding)
//     y[r,c] = sum_k A[r,k] * B[k,c]         (tcgen05.mma kind::f16, f32 accumulator in tensor memory)
// Each product carries two f16 roundings (2^-12 relative each, independent across k), so y differs from the reference's
// integer arithmetic by about 1e-4 of max|y| at K = 4096: inside the 1e-3 bar of mul_mat, not bit-comparable. The exact
// kernel above stays reachable (TLB_PROMPT_EXACT=1).
// A pair of CTAs (the two SMs of a cluster, tcgen05 cta_group::2) walks items: a tile of 256 weight rows x up to 256 (or 2 x 192) activation
// columns, or a stretch of its K. Per 256 elements of K each CTA brings its 128 rows of raw weights by TMA; sixteen warps strip the
// scales, turn the codes into scaled f16 and store them into its tensor memory (A operand, 32 columns per 64 elements of K); each
// CTA brings half of the tile's columns of the packed B (core matrix layout) and the matrix instruction reads both halves. One
// thread of the pair issues four MMAs of 256 x columns x 16 per 64 elements of K. Eight warps per CTA drain its accumulator once
// per item; tiles of at most 192 columns have two, so that the next item's MMAs do not wait for that.
//
// Why pairs: the copies of B bound wide tiles of single CTAs. 148 of them, each with the B of its own 128 rows, read 11 to 12.5 TB/s out
// of L2 (2.4 us per unit of 256 elements of K at 336 columns, 1.55 at 256, whose MMAs take 1.45 and 1.1); the pair reads each
// column once for 256 rows. The threads' arrivals on the leader's barriers are of CTA scope: they only pass tensor memory on, between
// tcgen05 fences (a release of cluster scope made a unit 2.0 us instead of 1.15 at 64 columns). The columns of B that the other CTA copied
// arrive on the leader's barrier by themselves. The expanding warps fetch and expand before they wait for their slot (the wait, fetch,
// expansion and store as one chain took 1000 cycles of a slot's round).
//
// What bounds it: narrow tiles the expansion's instructions (326 per warp and unit for Q4_K, 268 for Q8_0, four warps per scheduler; 404 with
// codes through f32 one by one: gate and up of 14336 x 4096 at 128 columns 52 -> 47 us); wide ones the tensor pipe: 16384 columns run at
// 1400 to 1456 TFLOP/s (1253 to 1346 with single CTAs).
// The tile's width follows from rows, columns and the measured time of a unit; tiles that leave SMs idle are cut along K and their
// parts added up by a second launch (mm_fold_plan). Matrices that share the activations are one launch. 333 columns, Q4_K, cold:
// [4096 x 14336] 70 -> 50 us, gate and up (14336 x 4096) 86 -> 82, [4096 x 4096] 31 either way; 65 columns of [4096 x 14336] 68 -> 32.
namespace tc8f {
constexpr int NW = MM_FOLD_NPAD;                         // widest column tile
constexpr int MAX_MATS = 3;
constexpr int KS = 64;                                   // elements of K per B stage
constexpr int HALF_NW = 192;                             // and of one of two that share their weights
constexpr int MAX_STAGES = 8, MAX_CUTS = 8;
constexpr int SMEM = 226 * 1024;
constexpr int TMA_RAW_WARP = 0, TMA_B_WARP = 1, MMA_WARP = 2;   // warp 3 idles (keeps the quadrant numbering of the rest aligned)
constexpr int DEQ_WARP0 = 4, DEQ_WARPS = 16, EPI_WARP0 = 20, EPI_WARPS = 8;
constexpr int THREADS = (EPI_WARP0 + EPI_WARPS) * 32;    // 896
// 4 int8 codes of a word -> two f16x2 of code * scale (exact integer first: (1024 + u) - 1152 with u = code + 128)
__device__ __forceinline__ void codes_to_f16(uint32_t w, uint32_t dd, uint32_t &lo, uint32_t &hi) {
    const uint32_t x = w ^ 0x80808080u;
    uint32_t a = __byte_perm(x, 0x64646464u, 0x4140), b = __byte_perm(x, 0x64646464u, 0x4342);
    const uint32_t k1152 = 0x64806480u;   // f16x2 (1152, 1152)
    asm("sub.f16x2 %0, %0, %1;" : "+r"(a) : "r"(k1152));
    asm("sub.f16x2 %0, %0, %1;" : "+r"(b) : "r"(k1152));
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(dd));
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(hi) : "r"(b), "r"(dd));
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
}
}  // namespace tc8f

// B operand of the kernel below from an ActLayout block: mm_fold_at, values f16(d_a * q8) in the order of K.
// `blk`: elements per activation scale (32 for Q8_0 activations, 256 for the Q8_K activations of Q4_K weights).
__global__ void __launch_bounds__(256) k_act_pack_q80_f16(const int8_t *__restrict__ qs, const float *__restrict__ ds, int64_t K, int N, int blk,
                                                           uint8_t *__restrict__ out) {
    const int st = blockIdx.x;   // stage of 64 elements
    const int groups = mm_fold_groups(N);
    const int u_end = min(groups * 8, (int)(blockIdx.y + 1) * tc8f::NW) * 8;
    for (int u = (int)blockIdx.y * tc8f::NW * 8 + threadIdx.x; u < u_end; u += blockDim.x) {
        const int n = u / 8;
        const int64_t k0 = (int64_t)st * tc8f::KS + u % 8 * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (n < N) {
            const uint2 q = *reinterpret_cast<const uint2 *>(qs + (size_t)n * K + k0);
            const float d = ds[(size_t)n * (K / blk) + k0 / blk];
            const uint32_t w[2] = {q.x, q.y};
            uint32_t h[4];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float f0 = (float)(int8_t)(w[i] & 0xff), f1 = (float)(int8_t)((w[i] >> 8) & 0xff), f2 = (float)(int8_t)((w[i] >> 16) & 0xff),
                            f3 = (float)(int8_t)(w[i] >> 24);
                const __half2 a = __floats2half2_rn(f0 * d, f1 * d), b = __floats2half2_rn(f2 * d, f3 * d);
                h[2 * i] = *reinterpret_cast<const uint32_t *>(&a);
                h[2 * i + 1] = *reinterpret_cast<const uint32_t *>(&b);
            }
            v = make_uint4(h[0], h[1], h[2], h[3]);
        }
        *reinterpret_cast<uint4 *>(out + mm_fold_at(n, k0, groups)) = v;
    }
}

struct Tc8fMaps {
    CUtensorMap m[tc8f::MAX_MATS];
    CUtensorMap act[2];   // pairs: the packed B as rows of eight columns x 64 of K, boxes of one CTA's share of a tile or of either half
};
// One pass of a pair: a tile's rows and columns and its stretch of K; part >= 0: the tile's sum is cut, this is its part's number.
struct FoldItem {
    int row_tile, col_tile, k0, k1, part;
};
struct Tc8fParams {
    const uint8_t *act;   // packed B operand
    float *out[tc8f::MAX_MATS];
    float *part;          // [part][column of the tile][tile_rows]
    int64_t M[tc8f::MAX_MATS], ldy[tc8f::MAX_MATS];
    int tile0[tc8f::MAX_MATS];   // first row tile of each matrix (past the end: not there)
    int N, nst, tile_rows, row_tiles, col_tiles, groups;
    int nw, width;               // columns of a tile or of its first half; of a tile
    int whole, cuts, items;      // tiles [whole, row_tiles * col_tiles) are cut into `cuts` stretches of K
    int raw_stages, b_stages;
    int *err;
    // Tile t: column tiles in bands of eight, the eight of a row tile one after the other. A band's share of B stays in L2 and the
    // weights come past it once per band (gate and up of a layer, 125 MB in Q8_0, do not fit into L2 beside it).
    __device__ __forceinline__ void at(int t, int &row_tile, int &col_tile) const {
        const int per = row_tiles * 8, band = t / per, in = t - band * per, width = min(8, col_tiles - band * 8);
        row_tile = in / width;
        col_tile = band * 8 + in - row_tile * width;
    }
    __device__ __forceinline__ FoldItem item(int i) const {
        FoldItem f{0, 0, 0, nst, -1};
        int t = i;
        if (i >= whole) {
            f.part = i - whole;
            const int c = f.part / cuts, s = f.part - c * cuts;
            t = whole + c;
            f.k0 = nst * s / cuts;
            f.k1 = nst * (s + 1) / cuts;
        }
        at(t, f.row_tile, f.col_tile);
        return f;
    }
    __device__ __forceinline__ int mat_of(int row_tile) const { return row_tile >= tile0[2] ? 2 : (row_tile >= tile0[1] ? 1 : 0); }
};
// (v & mask) | 0x64006400: two codes of a word as the f16 pair 1024 + code (x 16 for high nibbles in place)
__device__ __forceinline__ uint32_t code_pair(uint32_t v, uint32_t mask) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(v), "r"(mask), "r"(0x64006400u));
    return r;
}
// Four weights d * sc * q - b of the f16 pairs 1024 + (q0, q2) and 1024 + (q1, q3) in the order of K: sc * q is a whole number below
// 946, exact in f16; the rest is one f32 rounding, then f16. (s, s0: sc and -1024 sc as pairs.)
__device__ __forceinline__ void fold_four(uint32_t q02, uint32_t q13, uint32_t s, uint32_t s0, uint16_t d, float nb, uint32_t &w01, uint32_t &w23) {
    asm("{\n\t.reg .b32 t, u;\n\t.reg .b16 t0, t1, t2, t3;\n\t.reg .f32 x0, x1, x2, x3;\n\t"
        "fma.rn.f16x2 t, %2, %4, %5;\n\t"
        "fma.rn.f16x2 u, %3, %4, %5;\n\t"
        "mov.b32 {t0, t2}, t;\n\tmov.b32 {t1, t3}, u;\n\t"
        "fma.rn.f32.f16 x0, t0, %6, %7;\n\t"
        "fma.rn.f32.f16 x1, t1, %6, %7;\n\t"
        "fma.rn.f32.f16 x2, t2, %6, %7;\n\t"
        "fma.rn.f32.f16 x3, t3, %6, %7;\n\t"
        "cvt.rn.f16x2.f32 %0, x1, x0;\n\t"
        "cvt.rn.f16x2.f32 %1, x3, x2;\n\t}"
        : "=r"(w01), "=r"(w23) : "r"(q02), "r"(q13), "r"(s), "r"(s0), "h"(d), "f"(nb));
}

// ---- what the two CTAs of a pair need of each other (rank 0 leads)
__device__ __forceinline__ uint32_t pair_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
template <bool PAIR>
__device__ __forceinline__ void all_sync() {   // of a CTA, or of both
    if constexpr (!PAIR) {
        __syncthreads();
        return;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the shared-memory address of the leader's copy of `p`
__device__ __forceinline__ uint32_t of_leader(const void *p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(tc::su32(p)));
    return r;
}
// on a barrier of this CTA, or at an address that of_leader gave
__device__ __forceinline__ void arrive_at(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// a box of a tensor into this CTA's shared memory; its bytes arrive on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_2d_pair(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(tc::su32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void fold_tmem_alloc(uint32_t *dst_smem, uint32_t cols) {
    if constexpr (!PAIR) return tc::tmem_alloc(dst_smem, cols);
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::su32(dst_smem)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
template <bool PAIR>
__device__ __forceinline__ void fold_tmem_dealloc(uint32_t addr, uint32_t cols) {
    if constexpr (!PAIR) return tc::tmem_dealloc(addr, cols);
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// arrives on the barrier (of a pair: on both CTAs' at this offset) once the MMAs issued so far are done
template <bool PAIR>
__device__ __forceinline__ void fold_commit(uint64_t *bar) {
    if constexpr (!PAIR) return tc::umma_commit(bar);
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(tc::su32(bar)), "h"((uint16_t)3) : "memory");
}
// four MMAs over 64 elements of K: A 8 columns apart in tensor memory, B 16 (x 16 bytes) apart in shared memory; more = 0: the
// first one starts the sum. Of a pair: 256 rows, 128 of each CTA; each CTA holds half of the columns of B.
#define TLB_UMMA4(GROUP)                                                                                                            \
    asm volatile(                                                                                                                   \
        "{\n\t.reg .pred p, q;\n\t.reg .b64 b1, b2, b3;\n\t.reg .b32 a1, a2, a3;\n\tsetp.eq.b32 q, 0, 0;\n\t"                        \
        "setp.ne.b32 p, %4, 0;\n\t"                                                                                                 \
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"                                                      \
        "add.u64 b1, %2, 16;\n\tadd.u64 b2, %2, 32;\n\tadd.u64 b3, %2, 48;\n\t"                                                     \
        "tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], [%1], %2, %3, p;\n\t"                                                     \
        "tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], [a1], b1, %3, q;\n\t"                                                     \
        "tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], [a2], b2, %3, q;\n\t"                                                     \
        "tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], [a3], b3, %3, q;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(more)     \
        : "memory")
template <bool PAIR>
__device__ __forceinline__ void umma4_f16(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t more) {
    if constexpr (PAIR) TLB_UMMA4("2");
    else TLB_UMMA4("1");
}
#undef TLB_UMMA4

// 64 weights (group j of a unit of 256) of one row as f16 pairs, in the order of K.
// Q8_0: two blocks of 34 bytes. Q4_K (one 144-byte super-block: f16 d, dmin, twelve bytes of 6-bit scales and mins, 128 bytes of
// nibbles): f16(d * sc * q - dmin * m), dequantize_row_q4_K (ggml-quants.c); low nibbles are the first 32 values, high ones the rest.
template <bool WQ4K>
__device__ __forceinline__ void expand64(const uint8_t *rrow, int j, uint32_t (&lo)[16], uint32_t (&hi)[16]) {
    if constexpr (WQ4K) {
        const uint4 hdr = *reinterpret_cast<const uint4 *>(rrow);   // d, dmin, scales[12]
        // get_scale_min_k4 (ggml-quants.c:880-887), four sub-blocks at a time
        const uint32_t sc4 = j < 2 ? hdr.y & 0x3f3f3f3fu : (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u);
        const uint32_t mn4 = j < 2 ? hdr.z & 0x3f3f3f3fu : ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u);
        const int sh = (j & 1) * 16;
        const uint16_t d = (uint16_t)hdr.x;
        const float dmin = __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16)));
        const float b0 = -__fmul_rn(dmin, (float)((mn4 >> sh) & 0xff)), b1 = -__fmul_rn(dmin, (float)((mn4 >> (sh + 8)) & 0xff));
        // the scales as f16 pairs: 1024 + sc, less 1024; of the high nibbles (16 x code) a sixteenth
        auto scale = [](uint32_t sc) {
            const uint32_t v = (sc & 0xffu) | 0x6400u;
            uint32_t r;
            asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v | v << 16), "r"(0x64006400u));
            return r;
        };
        auto times = [](uint32_t a, uint32_t f) {
            uint32_t r;
            asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(f));
            return r;
        };
        const uint32_t s = scale(sc4 >> sh), s0 = times(s, 0xe400e400u);                             // x -1024
        const uint32_t t16 = scale(sc4 >> (sh + 8)), t = times(t16, 0x2c002c00u), t0 = times(t16, 0xd400d400u);   // / 16, x -64
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint4 qv = *reinterpret_cast<const uint4 *>(rrow + 16 + j * 32 + u * 16);
            const uint32_t w4[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int wi = 0; wi < 4; wi++) {
                const uint32_t x = w4[wi], y = x >> 8;
                const int at = (u * 4 + wi) * 2;
                fold_four(code_pair(x, 0x000f000fu), code_pair(y, 0x000f000fu), s, s0, d, b0, lo[at], lo[at + 1]);
                fold_four(code_pair(x, 0x00f000f0u), code_pair(y, 0x00f000f0u), t, t0, d, b1, hi[at], hi[at + 1]);
            }
        }
    } else {
        uint32_t qa[8], qb[8];
        float da, db;
        if (j == 0) tc8::split_blocks<0>(rrow, qa, qb, da, db);
        else if (j == 1) tc8::split_blocks<1>(rrow, qa, qb, da, db);
        else if (j == 2) tc8::split_blocks<2>(rrow, qa, qb, da, db);
        else tc8::split_blocks<3>(rrow, qa, qb, da, db);
        uint32_t dd = (uint32_t)__half_as_ushort(__float2half_rn(da));   // the block's own f16 scale, back from f32 unchanged
        dd |= dd << 16;
#pragma unroll
        for (int i = 0; i < 8; i++) tc8f::codes_to_f16(qa[i], dd, lo[2 * i], lo[2 * i + 1]);
        dd = (uint32_t)__half_as_ushort(__float2half_rn(db));
        dd |= dd << 16;
#pragma unroll
        for (int i = 0; i < 8; i++) tc8f::codes_to_f16(qb[i], dd, hi[2 * i], hi[2 * i + 1]);
    }
}

// SHAPE 0: one accumulator of up to 256 columns or (up to 128) two in turn, steps of 128 elements of K; 1: two accumulators of up to 192
// columns in turn, steps of 64; 2: two halves of up to 192 columns, which share the expanded weights, steps of 64. Behind the
// accumulators lie four A slots of a step each.
// PAIR: launched as clusters of two.
template <bool WQ4K, int SHAPE, bool PAIR>
__global__ void __launch_bounds__(tc8f::THREADS, 1) k_mm_q80_f16(const __grid_constant__ Tc8fMaps maps, const __grid_constant__ Tc8fParams p) {
    using namespace tc;
    using namespace tc8f;
    constexpr int ROWS = tc8::ROWS, CTAS = PAIR ? 2 : 1;
    constexpr int ROW_CHUNK = WQ4K ? 144 : tc8::ROW_CHUNK;   // raw bytes of a row per unit of 256 elements
    constexpr int RAW_BYTES = ROWS * ROW_CHUNK;
    constexpr int CT = SHAPE == 2 ? 2 : 1, STEP = SHAPE == 0 ? 2 : 1;   // halves; 64s of K in a step
    constexpr uint32_t ACOLS = SHAPE == 0 ? 256 : 2 * HALF_NW;   // first A column
    constexpr uint32_t ACC2 = SHAPE == 0 ? 128 : HALF_NW;        // second accumulator
    constexpr int A_RING = (512 - (int)ACOLS) / (32 * STEP);
    constexpr uint32_t IDESC0 = (1u << 4) | ((uint32_t)(CTAS * ROWS >> 4) << 24);   // f16 x f16 -> f32, K-major A and B; columns / 8 at bit 17
    const uint32_t idesc[2] = {IDESC0 | ((uint32_t)(p.nw >> 3) << 17), IDESC0 | ((uint32_t)((p.width - p.nw) >> 3) << 17)};
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (su32(smem_raw) & 1023u)) & 1023u);
    const int b_half = p.nw / CTAS * KS * 2, b_stage = b_half * STEP;   // this CTA's columns
    uint8_t *bst = smem;                                   // b_stages x b_stage
    uint8_t *raw = bst + p.b_stages * b_stage;             // raw_stages x RAW_BYTES
    __shared__ uint64_t bar_raw[MAX_STAGES], bar_rawfree[MAX_STAGES], bar_b[MAX_STAGES], bar_bfree[MAX_STAGES];
    __shared__ uint64_t bar_aready[A_RING], bar_afree[A_RING], bar_accfull[2], bar_accfree[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_fail;
    volatile int *fail = &s_fail;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = PAIR ? pair_rank() : 0u;
    const int pair = (int)blockIdx.x / CTAS, pairs = (int)gridDim.x / CTAS;
    const uint32_t accs = SHAPE == 1 || (SHAPE == 0 && p.nw <= 128) ? 2 : 1;   // accumulators in turn
    if (tid == 0) {
        for (int i = 0; i < MAX_STAGES; i++) {
            mbar_init(&bar_raw[i], 1);
            mbar_init(&bar_rawfree[i], tc8f::DEQ_WARPS);
            mbar_init(&bar_b[i], 1);
            mbar_init(&bar_bfree[i], 1);
        }
        for (int i = 0; i < A_RING; i++) {
            mbar_init(&bar_aready[i], CTAS * 4 * STEP);
            mbar_init(&bar_afree[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&bar_accfull[i], 1);
            mbar_init(&bar_accfree[i], CTAS * tc8f::EPI_WARPS);
        }
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) fold_tmem_alloc<PAIR>(&tmem_base_s, 512);
    tc_fence_before();
    all_sync<PAIR>();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    griddep_launch();
    // Every ring: slot s, parity ph of its current round; whoever fills it waits for the parity before (true of a fresh barrier).

    if (warp == tc8f::TMA_RAW_WARP) {
        // ---- raw weights: one box of 128 rows per unit (they do not depend on the kernel in front)
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (int t = pair; t < p.items; t += pairs) {
                const FoldItem f = p.item(t);
                const int mat = p.mat_of(f.row_tile);
                const CUtensorMap *wmap = mat == 0 ? &maps.m[0] : (mat == 1 ? &maps.m[1] : &maps.m[2]);
                const int row0 = (f.row_tile - (mat == 0 ? p.tile0[0] : (mat == 1 ? p.tile0[1] : p.tile0[2]))) * CTAS * ROWS + (int)rank * ROWS;
                for (int i = f.k0; i < f.k1; i++) {
                    mbar_wait_nap(&bar_rawfree[s], ph ^ 1u, fail, 64);
                    mbar_expect_tx(&bar_raw[s], RAW_BYTES);
                    tma_2d(raw + s * RAW_BYTES, wmap, i * (ROW_CHUNK / 2), row0, &bar_raw[s]);   // x in 16-bit elements
                    if (++s == p.raw_stages) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
    } else if (warp == tc8f::TMA_B_WARP) {
        // ---- packed activations: this CTA's columns of each half (at the end what there is, or what comes behind it: columns do not mix; a part
        // that is not there at all gets the last columns once more). Of a pair the copies of both CTAs arrive on the leader's barrier: its matrix
        // instruction reads both, so nothing but the copies themselves may stand between.
        if (lane == 0) {
            griddep_wait();
            const uint32_t bar_lead = PAIR ? of_leader(bar_b) : 0u;
            int s = 0;
            uint32_t ph = 0;
            for (int t = pair; t < p.items; t += pairs) {
                const FoldItem f = p.item(t);
                for (int i = f.k0 * 4; i < f.k1 * 4; i += STEP)
#pragma unroll
                    for (int ct = 0; ct < CT; ct++) {
                        const int mine = (ct == 0 ? p.nw : p.width - p.nw) / (8 * CTAS);   // groups of eight columns
                        const int g0 = min((f.col_tile * p.width + ct * p.nw) / 8 + (int)rank * mine, p.groups - 1);
                        const uint32_t bytes = (uint32_t)(PAIR ? mine : min(mine, p.groups - g0)) * 1024u;
                        mbar_wait_nap(&bar_bfree[s], ph ^ 1u, fail, 32);
                        if (rank == 0) mbar_expect_tx(&bar_b[s], bytes * STEP * CTAS);
#pragma unroll
                        for (int k = 0; k < STEP; k++) {
                            uint8_t *dst = bst + s * b_stage + k * b_half;
                            if constexpr (PAIR) tma_2d_pair(dst, &maps.act[ct], 0, (i + k) * p.groups + g0, bar_lead + (uint32_t)s * 8u);
                            else bulk_g2s(dst, p.act + ((size_t)(i + k) * p.groups + g0) * 1024, bytes, &bar_b[s]);
                        }
                        if (++s == p.b_stages) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
            }
        }
    } else if (warp == tc8f::MMA_WARP) {
        // ---- MMA issuer: one thread of the pair. Its own instructions are what bounds tiles of any width (a warp that probed and issued
        // with all lanes: 750 cycles per 64 elements of K, of which the four MMAs of 256 columns need 512).
        if (rank == 0 && elect_one()) {
            int bs = 0, as = 0;
            uint32_t bph = 0, aph = 0, it = 0;
            const uint64_t b_desc0 = smem_desc(su32(bst), 128, 1024);
            const uint32_t b_step = (uint32_t)b_stage >> 4;
            uint32_t b_at = 0;
            bool b_here = false, a_here = false;
            for (int t = pair; t < p.items; t += pairs, it++) {
                const FoldItem f = p.item(t);
                const uint32_t ai = it % accs;
                mbar_wait_nap(&bar_accfree[ai], ((it / accs) & 1u) ^ 1u, fail, 32);   // the tile before in this accumulator has been drained
                uint32_t more = 0;
#pragma unroll 1
                for (int i = (f.k1 - f.k0) * 4 / STEP; i > 0; i--) {
                    if (!a_here) mbar_wait_nap(&bar_aready[as], aph, fail, 0);
                    const uint32_t a0 = tmem_base + ACOLS + (uint32_t)as * (32u * STEP);
                    uint64_t *const afree = &bar_afree[as];
                    if (++as == A_RING) {
                        as = 0;
                        aph ^= 1u;
                    }
#pragma unroll
                    for (int ct = 0; ct < CT; ct++) {
                        if (!b_here) mbar_wait_nap(&bar_b[bs], bph, fail, 0);
                        if (ct == 0) tc_fence_after();
                        uint64_t *const bfree = &bar_bfree[bs];
                        const uint64_t desc = b_desc0 + b_at;
                        b_at += b_step;
                        if (++bs == p.b_stages) {
                            bs = 0;
                            b_at = 0;
                            bph ^= 1u;
                        }
                        if (ct == CT - 1) a_here = mbar_test(su32(&bar_aready[as]), aph);
                        b_here = mbar_test(su32(&bar_b[bs]), bph);
#pragma unroll
                        for (int k = 0; k < STEP; k++)
                            umma4_f16<PAIR>(tmem_base + (CT == 1 ? ai : (uint32_t)ct) * ACC2, a0 + (uint32_t)k * 32u, desc + (uint64_t)(k * (b_half >> 4)), idesc[ct], k ? 1u : more);
                        fold_commit<PAIR>(bfree);
                    }
                    fold_commit<PAIR>(afree);
                    more = 1;
                }
                fold_commit<PAIR>(&bar_accfull[ai]);
            }
        }
        __syncwarp();
    } else if (warp >= tc8f::DEQ_WARP0 && warp < tc8f::EPI_WARP0) {
        // ---- expanders: lane quadrant warp % 4 fixes the rows; of the four warps of a quadrant each takes 64 elements of a unit, a
        // slot of its own. (A slot's waits, loads and stores are a chain of about 1000 cycles whatever its size: eight warps
        // with 128 elements each took 1.3 us per unit.)
        const int q = warp & 3, j = (warp - tc8f::DEQ_WARP0) >> 2;
        const int r = q * 32 + lane;
        const uint32_t a_lane = tmem_base + ACOLS + ((uint32_t)(q * 32) << 16);
        const uint32_t aready = PAIR ? of_leader(bar_aready) : su32(bar_aready);
        int s = 0, as = j / STEP;
        uint32_t ph = 0, aph = 0;
        for (int t = pair; t < p.items; t += pairs) {
            const FoldItem f = p.item(t);
            for (int i = f.k1 - f.k0; i > 0; i--) {
                mbar_wait_nap(&bar_raw[s], ph, fail, 64);
                uint32_t lo[16], hi[16];
                expand64<WQ4K>(raw + s * RAW_BYTES + r * ROW_CHUNK, j, lo, hi);
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_rawfree[s]);
                mbar_wait_nap(&bar_afree[as], aph ^ 1u, fail, 0);   // the MMAs that read this slot are done
                tc_fence_after();
                const uint32_t to = a_lane + (uint32_t)as * (32u * STEP) + (uint32_t)(j % STEP) * 32u;
                tmem_st16(to, lo);
                tmem_st16(to + 16, hi);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_at(aready + (uint32_t)as * 8u);
                as += 4 / STEP;
                if (as >= A_RING) {
                    as -= A_RING;
                    aph ^= 1u;
                }
                if (++s == p.raw_stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp >= tc8f::EPI_WARP0) {
        // ---- draining warps, once per tile: lane quadrant warp % 4; of the two warps of a quadrant each takes every other 32
        // columns (CT = 1) or one of the halves (CT = 2)
        const int q = warp & 3, ch = (warp - tc8f::EPI_WARP0) >> 2;
        const int row_in_tile = q * 32 + lane, nw = CT == 2 && ch ? p.width - p.nw : p.nw, chunks = (nw + 31) / 32;
        const int c0 = CT == 1 ? ch : 0, step = CT == 1 ? 2 : 1;
        const uint32_t accfree = PAIR ? of_leader(bar_accfree) : su32(bar_accfree);
        uint32_t it = 0;
        for (int t = pair; t < p.items; t += pairs, it++) {
            const FoldItem f = p.item(t);
            const int in_tile = CT == 1 ? 0 : ch * p.nw, col0 = f.col_tile * p.width + in_tile, mat = p.mat_of(f.row_tile);
            const uint32_t ai = it % accs;
            const uint32_t lane_addr = tmem_base + (CT == 1 ? ai : (uint32_t)ch) * ACC2 + ((uint32_t)(q * 32) << 16);
            mbar_wait_nap(&bar_accfull[ai], (it / accs) & 1, fail, 128);
            tc_fence_after();
            int64_t row = (int64_t)(f.row_tile - (mat == 0 ? p.tile0[0] : (mat == 1 ? p.tile0[1] : p.tile0[2]))) * CTAS * ROWS + rank * ROWS + row_in_tile;
            int64_t M = mat == 0 ? p.M[0] : (mat == 1 ? p.M[1] : p.M[2]), ldy = mat == 0 ? p.ldy[0] : (mat == 1 ? p.ldy[1] : p.ldy[2]);
            float *o = (mat == 0 ? p.out[0] : (mat == 1 ? p.out[1] : p.out[2])) + (size_t)col0 * ldy + row;
            if (f.part >= 0) {
                ldy = CTAS * ROWS;
                o = p.part + ((size_t)f.part * p.width + in_tile) * ldy + rank * ROWS + row_in_tile;
            }
            if (c0 >= chunks) {
                if (lane == 0) arrive_at(accfree + ai * 8u);
                continue;
            }
            const int cols = min(nw, p.N - col0);
#pragma unroll 1
            for (int c = c0; c < chunks; c += step) {
                uint32_t v[32];
                tmem_ld32(lane_addr + (uint32_t)(c * 32), v);   // (past the tile's last column: other columns of the same 512, not used)
                tmem_ld_wait();
                if (c + step >= chunks) {   // everything of this warp's part is in registers: the accumulator may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_at(accfree + ai * 8u);
                }
                if (f.part >= 0 || row < M) {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (c * 32 + j < cols) o[(size_t)(c * 32 + j) * ldy] = __uint_as_float(v[j]);
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    all_sync<PAIR>();   // neither CTA of a pair ends while the other one may still arrive on its barriers or read its columns
    if (warp == 0) fold_tmem_dealloc<PAIR>(tmem_base, 512);
    if (tid == 0 && s_fail) report_error(p.err, 2);
}

// The parts of cut tiles, in the order of K. A thread: four rows of a column.
__global__ void __launch_bounds__(256) k_fold_sum(const __grid_constant__ Tc8fParams p) {
    griddep_launch();
    griddep_wait();
    const int quads = p.tile_rows / 4, r4 = (int)threadIdx.x % quads, c = (int)blockIdx.y * (256 / quads) + (int)threadIdx.x / quads;
    int row_tile, col_tile;
    p.at(p.whole + (int)blockIdx.x, row_tile, col_tile);
    const int64_t col = (int64_t)col_tile * p.width + c;
    if (c >= p.width || col >= p.N) return;
    const float4 *q = reinterpret_cast<const float4 *>(p.part) + ((size_t)blockIdx.x * p.cuts * p.width + c) * quads + r4;
    float4 v[tc8f::MAX_CUTS];
#pragma unroll
    for (int s = 0; s < tc8f::MAX_CUTS; s++) v[s] = s < p.cuts ? q[(size_t)s * p.width * quads] : make_float4(0.f, 0.f, 0.f, 0.f);
    float y[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
    for (int s = 1; s < tc8f::MAX_CUTS; s++) {
        if (s >= p.cuts) break;
        y[0] += v[s].x;
        y[1] += v[s].y;
        y[2] += v[s].z;
        y[3] += v[s].w;
    }
    const int mat = p.mat_of(row_tile);
    const int64_t row = (int64_t)(row_tile - (mat == 0 ? p.tile0[0] : (mat == 1 ? p.tile0[1] : p.tile0[2]))) * p.tile_rows + r4 * 4;
    const int64_t M = mat == 0 ? p.M[0] : (mat == 1 ? p.M[1] : p.M[2]), ldy = mat == 0 ? p.ldy[0] : (mat == 1 ? p.ldy[1] : p.ldy[2]);
    float *o = (mat == 0 ? p.out[0] : (mat == 1 ? p.out[1] : p.out[2])) + col * ldy + row;
    if (row + 4 <= M && ((uintptr_t)o & 15) == 0) {
        *reinterpret_cast<float4 *>(o) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (row + i < M) o[i] = y[i];
    }
}


cudaError_t tc_encode_2d(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows,
                         uint32_t elem_bytes);
cudaError_t tc_encode_2d_bytes(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows);
// Time of a unit (256 elements of K) of a tile in us, all SMs at work. Measured, Q4_K / Q8_0: pairs 1.02 / 0.90 at 64 columns, 1.10 / 1.00 at 128,
// 1.42 / 1.28 at 192, 1.72 / 1.70 at 256, in halves 2.20 / 2.10 at 352; single CTAs 1.15 at 80, 1.33 at 128, 2.1 at 256.
static double fold_unit_us(bool q4k, int ctas, int width) {
    if (ctas == 1) return (q4k ? 0.80 : 0.70) + 0.0048 * width;
    return q4k ? std::max(1.02, 0.50 + 0.0048 * width) : std::max(0.9, 0.35 + 0.005 * width);
}
// How a product is laid out over pairs of SMs or single ones. Of the even splits of the columns into tiles, and of the cuts of the K of those
// tiles that do not fill a wave, the one whose slowest SM has the least to do. A launch of pairs takes 2 to 3 us more than one of single CTAs
// (two sets of barriers to agree on, arrivals across the pair): they are for products of several units per SM.
FoldPlan mm_fold_plan(bool q4k, int n_mats, const int64_t *M, int64_t K, int64_t N, int sms) {
    FoldPlan f{};
    const int nst = (int)(K / 256);
    double best = 0;
    for (int form = 0; form < 3; form++) {   // single CTAs, pairs, pairs with two halves
        const int ctas = form == 0 ? 1 : 2, halves = form == 2 ? 2 : 1, workers = std::max(1, sms / ctas);
        const int widest = halves == 1 ? tc8f::NW : 2 * tc8f::HALF_NW, step = ctas == 1 ? 16 : 32;
        int64_t row_tiles = 0;
        for (int j = 0; j < n_mats; j++) row_tiles += (M[j] + 128 * ctas - 1) / (128 * ctas);
        for (int64_t ct = (N + widest - 1) / widest, last = ct + 12; ct <= (N + 63) / 64 && ct <= last; ct++) {
            const int width = (int)(((N + ct - 1) / ct + step - 1) / step * step), nw = halves == 1 ? width : (width / 2 + 31) / 32 * 32;
            if (nw == width && halves == 2) continue;
            const int64_t tiles = row_tiles * ((N + width - 1) / width), full = tiles / workers, rest = tiles % workers;
            const double unit = fold_unit_us(q4k, ctas, width), drain = halves == 1 && nw <= 192 ? 0.4 : 1.3;
            for (int cuts = 1; cuts <= tc8f::MAX_CUTS && (cuts == 1 || (rest > 0 && cuts <= nst)); cuts++) {
                const int64_t waves = (rest * cuts + workers - 1) / workers;
                const double t = (ctas == 2 ? 2.8 : 0.0) + (double)full * (nst * unit + drain) + (double)waves * ((nst + cuts - 1) / cuts * unit + drain) +
                                 (cuts > 1 ? 5.0 + (double)(rest * cuts) * width * (128 * ctas) * 8 / 6.5e6 : 0);
                if (f.width == 0 || t < best * 0.98) {
                    best = t;
                    f.ctas = ctas;
                    f.nw = nw;
                    f.width = width;
                    f.cuts = cuts;
                    f.whole = tiles - (cuts > 1 ? rest : 0);
                    f.partial_bytes = cuts > 1 ? (uint64_t)(rest * cuts) * width * (128 * ctas) * 4 : 0;
                }
            }
        }
    }
    return f;
}
cudaError_t launch_mm_fold_f16(bool q4k, int n_mats, const void *const *W, int64_t K, const int64_t *M, int64_t N, const void *blobs, float *const *y,
                               int64_t ldy, void *partial, int *err, cudaStream_t st, bool early) {
    if (n_mats < 1 || n_mats > tc8f::MAX_MATS) return cudaErrorInvalidValue;
    const int sms = current_sm_count();
    const FoldPlan plan = mm_fold_plan(q4k, n_mats, M, K, N, sms);
    if (plan.partial_bytes > 0 && partial == nullptr) return cudaErrorInvalidValue;
    Tc8fMaps maps;
    Tc8fParams p{};
    for (int j = 0; j < tc8f::MAX_MATS; j++) {
        if (j >= n_mats) {
            maps.m[j] = maps.m[0];
            p.tile0[j] = 1 << 30;
            continue;
        }
        const cudaError_t e = tc_encode_2d(&maps.m[j], W[j], (uint64_t)tlb_row_size(q4k ? TLB_TYPE_Q4_K : TLB_TYPE_Q8_0, K), (uint64_t)M[j], q4k ? 144 : tc8::ROW_CHUNK, tc8::ROWS, 2);
        if (e != cudaSuccess) return e;
        p.out[j] = y[j];
        p.M[j] = M[j];
        p.ldy[j] = n_mats > 1 ? M[j] : ldy;
        p.tile0[j] = p.row_tiles;
        p.row_tiles += (int)((M[j] + 128 * plan.ctas - 1) / (128 * plan.ctas));
    }
    p.act = (const uint8_t *)blobs;
    p.part = (float *)partial;
    p.N = (int)N;
    p.nst = (int)(K / 256);
    p.tile_rows = 128 * plan.ctas;
    p.nw = plan.nw;
    p.width = plan.width;
    p.col_tiles = (int)((N + p.width - 1) / p.width);
    const int tiles = p.row_tiles * p.col_tiles;
    p.whole = (int)plan.whole;
    p.cuts = plan.cuts;
    p.items = p.whole + (tiles - p.whole) * p.cuts;
    // raw stages: 128 rows x 256 elements (18 or 34 KB); what they leave goes to B
    const int raw_bytes = tc8::ROWS * (q4k ? 144 : tc8::ROW_CHUNK);
    const int shape = p.width > p.nw ? 2 : (p.nw > 128 && p.nw <= tc8f::HALF_NW ? 1 : 0);
    p.raw_stages = q4k ? 4 : (plan.ctas == 1 && p.nw > 128 ? 2 : 3);
    p.b_stages = std::min(tc8f::MAX_STAGES, (tc8f::SMEM - 1024 - p.raw_stages * raw_bytes) / (p.nw / plan.ctas * tc8f::KS * (shape == 0 ? 4 : 2)));
    if (p.b_stages < 2) return cudaErrorInvalidValue;
    p.groups = mm_fold_groups(N);
    if (plan.ctas == 2)
        for (int h = 0; h < 2; h++) {
            const int cols = h == 0 || p.width == p.nw ? p.nw : p.width - p.nw;
            const cudaError_t e = tc_encode_2d_bytes(&maps.act[h], blobs, 1024, (uint64_t)(K / tc8f::KS) * p.groups, 1024, (uint32_t)(cols / 16));
            if (e != cudaSuccess) return e;
        }
    p.err = err;
    const dim3 grid((unsigned)(plan.ctas * std::min(p.items, std::max(1, sms / plan.ctas))));
    auto go = [&](auto *k) { return launch_pdl_cluster(early, plan.ctas, k, grid, dim3(tc8f::THREADS), (size_t)tc8f::SMEM, st, maps, p); };
    cudaError_t e;
    if (shape == 2) e = q4k ? go(k_mm_q80_f16<true, 2, true>) : go(k_mm_q80_f16<false, 2, true>);
    else if (plan.ctas == 2 && shape == 1) e = q4k ? go(k_mm_q80_f16<true, 1, true>) : go(k_mm_q80_f16<false, 1, true>);
    else if (plan.ctas == 2) e = q4k ? go(k_mm_q80_f16<true, 0, true>) : go(k_mm_q80_f16<false, 0, true>);
    else if (shape == 1) e = q4k ? go(k_mm_q80_f16<true, 1, false>) : go(k_mm_q80_f16<false, 1, false>);
    else e = q4k ? go(k_mm_q80_f16<true, 0, false>) : go(k_mm_q80_f16<false, 0, false>);
    if (e != cudaSuccess || p.cuts == 1) return e;
    const int per = 1024 / p.tile_rows;   // columns of a CTA
    return launch_pdl(k_fold_sum, dim3((unsigned)(tiles - p.whole), (unsigned)((p.width + per - 1) / per)), dim3(256), 0, st, p);
}
cudaError_t launch_act_pack_fold(const ActLayout &a, const void *act, void *blobs, cudaStream_t st) {
    const char *ab = (const char *)act;
    k_act_pack_q80_f16<<<dim3((unsigned)(a.K / tc8f::KS), (unsigned)((a.N + tc8f::NW - 1) / tc8f::NW)), 256, 0, st>>>(
        (const int8_t *)(ab + a.qs_off), (const float *)(ab + a.d_off), a.K, (int)a.N, a.kind == ACT_Q8_K ? 256 : 32, (uint8_t *)blobs);
    return cudaGetLastError();
}

static size_t tc8w_smem() {   // Q4_0's raw stages are smaller
    return (size_t)tc8w::RAW_STAGES * tc8::RAW_BYTES + (size_t)tc8w::ACT_STAGES * tc8w::BLOB + (size_t)tc8w::A_RING * 8 * tc8::ROWS * sizeof(float) + 1024;
}

// ---------------------------------------------------------------- host side
// stages of raw weights: as many bytes in flight for either type
constexpr int tc8_raw_stages(bool q4) { return q4 ? 7 : 4; }
template <bool Q4, int NPAD, int AS>
static size_t tc8_smem() {
    return (size_t)tc8_raw_stages(Q4) * tc8::raw_bytes(Q4) + (size_t)AS * tc8_blob_bytes(NPAD) + (size_t)tc8::A_RING * 8 * tc8::ROWS * sizeof(float) + 1024;
}

template <bool Q4, int NPAD>
static void tc8_attr() {
    cudaFuncSetAttribute(k_mmq_tc_q80<Q4, NPAD, tc8_raw_stages(Q4), 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc8_smem<Q4, NPAD, 4>());
}
template <bool Q4, int NPAD>
static cudaError_t tc8_launch(bool early, dim3 grid, cudaStream_t st, const CUtensorMap &map, const Tc8Params &p) {
    return launch_pdl_if(early, k_mmq_tc_q80<Q4, NPAD, tc8_raw_stages(Q4), 4>, grid, dim3(tc8::THREADS), tc8_smem<Q4, NPAD, 4>(), st, map, p);
}

void mmq_tc8_configure() {
    tc8_attr<false, 16>();
    tc8_attr<false, 32>();
    tc8_attr<true, 16>();
    tc8_attr<true, 32>();
    cudaFuncSetAttribute(k_mmq_tc_q80_wide<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc8w_smem());
    cudaFuncSetAttribute(k_mmq_tc_q80_wide<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc8w_smem());
    auto fold = [](auto *k) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, tc8f::SMEM); };
    fold(k_mm_q80_f16<false, 0, false>);
    fold(k_mm_q80_f16<true, 0, false>);
    fold(k_mm_q80_f16<false, 1, false>);
    fold(k_mm_q80_f16<true, 1, false>);
    fold(k_mm_q80_f16<false, 0, true>);
    fold(k_mm_q80_f16<true, 0, true>);
    fold(k_mm_q80_f16<false, 1, true>);
    fold(k_mm_q80_f16<true, 1, true>);
    fold(k_mm_q80_f16<false, 2, true>);
    fold(k_mm_q80_f16<true, 2, true>);
}

bool mmq_tc8_supported(uint32_t type, int64_t K, int64_t M, int64_t N) {
    return (type == TLB_TYPE_Q8_0 || type == TLB_TYPE_Q4_0) && K % 256 == 0 && K >= 256 && M >= 1 && !few_column_faster(type, K, M, N) && N <= (int64_t)tc8w::NW * 65535;   // column tiles are grid.y
}

TcPlan mmq_tc8_plan(uint32_t type, int64_t K, int64_t M, int64_t N, int sm_count) {
    TcPlan t;
    t.nsb = (int)(K / 256);
    if (type == TLB_TYPE_Q8_0 && N > 64 && !getenv("TLB_NO_WIDE_TC") && !getenv("TLB_PROMPT_EXACT")) {
        // prompt-sized batches: scales folded into f16 operands (k_mm_q80_f16); tiles, pairs of CTAs and cuts of K by mm_fold_plan
        t.npad = tc8f::NW;
        t.n_split = 1;
        t.sb_per_split = t.nsb;
        t.streamk = 0;
        t.n_col_chunks = 1;
        t.blob_unit = 0;
        t.blob_bytes = mm_fold_bytes(K, N);
        t.partial_bytes = 0;
        return t;
    }
    // Q4_0 in 128-column tiles once they are a third of the SMs; fewer leave so much of the chip idle that passes of 32 columns with K cut
    // over the SMs are faster ([4096 x 14336] x 128, 32 tiles: 205 us against 100; x 256: 207 against 200). In a row of launches, tiles / passes (passes of eight
    // columns in k_gemv.cu): [4096 x 4096] x 200 60 / 64 (134), x 256 60 / 74 (173); [14336 x 4096] x 128 60 / 86 (212); [32000 x 2048] x 65 63 / 73 (142); rows of
    // 14336 weights cross later, a tile's K being one chain: [4096 x 14336] x 200 201 / 147 (377), x 400 202 / 273 (754).
    const bool wide = type == TLB_TYPE_Q8_0 || (M + tc8::ROWS - 1) / tc8::ROWS * ((N + tc8w::NW - 1) / tc8w::NW) >= sm_count / 3;
    if (N > 64 && wide && !getenv("TLB_NO_WIDE_TC")) {
        // the same batches with the reference's integer arithmetic (Q4_0, which has no other; TLB_PROMPT_EXACT=1): 128-column tiles, whole K per
        // CTA (k_mmq_tc_q80_wide), row tiles x column tiles fill the GPU
        t.npad = tc8w::NW;
        t.n_split = 1;
        t.sb_per_split = t.nsb;
        t.streamk = 0;
        t.n_col_chunks = (int)((N + t.npad - 1) / t.npad);
        t.blob_unit = (uint64_t)tc8_blob_bytes(t.npad);
        t.blob_bytes = (uint64_t)t.n_col_chunks * t.nsb * t.blob_unit;
        t.partial_bytes = 0;
        return t;
    }
    t.npad = N <= 16 ? 16 : 32;
    const int64_t tiles = (M + tc8::ROWS - 1) / tc8::ROWS;
    // same model as the Q4_K kernel, with the time per stage of Q8_0 (a stage of Q4_0 takes about 0.8 us instead of 1.0, so that it is cut a little more than it needs)
    int best = 1;
    double best_score = 1e30;
    for (int s = 1; s <= t.nsb && s <= 16; s++) {
        const int per = (t.nsb + s - 1) / s;
        if (s > 1 && per < 2) break;
        const int splits = (t.nsb + per - 1) / per;
        if (splits != s) continue;
        const int64_t waves = (tiles * splits + sm_count - 1) / sm_count;
        const double score = (double)waves * (2.3 + 1.0 * per) + (splits > 1 ? 2.0 : 0.0);
        if (score < best_score) { best_score = score; best = splits; }
    }
    t.n_split = best;
    t.sb_per_split = (t.nsb + best - 1) / best;
    t.streamk = 0;
    t.n_col_chunks = (int)((N + t.npad - 1) / t.npad);
    t.blob_unit = (uint64_t)tc8_blob_bytes(t.npad);
    t.blob_bytes = (uint64_t)t.n_col_chunks * t.nsb * t.blob_unit;
    t.partial_bytes = best > 1 ? (uint64_t)best * std::min<int64_t>(N, t.npad) * M * 4 : 0;
    return t;
}

cudaError_t launch_act_pack_tc8(const ActLayout &a, const void *act, int npad, void *blobs, cudaStream_t st) {
    const char *ab = (const char *)act;
    if (npad == tc8f::NW) {
        k_act_pack_q80_f16<<<dim3((unsigned)(a.K / tc8f::KS), (unsigned)((a.N + npad - 1) / npad)), 256, 0, st>>>(
            (const int8_t *)(ab + a.qs_off), (const float *)(ab + a.d_off), a.K, (int)a.N, a.kind == ACT_Q8_K ? 256 : 32, (uint8_t *)blobs);
        return cudaGetLastError();
    }
    return launch_pdl(k_act_pack_q80, dim3((unsigned)(a.K / 256), (unsigned)((a.N + npad - 1) / npad)), dim3(256), 0, st, (const int8_t *)(ab + a.qs_off), (const float *)(ab + a.d_off),
                      a.K, (int)a.N, npad, (uint8_t *)blobs);
}

cudaError_t tc_encode_2d(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows,
                         uint32_t elem_bytes);
void launch_mmq_reduce(const float *partial, float *y, int64_t total, int n_split, cudaStream_t st);

cudaError_t launch_mmq_tc8(uint32_t type, const TcPlan &t, const void *W, int64_t K, int64_t M, int64_t N, const void *blobs, float *y, int64_t ldy,
                           void *partial, int *err, cudaStream_t st, bool early) {
    CUtensorMap map;
    const bool q4 = type == TLB_TYPE_Q4_0;
    // described in 16-bit elements: a 272-byte box is 136 of them (the limit is 256 elements per dimension)
    cudaError_t e = tc_encode_2d(&map, W, (uint64_t)tlb_row_size(type, K), (uint64_t)M, (uint32_t)tc8::row_chunk(q4), tc8::ROWS, 2);
    if (e != cudaSuccess) return e;
    if (t.npad == tc8f::NW) return launch_mm_fold_f16(false, 1, &W, K, &M, N, blobs, &y, ldy, partial, err, st, early);
    if (t.npad == tc8w::NW) {
        Tc8Params p{};
        p.act = (const uint8_t *)blobs;
        p.out = y;
        p.M = M;
        p.N = (int)N;
        p.npad = t.npad;
        p.nst = p.st_per_split = t.nsb;
        p.n_split = 1;
        p.ldy = ldy;
        p.err = err;
        const dim3 grid((unsigned)((M + tc8::ROWS - 1) / tc8::ROWS), (unsigned)t.n_col_chunks);
        return q4 ? launch_pdl_if(early, k_mmq_tc_q80_wide<true>, grid, dim3(tc8w::THREADS), tc8w_smem(), st, map, p)
                  : launch_pdl_if(early, k_mmq_tc_q80_wide<false>, grid, dim3(tc8w::THREADS), tc8w_smem(), st, map, p);
    }
    dim3 grid((unsigned)((M + tc8::ROWS - 1) / tc8::ROWS), (unsigned)t.n_split);
    for (int c = 0; c < t.n_col_chunks; c++) {   // one launch per chunk of npad columns
        const int64_t n0 = (int64_t)c * t.npad, nc = std::min<int64_t>(t.npad, N - n0);
        Tc8Params p;
        p.act = (const uint8_t *)blobs + (size_t)c * t.nsb * t.blob_unit;
        p.M = M;
        p.N = (int)nc;
        p.npad = t.npad;
        p.nst = t.nsb;
        p.st_per_split = t.sb_per_split;
        p.n_split = t.n_split;
        p.err = err;
        float *yc = y + n0 * ldy;
        if (t.n_split > 1) {
            p.out = (float *)partial;
            p.ldy = M;
        } else {
            p.out = yc;
            p.ldy = ldy;
        }
        if (t.npad == 16) e = q4 ? tc8_launch<true, 16>(early, grid, st, map, p) : tc8_launch<false, 16>(early, grid, st, map, p);
        else e = q4 ? tc8_launch<true, 32>(early, grid, st, map, p) : tc8_launch<false, 32>(early, grid, st, map, p);
        if (e != cudaSuccess) return e;
        if (t.n_split > 1) {
            if (ldy != M) return cudaErrorInvalidValue;
            launch_mmq_reduce((const float *)partial, yc, nc * M, t.n_split, st);
            e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

}  // namespace tlb
