// MUL_MAT with Q6_K weights and a few f32 activation columns: decoded weights times the f32 values, the reference executor's
// own arithmetic (crates/kernels/src/cuda/native/mm.cu:16-42). For rows and columns that k_gemv_q6.cu does not take (gemv_q6_columns).
//
// What bounds it: decoding. A weight costs two integer operations (every other cycle each), a byte permutation that makes it an
// f32 and half an add; the multiply-adds work on pairs. One CTA per SM takes a contiguous range of rows. A producer thread copies tiles
// of whole rows through a ring with bulk copies; eight warps take units of two rows x 2048 weights off the tiles, a lane per 64
// weights (of one row's 2048, or of several short rows). The partial sums of a row go to shared memory and are added up at the end.
// Rows of 210-byte super-blocks need not start on 16 bytes: tiles do (up to eight rows).
// [32000 x 4096] x 1: 373 us with a warp per output element and a decoder call per weight; 47 us here.
#include <algorithm>
#include <cuda_fp16.h>
#include <numeric>

#include "kernels.h"
#include "pdl.cuh"
#include "tc_common.cuh"

namespace tlb {

namespace gemvf {

using namespace tc;   // mbarriers and copies

constexpr int WARPS = 8;                      // consumers
constexpr int THREADS = 32 * (WARPS + 1);     // and the producer
constexpr int MAX_STAGES = 16;
constexpr int PAD = 16;                       // word reads may run 2 bytes past a block
constexpr int OUT_BYTES = 8 * 1024;           // partial sums before they are added up
constexpr int RU = 2;                         // rows (or groups of short rows) of a unit

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory"); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t &>(d)) : "l"(reinterpret_cast<const uint64_t &>(a)), "l"(reinterpret_cast<const uint64_t &>(b)));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t &>(d))
        : "l"(reinterpret_cast<const uint64_t &>(a)), "l"(reinterpret_cast<const uint64_t &>(b)), "l"(reinterpret_cast<const uint64_t &>(c)));
    return d;
}

struct Params {
    const uint8_t *W;
    const float *x;         // column n at x + n * ldx
    float *y;               // column n at y + n * ldy
    int64_t M, ldx, ldy;
    int K, row_bytes, align_rows;
    int tile_rows, units_per_tile, its, group_rows, parts, reduce_lanes;   // group_rows: rows side by side in a unit's 32 lanes
    int sets, set_warps;    // sets of warps that take tiles in turn; the stage count is a multiple, so a stage always meets the same set
    int stages, stage_stride, epoch_tiles;
    int act_stride;         // bytes of a column in shared memory
    int n0;                 // first column of this pass
    int *err;
};

// ---------------------------------------------------------------- activations into shared memory
// Piece j (four values) of slot s (64 weights) lies at (j * slots + s) * 16: the 32 lanes of a unit read it without conflicts.
// Element h * 128 + run * 32 + is * 16 + i of a super-block belongs to its slot 2 h + is, piece run * 4 + i / 4.
template <int NC>
__device__ __forceinline__ void load_activations(const Params &p, uint8_t *act) {
    const int slots = p.K / 64;
#pragma unroll
    for (int n = 0; n < NC; n++) {
        const float *x = p.x + (int64_t)(p.n0 + n) * p.ldx;
#pragma unroll 4
        for (int k = threadIdx.x * 4; k < p.K; k += WARPS * 32 * 4) {
            const int e = k & 255, slot = (k >> 8) * 4 + (e >> 7) * 2 + ((e >> 4) & 1), piece = ((e >> 5) & 3) * 4 + ((e & 15) >> 2);
            *reinterpret_cast<float4 *>(act + (size_t)n * p.act_stride + ((size_t)piece * slots + slot) * 16) = *reinterpret_cast<const float4 *>(x + k);
        }
    }
    consumers_sync();
}

// ---------------------------------------------------------------- 64 weights of RU rows against the same activations
// A slot of a 210-byte super-block {ql[128], qh[64], i8 scales[16], f16 d} is the four 16-value runs that share 16 bytes of
// ql (two of them), of ql + 32 and of qh. Super-blocks start on 2-byte boundaries.
template <int RU, int NC>
__device__ __forceinline__ void dot_q6_K(const Params &p, const uint8_t *const (&row)[RU], int slot, const uint8_t *act, float (&f)[RU][NC]) {
    const int sb = slot >> 2, h = (slot >> 1) & 1, is = slot & 1, slots = p.K / 64;
#pragma unroll
    for (int r = 0; r < RU; r++)
#pragma unroll
        for (int n = 0; n < NC; n++) f[r][n] = 0.f;
    const uint8_t *blk[RU];
    uint32_t sc[RU];
#pragma unroll
    for (int r = 0; r < RU; r++) {
        blk[r] = row[r] + sb * 210;
        const uint8_t *s = blk[r] + 192 + h * 8 + is;   // scales of the runs: every other byte
        sc[r] = (uint32_t)s[0] | (uint32_t)s[2] << 8 | (uint32_t)s[4] << 16 | (uint32_t)s[6] << 24;
    }
    float2 acc[RU][NC][4];
#pragma unroll
    for (int r = 0; r < RU; r++)
#pragma unroll
        for (int n = 0; n < NC; n++)
#pragma unroll
            for (int u = 0; u < 4; u++) acc[r][n][u] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; i++) {   // four weights of every run at a time
        float4 x[NC][4];
#pragma unroll
        for (int n = 0; n < NC; n++)
#pragma unroll
            for (int u = 0; u < 4; u++) x[n][u] = *reinterpret_cast<const float4 *>(act + (size_t)n * p.act_stride + ((size_t)(u * 4 + i) * slots + slot) * 16);
#pragma unroll
        for (int r = 0; r < RU; r++) {
            auto word = [&](int off) {   // 2-byte aligned
                const unsigned short *s = reinterpret_cast<const unsigned short *>(blk[r] + off + 4 * i);
                return (uint32_t)s[0] | (uint32_t)s[1] << 16;
            };
            const uint32_t q0 = word(h * 64 + is * 16), q1 = word(h * 64 + 32 + is * 16), qh = word(128 + h * 32 + is * 16);
            const uint32_t c[4] = {(q0 & 0x0f0f0f0fu) | ((qh << 4) & 0x30303030u), (q1 & 0x0f0f0f0fu) | ((qh << 2) & 0x30303030u),
                                   ((q0 >> 4) & 0x0f0f0f0fu) | (qh & 0x30303030u), ((q1 >> 4) & 0x0f0f0f0fu) | ((qh >> 2) & 0x30303030u)};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                // byte b of a word behind 0x4b0000 is the f32 2^23 + b
                const float2 a = add2(make_float2(__uint_as_float(__byte_perm(c[u], 0x4b000000u, 0x7440)), __uint_as_float(__byte_perm(c[u], 0x4b000000u, 0x7441))), make_float2(-8388640.f, -8388640.f));
                const float2 b = add2(make_float2(__uint_as_float(__byte_perm(c[u], 0x4b000000u, 0x7442)), __uint_as_float(__byte_perm(c[u], 0x4b000000u, 0x7443))), make_float2(-8388640.f, -8388640.f));
#pragma unroll
                for (int n = 0; n < NC; n++) acc[r][n][u] = fma2(b, make_float2(x[n][u].z, x[n][u].w), fma2(a, make_float2(x[n][u].x, x[n][u].y), acc[r][n][u]));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RU; r++) {
        const float d = __half2float(*reinterpret_cast<const __half *>(blk[r] + 208));
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float ds = d * (float)(int8_t)((sc[r] >> (8 * u)) & 0xff);
#pragma unroll
            for (int n = 0; n < NC; n++) f[r][n] = fmaf(ds, acc[r][n][u].x + acc[r][n][u].y, f[r][n]);
        }
    }
}

// ---------------------------------------------------------------- the kernel
template <int NC>
__global__ void __launch_bounds__(THREADS, NC <= 2 ? 2 : 1) k_gemv_f32(const __grid_constant__ Params p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES];
    griddep_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t *act = smem + p.stages * p.stage_stride;
    float *part = reinterpret_cast<float *>(act + NC * p.act_stride);
    // this CTA's rows: a contiguous range
    const int64_t groups = (p.M + p.align_rows - 1) / p.align_rows;
    const int64_t r0 = groups * blockIdx.x / gridDim.x * p.align_rows, r1 = min(p.M, groups * (blockIdx.x + 1) / gridDim.x * p.align_rows);
    const int n_tiles = (int)((r1 - r0 + p.tile_rows - 1) / p.tile_rows);
    if (tid == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], (uint32_t)p.units_per_tile);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == WARPS) {
        // ---- producer: the weights do not depend on the kernel in front
        if (lane != 0) return;
        int s = 0, issued = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = 0; t < n_tiles; t++) {
            if (t >= p.stages && !(ok = mbar_wait_limit(&empty[s], ph ^ 1u))) break;
            const int64_t row0 = r0 + (int64_t)t * p.tile_rows;
            const int rows = (int)min((int64_t)p.tile_rows, r1 - row0);
            const uint32_t bytes = (uint32_t)(rows * p.row_bytes + 15) & ~15u;   // the last rows of a matrix may end between two 16-byte boundaries
            mbar_expect_tx(&full[s], bytes);
            bulk_g2s(smem + s * p.stage_stride, p.W + row0 * p.row_bytes, bytes, &full[s]);
            issued = t + 1;
            if (++s == p.stages) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (!ok) {
            // the consumers stopped releasing stages: record it, then wait (bounded) for the copies still in flight
            report_error(p.err, 1);
            for (int t = max(0, issued - p.stages); t < issued; t++) mbar_wait_limit(&full[t % p.stages], (uint32_t)((t / p.stages) & 1));
        }
        return;
    }

    // ---- consumers
    griddep_wait();
    load_activations<NC>(p, act);
    const int slots = p.K / 64;
    const int sub = p.its == 1 ? lane / slots : 0, slot_lane = p.its == 1 ? lane % slots : lane;
    // A set waits for every use of its stages, so a barrier is never more than one phase from the one it waits for.
    const int set = warp / p.set_warps, unit0 = warp % p.set_warps;
    int t = set < p.sets ? set : n_tiles, s = set;
    uint32_t ph = 0;
    bool ok = true;
    for (int e0 = 0; e0 < n_tiles; e0 += p.epoch_tiles) {
        const int e1 = min(n_tiles, e0 + p.epoch_tiles);
        for (; t < e1; t += p.sets) {
            if (ok && !mbar_wait_limit(&full[s], ph)) {
                if (lane == 0) report_error(p.err, 1);
                ok = false;   // this warp stops releasing stages; the producer's bounded wait ends the copies
            }
            const uint8_t *tile = smem + s * p.stage_stride;
            for (int u0 = unit0; u0 < p.units_per_tile; u0 += p.set_warps) {
                const int it = p.its == 1 ? 0 : u0 % p.its, grp = p.its == 1 ? u0 : u0 / p.its;
                const int slot = it * 32 + slot_lane, first = grp * RU * p.group_rows + sub;
                const bool live = slot < slots && sub < p.group_rows;   // a lane without weights computes those of slot 0
                // rows past a matrix's end hold what the stage held before; their sums are not used
                const uint8_t *rp[RU];
#pragma unroll
                for (int u = 0; u < RU; u++) rp[u] = tile + (live ? first + u * p.group_rows : 0) * p.row_bytes;
                float f[RU][NC];
                dot_q6_K<RU, NC>(p, rp, live ? slot : 0, act, f);
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(&empty[s]);
                float *o = part + ((size_t)(t - e0) * p.tile_rows + first) * p.parts * NC;
                if (p.reduce_lanes == 32 && NC != 3) {
                    // all values of the unit at once: half of them change lanes in every step until a lane group holds one
                    float v[RU * NC];
#pragma unroll
                    for (int i = 0; i < RU * NC; i++) v[i] = live ? f[i / NC][i % NC] : 0.f;
                    int bit = 16, which = 0;
#pragma unroll
                    for (int n = RU * NC; n > 1; n >>= 1, bit >>= 1) {
                        const bool up = (lane & bit) != 0;
                        which = which * 2 + up;
#pragma unroll
                        for (int i = 0; i < n / 2; i++) {
                            const float keep = up ? v[i + n / 2] : v[i], send = up ? v[i] : v[i + n / 2];
                            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                        }
                    }
#pragma unroll
                    for (; bit > 0; bit >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
                    if ((lane & (32 / (RU * NC) - 1)) == 0) o[((which / NC) * p.group_rows * p.parts + it) * NC + which % NC] = v[0];
                } else {
#pragma unroll
                    for (int u = 0; u < RU; u++)
#pragma unroll
                        for (int n = 0; n < NC; n++) {
                            float v = live ? f[u][n] : 0.f;
                            for (int x = p.reduce_lanes >> 1; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
                            if (live && slot_lane % p.reduce_lanes == 0) o[(u * p.group_rows * p.parts + (p.its == 1 ? slot_lane / p.reduce_lanes : it)) * NC + n] = v;
                        }
                }
            }
            s += p.sets;
            if (s >= p.stages) {
                s -= p.stages;
                ph ^= 1u;
            }
        }
        consumers_sync();
        // ---- the rows of this stretch: their parts in order
        const int n_rows = (e1 - e0) * p.tile_rows;
        for (int i = tid; i < n_rows * NC; i += WARPS * 32) {
            const int n = i / n_rows, ri = i % n_rows;
            const int64_t row = r0 + (int64_t)e0 * p.tile_rows + ri;
            if (row >= r1) continue;
            float v = 0.f;
            for (int x = 0; x < p.parts; x++) v += part[(ri * p.parts + x) * NC + n];
            p.y[(p.n0 + n) * p.ldy + row] = v;
        }
        if (e1 < n_tiles) consumers_sync();
    }
}

}  // namespace gemvf

// ---------------------------------------------------------------- host side
using gemvf::k_gemv_f32;

constexpr int GEMV_SMEM_ONE = 216 * 1024;   // one CTA per SM
constexpr int GEMV_SMEM_TWO = 110 * 1024;   // two

// fills the geometry of a launch of nc columns; false when a row does not fit
static bool gemv_geometry(gemvf::Params &p, uint32_t type, int64_t K, int nc, int64_t rows_per_cta, size_t &smem) {
    p.K = (int)K;
    p.row_bytes = (int)tlb_row_size(type, K);
    p.align_rows = 16 / std::gcd(16, p.row_bytes);
    const int slots = (int)(K / 64);
    p.its = (slots + 31) / 32;
    p.group_rows = p.its == 1 ? 32 / slots : 1;
    p.reduce_lanes = p.its > 1 ? 32 : ((slots & (slots - 1)) == 0 ? slots : 4);
    p.parts = p.its > 1 ? p.its : slots / p.reduce_lanes;
    p.act_stride = (int)(K * 4);
    // rows of a tile: whole units and 16-byte groups, 12 to 24 KB where rows allow; among those the count that leaves the
    // fewest warps without a unit
    const int ru = gemvf::RU, quantum = (int)std::lcm(ru * p.group_rows, p.align_rows);
    int rows = quantum;
    double best = -1;
    for (int r = quantum; r == quantum || ((int64_t)r * p.row_bytes <= 24 * 1024 && r <= rows_per_cta); r += quantum) {
        const int u = r / (ru * p.group_rows) * p.its;
        const double used = u >= gemvf::WARPS ? (double)u / ((u + gemvf::WARPS - 1) / gemvf::WARPS * gemvf::WARPS) : (double)(gemvf::WARPS / u * u) / gemvf::WARPS;
        const double score = used * std::min(1.0, (double)r * p.row_bytes / (12 * 1024));
        if (score > best + 1e-9) {
            best = score;
            rows = r;
        }
    }
    p.tile_rows = rows;
    p.units_per_tile = rows / (ru * p.group_rows) * p.its;
    p.set_warps = std::min(gemvf::WARPS, p.units_per_tile);
    p.sets = gemvf::WARPS / p.set_warps;
    p.stage_stride = (rows * p.row_bytes + 15 + gemvf::PAD + 127) / 128 * 128;
    p.epoch_tiles = std::max(1, gemvf::OUT_BYTES / (rows * p.parts * nc * 4));
    const int out = p.epoch_tiles * rows * p.parts * nc * 4;
    const int fixed = nc * p.act_stride + out;
    const int budget = nc <= 2 && fixed + 3 * p.stage_stride <= GEMV_SMEM_TWO ? GEMV_SMEM_TWO : GEMV_SMEM_ONE;
    p.stages = std::min(gemvf::MAX_STAGES, (budget - fixed) / p.stage_stride);
    while (p.sets > 1 && p.stages < 2 * p.sets && p.stages % p.sets) p.sets--;
    p.stages -= p.stages % p.sets;
    smem = (size_t)std::max(p.stages, 0) * p.stage_stride + fixed;
    return p.stages >= 2;
}

bool gemv_f32_supported(uint32_t type, int64_t K, int64_t M, int64_t N) {
    if (type != TLB_TYPE_Q6_K || K % 256 != 0 || K < 256 || K > (1 << 20) || M < 1 || N < 1) return false;
    gemvf::Params p{};
    size_t smem;
    return gemv_geometry(p, type, K, 1, 1 << 20, smem);
}

void gemv_f32_configure() {
    gemv_q6_configure();
    auto set = [](auto *k) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMV_SMEM_ONE); };
    set(k_gemv_f32<1>);
    set(k_gemv_f32<2>);
    set(k_gemv_f32<3>);
    set(k_gemv_f32<4>);
}

cudaError_t launch_gemv_f32(const GemvArgs &g, int sm_count, int *err, cudaStream_t st) {
    if (g.n_mats != 1 || g.glu || g.act.mode != RQ_PLAIN) return cudaErrorInvalidValue;
    if (g.N <= gemv_q6_columns(g.K, g.M[0])) return launch_gemv_q6(g, sm_count, err, st);
    gemvf::Params p{};
    p.W = (const uint8_t *)g.W[0];
    p.x = g.act.a;
    p.ldx = g.act.lda;
    p.y = g.y[0];
    p.M = g.M[0];
    p.ldy = g.ldy[0];
    p.err = err;
    for (int64_t n0 = 0; n0 < g.N;) {
        size_t smem = 0;
        int nc = (int)std::min<int64_t>(4, g.N - n0);
        while (nc > 1 && !gemv_geometry(p, g.type, g.K, nc, g.M[0] / sm_count + 1, smem)) nc--;
        if (!gemv_geometry(p, g.type, g.K, nc, g.M[0] / sm_count + 1, smem)) return cudaErrorInvalidValue;
        p.n0 = (int)n0;
        const dim3 grid((unsigned)sm_count), block(gemvf::THREADS);
        cudaError_t e;
        switch (nc) {
            case 1: e = launch_pdl_if(g.early, k_gemv_f32<1>, grid, block, smem, st, p); break;
            case 2: e = launch_pdl_if(g.early, k_gemv_f32<2>, grid, block, smem, st, p); break;
            case 3: e = launch_pdl_if(g.early, k_gemv_f32<3>, grid, block, smem, st, p); break;
            default: e = launch_pdl_if(g.early, k_gemv_f32<4>, grid, block, smem, st, p); break;
        }
        if (e != cudaSuccess) return e;
        n0 += nc;
    }
    return cudaSuccess;
}

}  // namespace tlb
