// MUL_MAT with Q6_K weights and a few f32 activation columns on the integer matrix instruction.
//
// The reference multiplies decoded weights with the f32 activations (crates/kernels/src/cuda/native/mm.cu:16-42). Decoding a weight to f32 costs 13 issue
// slots per 32 weights (k_gemv_f32.cu), so here the activations go to the weights' side: each 256 of them become fixed-point numbers of 61 bits
// and a sign at the scale of their largest, as eight signed base-256 digits. That holds every f32 down to 2^-37 of the largest to its last bit (a
// super-block with a smaller one, or with one that is not finite, is summed value by value). Four digits held what is above 2^-30 of the largest only, and a
// large activation over a weight of zero took the others' bits: 4.5e-6 of a row's norm beside 1e4, 3.7e-2 beside 1e8. The products of digits
// and 6-bit codes, their sums over a 16-weight group and the sums over a super-block with the groups' 8-bit scales are whole numbers below 2^31,
// exact; only the sums of super-blocks are f32. Relative error against f64, k_gemv_f32.cu and here, one column: 1.0e-7 / 7.5e-8 at [300 x 4096], 1.2e-7 / 9.0e-8 at
// [300 x 14336], 1.1e-7 / 8.9e-8 at [20000 x 14336]; activations over five decades 7.4e-8 / 5.9e-8, 9.9e-8 / 8.5e-8, 1.1e-7 / 9.8e-8.
//
// m16n8k16 takes a group of 16 rows against the eight digits of a column. A code costs one integer operation: bytes of 4 * (q - 32) are put together in place
// (shift, mask and merge on words of four). What bounds it is a unit's chain of shared-memory loads, matrix instructions and multiply-adds with two
// or four warps per scheduler. One column, cold, k_gemv_f32.cu and here: [32000 x 4096] 52.5 -> 39.0 us (the stream needs 17), [4096 x 4096] 17.5 -> 16.4,
// [4096 x 14336] 36.2 -> 32.3, [30000 x 512] 18.2 -> 15.0, [20000 x 1024] 19.8 -> 16.7 (four digits, m16n8k32 over two groups: 35.5, 15.6, 28.0, 14.8, 15.8).
//
// Layout of the work as in k_gemv.cu: a CTA (two per SM) takes a contiguous range of 16-row groups, a producer thread copies tiles through a
// ring, eight warps take a super-block of 16 rows each. Rows of whole 8-super-block segments are copied by 2-D boxes of 16 x 1680
// bytes (16 bytes past a multiple of 128: eight rows on different banks), shorter rows as 16 rows in one piece.
#include <algorithm>
#include <cstdlib>
#include <cuda_fp16.h>

#include "dequant.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "tc_common.cuh"

namespace tlb {

cudaError_t tc_encode_2d_bytes(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_bytes, uint32_t box_rows);

namespace gemvq6 {

using namespace tc;   // mbarriers and copies

constexpr int WARPS = 8;
constexpr int THREADS = 32 * (WARPS + 1);
constexpr int MAX_STAGES = 12;
constexpr int PAD = 16;           // word reads may run past a block
constexpr int epoch(int nc) { return nc == 1 ? 16 : 8; }   // row groups (per group of a tile) between two additions of the parts
constexpr int BLOCK = 210;
constexpr int DIGITS = 8;

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory"); }

struct Params {
    const uint8_t *W;
    const float *x;         // column n at x + n * ldx
    float *y;               // column n at y + n * ldy
    int64_t M, ldx, ldy;
    int units, row_bytes;             // super-blocks and bytes of a row
    int boxes;                        // 1: 2-D boxes of eight super-blocks; 0: whole rows
    int segs, groups;                 // tiles of a row group; row groups of a tile (rows of less than eight super-blocks)
    int row_stride, stage_stride, stages;
    int plane, act_bytes;             // bytes of a digit's plane of a column; of all columns and their scales
    int *err;
};

// D = A B with 8-bit operands
__device__ __forceinline__ void imma16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3},{%4,%5},{%6},{%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}

// a byte of w as a signed number; sel: its index in every nibble, the upper three with the bit that replicates its sign
__device__ __forceinline__ int signed_byte(uint32_t w, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "r"(sel));
    return (int)r;
}

// ---------------------------------------------------------------- activations as digits
__device__ __forceinline__ void put_digits(int z, int e, uint32_t (&q)[4][2]) {
#pragma unroll
    for (int j = 3; j >= 0; j--) {
        const int digit = (int)(int8_t)(z & 0xff);
        q[j][e >> 2] |= (uint32_t)(digit & 0xff) << (8 * (e & 3));
        z = (z - digit) >> 8;
    }
}

// Plane j of a column: its j-th digit (the highest first) of every value in order. A block that the digits do not hold to the last bit (values that
// are not finite, or that have bits 2^61 below the largest) has the scale NaN: its sums are taken value by value.
template <int NC>
__device__ __forceinline__ void load_digits(const Params &p, uint8_t *act) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *const scales = reinterpret_cast<float *>(act + NC * DIGITS * p.plane);   // [column][super-block]
#pragma unroll 1
    for (int i = warp; i < NC * p.units; i += WARPS) {
        const int n = NC == 1 ? 0 : i / p.units, sb = NC == 1 ? i : i % p.units;
        const float *x = p.x + (int64_t)n * p.ldx + sb * 256 + lane * 8;
        const float4 u = *reinterpret_cast<const float4 *>(x), w = *reinterpret_cast<const float4 *>(x + 4);
        const float v[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
        uint32_t top = 0;   // magnitudes order like their bits; NaNs lie above infinity
#pragma unroll
        for (int e = 0; e < 8; e++) top = max(top, __float_as_uint(v[e]) & 0x7fffffffu);
        top = __reduce_max_sync(0xffffffffu, top);
        uint32_t hi[4][2] = {}, lo[4][2] = {};
        float scale = 0.f;
        if (top >= 0x7f800000u) {
            scale = __uint_as_float(0x7fc00000u);
        } else if (top != 0) {
            // 2^(ex + 1) is above every value; scaled to below 2^30. In two steps: either factor alone may be outside f32
            const int ex = max((int)(top >> 23) - 127, -120);
            const int up = 29 - ex, a = min(up, 127), b = up - a;   // 0 <= b <= 22; up >= -98
            const float fa = __uint_as_float((uint32_t)(a + 127) << 23), fb = __uint_as_float((uint32_t)(b + 127) << 23);
            bool lost = false;
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const float f = v[e] * fa * fb;
                const int z = __float2int_rn(f);
                const float rest = (f - (float)z) * 2147483648.f;   // exact: f has no bits below one from 2^23 on, and z is at most 2^24 below that
                const int y = __float2int_rn(rest);
                lost |= (float)y != rest || (f == 0.f && v[e] != 0.f);
                put_digits(z, e, hi);
                put_digits(y, e, lo);
            }
            // 2^-up: down to 2^-149, below 2^-126 as a subnormal
            scale = up <= 126 ? __uint_as_float((uint32_t)(127 - up) << 23) : __uint_as_float(1u << (149 - up));
            if (__any_sync(0xffffffffu, lost)) scale = __uint_as_float(0x7fc00000u);
        }
        uint8_t *o = act + n * DIGITS * p.plane + sb * 256 + lane * 8;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            *reinterpret_cast<uint2 *>(o + j * p.plane) = make_uint2(hi[j][0], hi[j][1]);
            *reinterpret_cast<uint2 *>(o + (4 + j) * p.plane) = make_uint2(lo[j][0], lo[j][1]);
        }
        if (lane == 0) scales[n * p.units + sb] = scale;
    }
    consumers_sync();
}

// ---------------------------------------------------------------- a super-block of 16 rows
// {ql[128], qh[64], i8 scales[16], f16 d}; starts on 2-byte boundaries. Lane (g, t) brings words 4t of rows g and g + 8 and of digit g of
// each column, and gets sums of those rows with digits 2t and 2t + 1. b: this lane's word of group 0 of this super-block, of column 0.
// f[2 * n], f[2 * n + 1]: rows g and g + 8 with column n, the part of this lane's two digits. x: the columns' values of this super-block.
template <int NC>
__device__ __forceinline__ void unit_q6_K(const uint8_t *r0, const uint8_t *r1, const uint8_t *b, int col_planes, const float *scale, int col_scales, const float *x, int64_t ldx,
                                          float (&f)[2 * NC]) {
    const int lane = threadIdx.x & 31, t = lane & 3;
    const uint32_t *w[2] = {reinterpret_cast<const uint32_t *>((uintptr_t)r0 & ~(uintptr_t)3), reinterpret_cast<const uint32_t *>((uintptr_t)r1 & ~(uintptr_t)3)};
    const uint32_t sh[2] = {(uint32_t)((uintptr_t)r0 & 2) * 8, (uint32_t)((uintptr_t)r1 & 2) * 8};
    auto word = [&](int r, int at) { return __funnelshift_r(w[r][at], w[r][at + 1], sh[r]); };   // word `at` of the block
    int acc[NC][4] = {};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t sc[2][2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            sc[r][0] = word(r, 48 + h * 2);
            sc[r][1] = word(r, 49 + h * 2);
        }
#pragma unroll
        for (int is = 0; is < 2; is++) {
            uint32_t c[2][4];   // four codes of each run of 32: 4 * (q - 32) as signed bytes
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t q0 = word(r, h * 16 + is * 4 + t), q1 = word(r, h * 16 + 8 + is * 4 + t), qh = word(r, 32 + h * 8 + is * 4 + t);
                c[r][0] = ((q0 << 2) & 0x3c3c3c3cu) | (((qh << 6) & 0xc0c0c0c0u) ^ 0x80808080u);
                c[r][1] = ((q1 << 2) & 0x3c3c3c3cu) | (((qh << 4) & 0xc0c0c0c0u) ^ 0x80808080u);
                c[r][2] = ((q0 >> 2) & 0x3c3c3c3cu) | (((qh << 2) & 0xc0c0c0c0u) ^ 0x80808080u);
                c[r][3] = ((q1 >> 2) & 0x3c3c3c3cu) | ((qh & 0xc0c0c0c0u) ^ 0x80808080u);
            }
            const uint8_t *bg = b + h * 128 + is * 16;
#pragma unroll
            for (int run = 0; run < 4; run++) {
                const uint32_t sel = 0x8880u + 0x1111u * (uint32_t)(2 * (run & 1) + is);   // the group's scale byte with its sign
                const int s0 = signed_byte(sc[0][run >> 1], sel), s1 = signed_byte(sc[1][run >> 1], sel);
#pragma unroll
                for (int n = 0; n < NC; n++) {
                    int d[4];
                    imma16(d, c[0][run], c[1][run], *reinterpret_cast<const uint32_t *>(bg + n * col_planes + run * 32));
                    acc[n][0] += s0 * d[0];
                    acc[n][1] += s0 * d[1];
                    acc[n][2] += s1 * d[2];
                    acc[n][3] += s1 * d[3];
                }
            }
        }
    }
    const float d0 = __half2float(*reinterpret_cast<const __half *>(r0 + 208)), d1 = __half2float(*reinterpret_cast<const __half *>(r1 + 208));
    // of digits 2t and 2t + 1: 2^16, 1, 2^-15, 2^-31; the codes are 4 * (q - 32)
    const float weight = __uint_as_float((t == 0 ? 141u : t == 1 ? 125u : t == 2 ? 110u : 94u) << 23);
#pragma unroll
    for (int n = 0; n < NC; n++) {
        const float xs = scale[n * col_scales];   // (multiplied last: it may be subnormal)
        if (xs != xs || !isfinite(d0) || !isfinite(d1)) {   // value by value, a quarter of the super-block per lane
            f[2 * n] += q6_K_slot_sum(r0, x + n * ldx, t);
            f[2 * n + 1] += q6_K_slot_sum(r1, x + n * ldx, t);
            continue;
        }
        f[2 * n] = fmaf(d0 * fmaf((float)acc[n][0], 256.f, (float)acc[n][1]) * weight, xs, f[2 * n]);
        f[2 * n + 1] = fmaf(d1 * fmaf((float)acc[n][2], 256.f, (float)acc[n][3]) * weight, xs, f[2 * n + 1]);
    }
    __syncwarp();
}

// ---------------------------------------------------------------- the kernel
// NC: columns
template <int NC>
__global__ void __launch_bounds__(THREADS, 2) k_gemv_q6(const __grid_constant__ CUtensorMap map, const __grid_constant__ Params p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES];
    griddep_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t *act = smem + p.stages * p.stage_stride;
    float *part = reinterpret_cast<float *>(act + p.act_bytes);
    // this CTA's row groups of 16 (tiles of p.groups of them): a contiguous range
    const int64_t tiles_all = (p.M + 16 * p.groups - 1) / (16 * p.groups);
    const int64_t t0 = tiles_all * blockIdx.x / gridDim.x;
    const int tiles = (int)(tiles_all * (blockIdx.x + 1) / gridDim.x - t0);
    if (tid == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], WARPS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp == WARPS) {
        // ---- producer: the weights do not depend on the kernel in front
        if (lane != 0) return;
        int s = 0, turn = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int t = 0; t < tiles && ok; t++) {
            const int64_t row0 = (t0 + t) * 16 * p.groups;
            for (int seg = 0; seg < p.segs && ok; seg++, turn++) {
                if (turn >= p.stages && !(ok = mbar_wait_limit(&empty[s], ph ^ 1u))) break;
                if (p.boxes) {
                    mbar_expect_tx(&full[s], (uint32_t)(16 * p.row_stride));
                    tma_2d(smem + s * p.stage_stride, &map, seg * (8 * BLOCK / 8), (int)row0, &full[s]);   // x in 8-byte elements; rows past the matrix read as zero
                } else {
                    const int64_t rows = min((int64_t)16 * p.groups, p.M - row0);
                    const uint32_t bytes = (uint32_t)(rows * p.row_bytes + 15) & ~15u;   // the last rows of a matrix may end between two 16-byte boundaries
                    mbar_expect_tx(&full[s], bytes);
                    bulk_g2s(smem + s * p.stage_stride, p.W + row0 * p.row_bytes, bytes, &full[s]);
                }
                if (++s == p.stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        if (!ok) {
            // the consumers stopped releasing stages: record it, then wait (bounded) for the copies still in flight
            report_error(p.err, 1);
            for (int st = 0; st < p.stages; st++)
                if (mbar_wait_limit(&full[st], 0, 1u << 12)) mbar_wait_limit(&full[st], 1, 1u << 12);   // one of the two phases has passed
        }
        return;
    }

    // ---- consumers
    griddep_wait();
    load_digits<NC>(p, act);
    const float *const scales = reinterpret_cast<const float *>(act + NC * DIGITS * p.plane);
    const int g = lane >> 2, t4 = lane & 3;
    const int per_group = p.groups > 1 ? p.units : WARPS;   // warps of a row group
    const int gr = warp / per_group, u0 = warp % per_group;
    const bool works = gr < p.groups;
    const uint8_t *const b0 = act + g * p.plane + t4 * 4;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int e0 = 0; e0 < tiles; e0 += epoch(NC)) {
        const int e1 = min(tiles, e0 + epoch(NC));
        for (int t = e0; t < e1; t++) {
            float f[2 * NC] = {};
            for (int seg = 0; seg < p.segs; seg++) {
                if (ok && !mbar_wait_limit(&full[s], ph)) {
                    if (lane == 0) report_error(p.err, 1);
                    ok = false;   // this warp stops releasing stages; the producer's bounded wait ends the copies
                }
                // rows past a matrix's end hold what the stage held before; their sums are not used
                const uint8_t *tile = smem + s * p.stage_stride + (gr * 16 + g) * p.row_stride;
                if (works)
                    for (int u = u0; u < (p.boxes ? 8 : p.units); u += per_group) {
                        const int sb = seg * 8 + u;
                        unit_q6_K<NC>(tile + u * BLOCK, tile + 8 * p.row_stride + u * BLOCK, b0 + sb * 256, DIGITS * p.plane, scales + sb, p.units, p.x + sb * 256, p.ldx, f);
                    }
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(&empty[s]);
                if (++s == p.stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // the lanes of a row: its digits
#pragma unroll
            for (int i = 0; i < 2 * NC; i++) {
                f[i] += __shfl_xor_sync(0xffffffffu, f[i], 2);
                f[i] += __shfl_xor_sync(0xffffffffu, f[i], 1);
            }
            // part [tile of the epoch][warp][column][row]
            float *o = part + ((t - e0) * WARPS + warp) * NC * 16;
            if (works && t4 == 0) {
#pragma unroll
                for (int n = 0; n < NC; n++) {
                    o[n * 16 + g] = f[2 * n];
                    o[n * 16 + g + 8] = f[2 * n + 1];
                }
            }
        }
        consumers_sync();
        // ---- the rows of this stretch: their parts in order
        const int rows = (e1 - e0) * p.groups * 16;
        for (int i = tid; i < rows * NC; i += WARPS * 32) {
            const int n = NC == 1 ? 0 : i / rows, ri = NC == 1 ? i : i % rows, grp = ri >> 4;
            const int64_t row = (t0 + e0) * 16 * p.groups + ri;
            if (row >= p.M) continue;
            const float *q = part + ((grp / p.groups * WARPS + grp % p.groups * per_group) * NC + n) * 16 + (ri & 15);
            float v = 0.f;
            for (int k = 0; k < per_group; k++) v += q[k * NC * 16];
            p.y[n * p.ldy + row] = v;
        }
        if (e1 < tiles) consumers_sync();
    }
}

}  // namespace gemvq6

// ---------------------------------------------------------------- host side
constexpr int Q6_SMEM_ONE = 220 * 1024, Q6_SMEM_TWO = 110 * 1024;   // one CTA per SM, two

// fills the geometry of a launch of nc columns; false when it does not fit. Two CTAs per SM with two stages each beat one with six (39.0 and 43.5 us
// for [32000 x 4096] x 1).
static bool gemv_q6_geometry(gemvq6::Params &p, int64_t K, int nc, size_t &smem, int &per_sm) {
    p.units = (int)(K / 256);
    p.row_bytes = p.units * gemvq6::BLOCK;
    p.boxes = p.units % 8 == 0;
    p.segs = p.boxes ? p.units / 8 : 1;
    p.groups = p.units < gemvq6::WARPS ? gemvq6::WARPS / p.units : 1;
    p.row_stride = p.boxes ? 8 * gemvq6::BLOCK : p.row_bytes;
    p.stage_stride = (16 * p.groups * p.row_stride + 15 + gemvq6::PAD + 127) / 128 * 128;
    p.plane = (int)K + 16;   // the planes of a lane's word on different banks
    p.act_bytes = (nc * gemvq6::DIGITS * p.plane + nc * p.units * 4 + 127) / 128 * 128;
    const int fixed = p.act_bytes + gemvq6::epoch(nc) * gemvq6::WARPS * nc * 64;
    per_sm = fixed + 2 * p.stage_stride <= Q6_SMEM_TWO ? 2 : 1;
    p.stages = std::min(gemvq6::MAX_STAGES, ((per_sm == 2 ? Q6_SMEM_TWO : Q6_SMEM_ONE) - fixed) / p.stage_stride);
    smem = (size_t)std::max(p.stages, 0) * p.stage_stride + fixed;
    return p.stages >= 2;
}
// One column, and as many as make 32 KB of digits. us of a launch, cold, this kernel / k_gemv_f32.cu: two columns of [30000 x 512] 16.6 / 21.1, [20000 x 1024]
// 18.0 / 23.8, [1500 x 2048] 14.5 / 13.4, [3000 x 2816] 17.7 / 17.4, [4096 x 4096] 21.5 / 18.1, [4096 x 14336] 55.5 / 39.2; four of [30000 x 512] 18.7 /
// 27.8, [20000 x 1024] 23.2 / 32.5, [1500 x 2048] 16.2 / 15.8, [4096 x 4096] 27.8 / 22.4. A CTA takes 16 rows at least, so fewer than 148 of these leave
// SMs idle, and k_gemv_f32.cu spreads them further: one column in a row of launches [1024 x 4096] 8.8 / 5.2, [1500 x 2048] 5.9 / 4.8 (two: 7.9 / 5.5),
// [4096 x 4096] 9.0 / 9.3.
// (TLB_Q6_DIGITS: small matrices here and in k_mm_q6.cu all the same, for tests of their edges)
constexpr int64_t Q6_ROWS = 16 * 148;
int gemv_q6_columns(int64_t K, int64_t M) {
    gemvq6::Params p{};
    size_t smem;
    int per_sm, nc = 0;
    if (!tc_available() || (M < Q6_ROWS && !getenv("TLB_Q6_DIGITS")) || K % 256 != 0 || K < 256 || K > (1 << 20)) return 0;
    while (nc < 4 && (nc == 0 || (nc + 1) * K <= 4096) && gemv_q6_geometry(p, K, nc + 1, smem, per_sm)) nc++;
    return nc;
}
void gemv_q6_configure() {
    auto set = [](auto *k) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Q6_SMEM_ONE); };
    set(gemvq6::k_gemv_q6<1>);
    set(gemvq6::k_gemv_q6<2>);
    set(gemvq6::k_gemv_q6<3>);
    set(gemvq6::k_gemv_q6<4>);
}
cudaError_t launch_gemv_q6(const GemvArgs &g, int sm_count, int *err, cudaStream_t st) {
    gemvq6::Params p{};
    p.W = (const uint8_t *)g.W[0];
    p.x = g.act.a;
    p.ldx = g.act.lda;
    p.y = g.y[0];
    p.M = g.M[0];
    p.ldy = g.ldy[0];
    p.err = err;
    CUtensorMap map{};
    size_t smem = 0;
    int per_sm = 1;
    if (g.N < 1 || g.N > gemv_q6_columns(g.K, g.M[0]) || !gemv_q6_geometry(p, g.K, (int)g.N, smem, per_sm)) return cudaErrorInvalidValue;
    if (p.boxes) {
        const cudaError_t e = tc_encode_2d_bytes(&map, g.W[0], (uint64_t)p.row_bytes, (uint64_t)p.M, (uint32_t)p.row_stride, 16);
        if (e != cudaSuccess) return e;
    }
    const dim3 grid((unsigned)(per_sm * sm_count)), block(gemvq6::THREADS);
    switch (g.N) {
        case 1: return launch_pdl_if(g.early, gemvq6::k_gemv_q6<1>, grid, block, smem, st, map, p);
        case 2: return launch_pdl_if(g.early, gemvq6::k_gemv_q6<2>, grid, block, smem, st, map, p);
        case 3: return launch_pdl_if(g.early, gemvq6::k_gemv_q6<3>, grid, block, smem, st, map, p);
        default: return launch_pdl_if(g.early, gemvq6::k_gemv_q6<4>, grid, block, smem, st, map, p);
    }
}

}  // namespace tlb
