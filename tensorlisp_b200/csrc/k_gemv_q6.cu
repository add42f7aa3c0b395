// MUL_MAT with Q6_K weights and a few f32 activation columns on the integer matrix instruction.
//
// The reference multiplies decoded weights with the f32 activations (crates/kernels/src/cuda/native/mm.cu:16-42). Decoding a weight to f32
// costs 13 issue slots per 32 weights (k_gemv_f32.cu), so here the activations go to
// the weights' side: each 256 of them become 32-bit fixed-point numbers at the scale of their largest, split into four signed base-256
// digits. The products of digits and 6-bit codes, their sums over a 16-weight group and the sums over a super-block with the groups' 8-bit
// scales are whole numbers below 2^31, exact; only the sums of super-blocks are f32. A value is off by 2^-30 of the largest of its 256 at most,
// which is less than the f32 rounding of any sum that has the largest in it. Relative error against f64, here and there: 5.4e-8 / 7.9e-8 at 256
// weights a row, 8.3e-8 / 1.0e-7 at 4096, 1.0e-7 / 1.2e-7 at 14336; activations that spread over five decades 7.1e-8 / 1.0e-7 at 4096.
//
// Measured there and here, cold: [32000 x 4096] x 1 52.5 -> 36.3 us (a call with its copies 82 -> 54; the stream needs 17), x 4 74 -> 50, x 64
// 1003 -> 661; [4096 x 14336] x 1 35.7 -> 27.8; [30000 x 512] x 64 293 -> 147. What is left is a unit's chain of shared-memory loads,
// matrix instructions and multiply-adds with two or four warps per scheduler.
//
// m16n8k32 takes two groups of 16 rows against eight columns: one activation column as four digits beside four zero columns of the other
// group each. Two columns and more: m16n8k16, a pair of columns as eight. A code costs one integer operation: bytes of 4 * (q - 32)
// are put together in place (shift, mask and merge on words of four).
//
// Layout of the work as in k_gemv.cu: a CTA (two per SM) takes a contiguous range of 16-row groups, a producer thread copies tiles through a
// ring, eight warps take a super-block of 16 rows each. Rows of whole 8-super-block segments are copied by 2-D boxes of 16 x 1680
// bytes (16 bytes past a multiple of 128: eight rows on different banks), shorter rows as 16 rows in one piece.
#include <algorithm>
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
constexpr int EPOCH = 16;         // row groups (per group of a tile) between two additions of the parts
constexpr int BLOCK = 210;

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory"); }

struct Params {
    const uint8_t *W;
    const float *x;         // column n at x + n * ldx
    float *y;
    int64_t M, ldx, ldy;
    int units, row_bytes;             // super-blocks and bytes of a row
    int boxes;                        // 1: 2-D boxes of eight super-blocks; 0: whole rows
    int segs, groups;                 // tiles of a row group; row groups of a tile (rows of less than eight super-blocks)
    int row_stride, stage_stride, stages;
    int plane, act_bytes;             // bytes of a digit's plane of a column; of all columns and their scales
    int n0;
    int *err;
};

// D += A B with 8-bit operands
__device__ __forceinline__ void imma32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
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
// Plane j of a column: its j-th digit (the highest first) of every value in order. A block whose values are not all finite has the scale NaN:
// its sums are taken value by value.
template <int NC>
__device__ __forceinline__ void load_digits(const Params &p, uint8_t *act) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float *const scales = reinterpret_cast<float *>(act + NC * 4 * p.plane);   // [column][super-block]
#pragma unroll 1
    for (int i = warp; i < NC * p.units; i += WARPS) {
        const int n = NC == 1 ? 0 : i / p.units, sb = NC == 1 ? i : i % p.units;
        const float *x = p.x + (int64_t)(p.n0 + n) * p.ldx + sb * 256 + lane * 8;
        const float4 u = *reinterpret_cast<const float4 *>(x), w = *reinterpret_cast<const float4 *>(x + 4);
        float v[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
        uint32_t top = 0;   // magnitudes order like their bits; NaNs lie above infinity
#pragma unroll
        for (int e = 0; e < 8; e++) top = max(top, __float_as_uint(v[e]) & 0x7fffffffu);
        top = __reduce_max_sync(0xffffffffu, top);
        // 2^(ex + 1) is above every value; scaled to below 2^30. In two steps: either factor alone may be outside f32
        const int ex = max((int)(top >> 23) - 127, -120);
        float scale = 0.f;
        if (top >= 0x7f800000u) {
            scale = __uint_as_float(0x7fc00000u);
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = 0.f;
        } else if (top != 0) {
            const int up = 29 - ex, a = min(up, 127), b = up - a;   // 0 <= b <= 22; up >= -98
            const float fa = __uint_as_float((uint32_t)(a + 127) << 23), fb = __uint_as_float((uint32_t)(b + 127) << 23);
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = v[e] * fa * fb;
            // 2^-up: down to 2^-149, below 2^-126 as a subnormal
            scale = up <= 126 ? __uint_as_float((uint32_t)(127 - up) << 23) : __uint_as_float(1u << (149 - up));
        }
        uint32_t q[4][2] = {};
#pragma unroll
        for (int e = 0; e < 8; e++) {
            int z = __float2int_rn(v[e]);
#pragma unroll
            for (int j = 3; j >= 0; j--) {
                const int digit = (int)(int8_t)(z & 0xff);
                q[j][e >> 2] |= (uint32_t)(digit & 0xff) << (8 * (e & 3));
                z = (z - digit) >> 8;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<uint2 *>(act + (n * 4 + j) * p.plane + sb * 256 + lane * 8) = make_uint2(q[j][0], q[j][1]);
        if (lane == 0) scales[n * p.units + sb] = scale;
    }
    consumers_sync();
}

// ---------------------------------------------------------------- a super-block of 16 rows
// {ql[128], qh[64], i8 scales[16], f16 d}; starts on 2-byte boundaries. Lane (g, t) brings words 4t of rows g and g + 8 and of column g of
// the digits, and gets sums of those rows with columns 2t and 2t + 1. b: this lane's word of group 0 of this super-block.
// NT = 0: one column; columns 0..3 are its digits against the first group of an instruction, 4..7 against the second.
// f[2 * nt], f[2 * nt + 1]: rows g and g + 8, the part of this lane's two digits. x: the columns' values of this super-block.
template <int NT>
__device__ __forceinline__ void unit_q6_K(const uint8_t *r0, const uint8_t *r1, const uint8_t *b, int pair_planes, const float *scale, int col_scales, const float *x, int64_t ldx,
                                          float (&f)[NT ? 2 * NT : 2]) {
    constexpr int N = NT ? NT : 1;
    const int lane = threadIdx.x & 31, t = lane & 3;
    const bool second = NT == 0 && lane >= 16;
    const uint32_t *w[2] = {reinterpret_cast<const uint32_t *>((uintptr_t)r0 & ~(uintptr_t)3), reinterpret_cast<const uint32_t *>((uintptr_t)r1 & ~(uintptr_t)3)};
    const uint32_t sh[2] = {(uint32_t)((uintptr_t)r0 & 2) * 8, (uint32_t)((uintptr_t)r1 & 2) * 8};
    auto word = [&](int r, int at) { return __funnelshift_r(w[r][at], w[r][at + 1], sh[r]); };   // word `at` of the block
    int acc[N][4] = {};
    // sign-extended scale bytes; one column: of this lane's group of the two
    const uint32_t sel0 = 0x8880u + 0x1111u * (uint32_t)(NT ? 0 : (t >> 1) * 2), sel1 = sel0 + 0x1111u;
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
            if constexpr (NT == 0) {
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const uint32_t x = *reinterpret_cast<const uint32_t *>(bg + m * 64 + (second ? 32 : 0));
                    int d[4];
                    imma32(d, c[0][2 * m], c[1][2 * m], c[0][2 * m + 1], c[1][2 * m + 1], second ? 0u : x, second ? x : 0u);
                    const int s0 = signed_byte(sc[0][m], is ? sel1 : sel0), s1 = signed_byte(sc[1][m], is ? sel1 : sel0);
                    acc[0][0] += s0 * d[0];
                    acc[0][1] += s0 * d[1];
                    acc[0][2] += s1 * d[2];
                    acc[0][3] += s1 * d[3];
                }
            } else {
#pragma unroll
                for (int run = 0; run < 4; run++) {
                    const int s0 = signed_byte(sc[0][run >> 1], (is ? sel1 : sel0) + 0x2222u * (run & 1)), s1 = signed_byte(sc[1][run >> 1], (is ? sel1 : sel0) + 0x2222u * (run & 1));
#pragma unroll
                    for (int nt = 0; nt < N; nt++) {
                        int d[4];
                        imma16(d, c[0][run], c[1][run], *reinterpret_cast<const uint32_t *>(bg + nt * pair_planes + run * 32));
                        acc[nt][0] += s0 * d[0];
                        acc[nt][1] += s0 * d[1];
                        acc[nt][2] += s1 * d[2];
                        acc[nt][3] += s1 * d[3];
                    }
                }
            }
        }
    }
    const float d0 = __half2float(*reinterpret_cast<const __half *>(r0 + 208)), d1 = __half2float(*reinterpret_cast<const __half *>(r1 + 208));
    const float weight = (t & 1) ? 0.25f : 16384.f;   // digits 2 and 3, or 0 and 1; the codes are 4 * (q - 32)
#pragma unroll
    for (int nt = 0; nt < N; nt++) {
        const float xs = scale[NT ? (2 * nt + (t >> 1)) * col_scales : 0];   // (multiplied last: it may be subnormal)
        float v0 = d0 * fmaf((float)acc[nt][0], 256.f, (float)acc[nt][1]) * weight, v1 = d1 * fmaf((float)acc[nt][2], 256.f, (float)acc[nt][3]) * weight;
        if (xs != xs || !isfinite(d0) || !isfinite(d1)) {
            // value by value, a quarter of the super-block per lane (of two columns: two quarters)
            const float *const col = x + (NT ? 2 * nt + (t >> 1) : 0) * ldx;
            for (int slot = NT ? 2 * (t & 1) : t, end = NT ? slot + 2 : slot + 1; slot < end; slot++) {
                f[2 * nt] += q6_K_slot_sum(r0, col, slot);
                f[2 * nt + 1] += q6_K_slot_sum(r1, col, slot);
            }
            continue;
        }
        f[2 * nt] = fmaf(v0, xs, f[2 * nt]);
        f[2 * nt + 1] = fmaf(v1, xs, f[2 * nt + 1]);
    }
    __syncwarp();
}

// ---------------------------------------------------------------- the kernel
// NT: pairs of columns of this pass (0: a single column)
template <int NT>
__global__ void __launch_bounds__(THREADS, 2) k_gemv_q6(const __grid_constant__ CUtensorMap map, const __grid_constant__ Params p) {
    constexpr int NC = NT ? 2 * NT : 1;
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
    const float *const scales = reinterpret_cast<const float *>(act + NC * 4 * p.plane);
    const int g = lane >> 2, t4 = lane & 3;
    const int per_group = p.groups > 1 ? p.units : WARPS;   // warps of a row group
    const int gr = warp / per_group, u0 = warp % per_group;
    const bool works = gr < p.groups;
    // plane of this lane's column: digit g % 4 (of column g / 4 of the pair)
    const float *const x = p.x + (int64_t)p.n0 * p.ldx;
    const uint8_t *const b0 = act + (NT ? g : g & 3) * p.plane + t4 * 4;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int e0 = 0; e0 < tiles; e0 += EPOCH) {
        const int e1 = min(tiles, e0 + EPOCH);
        for (int t = e0; t < e1; t++) {
            float f[NT ? 2 * NT : 2] = {};
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
                        unit_q6_K<NT>(tile + u * BLOCK, tile + 8 * p.row_stride + u * BLOCK, b0 + sb * 256, 8 * p.plane, scales + sb, p.units, x + sb * 256, p.ldx, f);
                    }
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(&empty[s]);
                if (++s == p.stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            // the lanes of a row: its digits (one column: and the two groups of an instruction)
#pragma unroll
            for (int i = 0; i < (NT ? 2 * NT : 2); i++) {
                f[i] += __shfl_xor_sync(0xffffffffu, f[i], 1);
                if (NT == 0) f[i] += __shfl_xor_sync(0xffffffffu, f[i], 2);
            }
            // part [tile of the epoch][warp][column][row]
            float *o = part + ((t - e0) * WARPS + warp) * NC * 16;
            if (works && (NT ? (t4 & 1) == 0 : t4 == 0)) {
#pragma unroll
                for (int nt = 0; nt < (NT ? NT : 1); nt++) {
                    const int n = NT ? 2 * nt + (t4 >> 1) : 0;
                    o[n * 16 + g] = f[2 * nt];
                    o[n * 16 + g + 8] = f[2 * nt + 1];
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
            p.y[(p.n0 + n) * p.ldy + row] = v;
        }
        if (e1 < tiles) consumers_sync();
    }
}

}  // namespace gemvq6

// ---------------------------------------------------------------- host side
constexpr int Q6_SMEM_ONE = 220 * 1024, Q6_SMEM_TWO = 110 * 1024;   // one CTA per SM, two

// fills the geometry of a pass of nc columns (1, 2 or 4); false when it does not fit
static bool gemv_q6_geometry(gemvq6::Params &p, int64_t K, int nc, size_t &smem, int &per_sm) {
    p.units = (int)(K / 256);
    p.row_bytes = p.units * gemvq6::BLOCK;
    p.boxes = p.units % 8 == 0;
    p.segs = p.boxes ? p.units / 8 : 1;
    p.groups = p.units < gemvq6::WARPS ? gemvq6::WARPS / p.units : 1;
    p.row_stride = p.boxes ? 8 * gemvq6::BLOCK : p.row_bytes;
    p.stage_stride = (16 * p.groups * p.row_stride + 15 + gemvq6::PAD + 127) / 128 * 128;
    p.plane = (int)K + (nc == 1 ? 32 : 16);   // the planes of a lane's word on different banks
    p.act_bytes = (nc * 4 * p.plane + nc * p.units * 4 + 127) / 128 * 128;
    const int fixed = p.act_bytes + gemvq6::EPOCH * gemvq6::WARPS * nc * 64;
    per_sm = fixed + 3 * p.stage_stride <= Q6_SMEM_TWO ? 2 : 1;
    p.stages = std::min(gemvq6::MAX_STAGES, ((per_sm == 2 ? Q6_SMEM_TWO : Q6_SMEM_ONE) - fixed) / p.stage_stride);
    smem = (size_t)std::max(p.stages, 0) * p.stage_stride + fixed;
    return p.stages >= 2;
}
bool gemv_q6_supported(int64_t K) {
    gemvq6::Params p{};
    size_t smem;
    int per_sm;
    return tc_available() && K % 256 == 0 && K >= 256 && K <= (1 << 20) && gemv_q6_geometry(p, K, 1, smem, per_sm);
}
void gemv_q6_configure() {
    auto set = [](auto *k) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Q6_SMEM_ONE); };
    set(gemvq6::k_gemv_q6<0>);
    set(gemvq6::k_gemv_q6<1>);
    set(gemvq6::k_gemv_q6<2>);
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
    for (int64_t n0 = 0; n0 < g.N;) {
        size_t smem = 0;
        int per_sm = 1, nc = g.N - n0 >= 4 ? 4 : (g.N - n0 >= 2 ? 2 : 1);
        while (!gemv_q6_geometry(p, g.K, nc, smem, per_sm)) {
            if (nc == 1) return cudaErrorInvalidValue;
            nc /= 2;
        }
        p.n0 = (int)n0;
        if (p.boxes && n0 == 0) {
            const cudaError_t e = tc_encode_2d_bytes(&map, g.W[0], (uint64_t)p.row_bytes, (uint64_t)p.M, (uint32_t)p.row_stride, 16);
            if (e != cudaSuccess) return e;
        }
        const dim3 grid((unsigned)(per_sm * sm_count)), block(gemvq6::THREADS);
        cudaError_t e;
        if (nc == 1) e = launch_pdl_if(g.early, gemvq6::k_gemv_q6<0>, grid, block, smem, st, map, p);
        else if (nc == 2) e = launch_pdl_if(g.early, gemvq6::k_gemv_q6<1>, grid, block, smem, st, map, p);
        else e = launch_pdl_if(g.early, gemvq6::k_gemv_q6<2>, grid, block, smem, st, map, p);
        if (e != cudaSuccess) return e;
        n0 += nc;
    }
    return cudaSuccess;
}

}  // namespace tlb
