// The dot products of a one-token GEMV on warp-level integer tensor products (mma.sync m16n8k32): 16 rows x 4 blocks of 32
// columns a step. The weight stream of one token meets one vector, so a product of matrix shape is not there; what this form
// saves against dp4a is instructions. A lane takes whole 16-byte code blocks of two rows, masks its nibbles apart (three logic
// instructions per eight weights, the codes are the A operand as they come) and four products do what 64 dp4a a lane did.
//   * The 32 columns a product contracts are word j of FOUR blocks, one of each group of lanes, since that is how 16-byte loads
//     hand the codes out. Blocks have scales of their own, so they must not meet in one sum: column 2 n + d of the B operand
//     holds byte plane d of block n and zero for the other blocks. Eight columns are four blocks times two planes, all in use,
//     and lane (g, t) ends with both planes of block t for rows g and g + 8, the block whose scales it has loaded.
//   * x is fixed point per block of 32 columns, in two signed bytes (digits of base 256) against the block's largest magnitude / 32 639.
//     The sums are exact integers; one conversion and one multiply by (block scale x step) per row and block follow. x is off by at
//     most half a step, 1.5e-5 of the block's largest magnitude (the powers of two of gemv_device.cuh, P = 2: 1.5e-5 .. 3.1e-5 of
//     that of 16 values). An outlier coarsens twice as many values here, with a finer step. Relative error of a product of 2 560
//     columns, here and with P = 2: normal x 2.1e-5, 2.9e-5; one column of 64 times 30 4.6e-5, 4.9e-5, times 300 4.7e-5, 5.1e-5, and
//     for rows that have no weight on those columns 1.8e-3, 1.9e-3; Student's t of 1.5 degrees 4.7e-5, 5.2e-5.
// mma.sync m16n8k32 takes 8 cycles of an SM's quarter here, twice the rate of dp4a (which takes 2 for 128 weights and one plane).
#pragma once
#include "gemv_device.cuh"

namespace brasa_dev {

// Shared-memory form of x: planes [block][2][32 bytes], the words of a plane in the order the products take them (word 2 j: columns
// 4 j .. of the block, which are low nibbles; word 2 j + 1: columns 16 + 4 j .., high nibbles), and per block the bias term
// -BIAS x sum(X) and the step.
constexpr uint32_t X_PLANE_BYTES = 64, X_META_BYTES = 8, X_BLOCK_BYTES = X_PLANE_BYTES + X_META_BYTES;

__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Eight values of a block of 32 (columns 4 j .. and 16 + 4 j .., j = 0 .. 3) to fixed point; the block's four lanes are neighbours.
// Infinities and NaNs travel in the step; a block of zeros or denormals has step 0.
__device__ __forceinline__ void x_eighth_to_planes(uint8_t *planes, uint8_t *meta, uint32_t block, uint32_t j, float (&v)[8], int bias) {
    // (magnitudes compared as integers, so that a NaN is the largest of all)
    uint32_t most = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) most = max(most, __float_as_uint(v[k]) & 0x7FFFFFFFu);
    most = max(most, __shfl_xor_sync(0xffffffffu, most, 1));
    most = max(most, __shfl_xor_sync(0xffffffffu, most, 2));
    const float amax = __uint_as_float(most);
    const uint32_t ebits = most & 0x7F800000u;
    float step = amax * (1.0f / 32639.0f), inv;  // 127 x 256 + 127: the largest number two signed digits hold either way
    asm("rcp.approx.f32 %0, %1;" : "=f"(inv) : "f"(amax));  // (an ulp off moves no rounded value by more than 0.004)
    inv *= 32639.0f;
    if (!(ebits > (15u << 23) && ebits < 0x7F800000u)) {
        step = ebits == 0x7F800000u ? amax : 0.0f;
        inv = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 0.0f;
    }
    // 1.5 x 2^23 + 128 added: the sum's last bits are the integer, rounded to nearest even, plus 128, which turns the borrows of signed
    // digits into the bytes of an unsigned number
    uint32_t U[8];
    int total = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        U[k] = __float_as_uint(fmaf(v[k], inv, 12582912.0f + 128.0f));
        total += (int)(U[k] - 0x4B400080u);
    }
    uint32_t w[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t *u = U + 4 * h;
        const uint32_t lo01 = __byte_perm(u[0], u[1], 0x5140), lo23 = __byte_perm(u[2], u[3], 0x5140);
        w[0][h] = __byte_perm(lo01, lo23, 0x5410) ^ 0x80808080u;
        w[1][h] = __byte_perm(lo01, lo23, 0x7632);
    }
    total += __shfl_xor_sync(0xffffffffu, total, 1);
    total += __shfl_xor_sync(0xffffffffu, total, 2);
    uint8_t *dst = planes + (size_t)block * X_PLANE_BYTES + 8 * j;
    *reinterpret_cast<uint2 *>(dst) = make_uint2(w[0][0], w[0][1]);
    *reinterpret_cast<uint2 *>(dst + 32) = make_uint2(w[1][0], w[1][1]);
    if (j == 0) *reinterpret_cast<uint2 *>(meta + (size_t)block * X_META_BYTES) = make_uint2((uint32_t)(-bias * total), __float_as_uint(step));
}

// Where a lane finds its share of x: its B fragments and its block's bias term and step, group g0 first. Lanes whose column belongs to
// another block than their own read zeros.
struct XLane {
    const uint8_t *b, *meta;
    uint32_t bs;
};
__device__ __forceinline__ XLane x_lane(const uint8_t *planes, const uint8_t *meta, const uint8_t *zeros, uint32_t lane, uint32_t g0) {
    const uint32_t g = lane >> 2, t = lane & 3, block = 4 * g0 + t;
    const bool mine = (g >> 1) == t;
    XLane x;
    x.b = mine ? planes + block * X_PLANE_BYTES + (g & 1) * 32 : zeros;
    x.bs = mine ? 4 * X_PLANE_BYTES : 0u;
    x.meta = meta + block * X_META_BYTES;
    return x;
}
// A lane's places in a row: codes, scales and (q6_0) high bits of its block of group g0.
template <int QT>
struct TileRows {
    uint32_t c, s, h;
    __device__ __forceinline__ void set(uint32_t cols, uint32_t g0, uint32_t lane) {
        const uint32_t block = 4 * g0 + (lane & 3);
        c = block * 16;
        s = tiled_scale_off(QT, cols) + block * 2;
        h = tiled_hi_off(cols) + block * 8;
    }
    // Rows ra and rb, in shared memory (MMA rows g and g + 8) times group i of x, added to the lane's sums over its own block.
    __device__ __forceinline__ void group(const uint8_t *ra, const uint8_t *rb, bool both, const XLane &x, uint32_t i, float &acc_a, float &acc_b) const {
        const uint4 ca = *reinterpret_cast<const uint4 *>(ra + c + 64 * i);
        uint4 cb = make_uint4(0, 0, 0, 0);  // (a tile of up to eight rows: rb is not read)
        if (both) cb = *reinterpret_cast<const uint4 *>(rb + c + 64 * i);
        uint2 ha = make_uint2(0, 0), hb = ha;
        if (QT == BRASA_Q6_0) {
            ha = *reinterpret_cast<const uint2 *>(ra + h + 32 * i);
            if (both) hb = *reinterpret_cast<const uint2 *>(rb + h + 32 * i);
        }
        const float da = __half2float(*reinterpret_cast<const __half *>(ra + s + 8 * i)), db = both ? __half2float(*reinterpret_cast<const __half *>(rb + s + 8 * i)) : 0.0f;
        const uint4 *bp = reinterpret_cast<const uint4 *>(x.b + i * x.bs);
        const uint4 b0 = bp[0], b1 = bp[1];
        const uint2 meta = *reinterpret_cast<const uint2 *>(x.meta + i * 4 * X_META_BYTES);
        const float step = __uint_as_float(meta.y);
        const uint32_t wa[4] = {ca.x, ca.y, ca.z, ca.w}, wb[4] = {cb.x, cb.y, cb.z, cb.w};
        const uint32_t bw[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        int acc[4] = {(int)meta.x, 0, (int)meta.x, 0};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t a0 = wa[j] & 0x0F0F0F0Fu, a2 = (wa[j] >> 4) & 0x0F0F0F0Fu, a1 = wb[j] & 0x0F0F0F0Fu, a3 = (wb[j] >> 4) & 0x0F0F0F0Fu;
            if (QT == BRASA_Q6_0) {  // two high bits of every code: words 0 and 1 of a block share a word of them, 2 and 3 the other
                const uint32_t u = j < 2 ? ha.x : ha.y, v = j < 2 ? hb.x : hb.y;
                a0 = lop_and_or(j & 1 ? u << 2 : u, 0x30303030u, a0);
                a2 = lop_and_or(j & 1 ? u << 4 : u >> 2, 0x30303030u, a2);
                a1 = lop_and_or(j & 1 ? v << 2 : v, 0x30303030u, a1);
                a3 = lop_and_or(j & 1 ? v << 4 : v >> 2, 0x30303030u, a3);
            }
            imma(acc, a0, a1, a2, a3, bw[2 * j], bw[2 * j + 1]);
        }
        const float fa = (float)(acc[0] + acc[1] * 256), fb = (float)(acc[2] + acc[3] * 256);
        acc_a = fmaf(da * step, fa, acc_a);
        acc_b = fmaf(db * step, fb, acc_b);
    }
};

}  // namespace brasa_dev
