// RoPE, rms-norm and scale of a 128-wide head row held by a half-warp, bit-exact against the eager bf16 path (append.cu says how).
#pragma once

#include "nckv_common.cuh"

namespace nckv {

__device__ __forceinline__ void unpack4(const uint2 &v, float (&f)[4]) {
    f[0] = bf16lo(v.x); f[1] = bf16hi(v.x);
    f[2] = bf16lo(v.y); f[3] = bf16hi(v.y);
}
__device__ __forceinline__ uint2 pack4(const float (&f)[4]) {
    return make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
}
__device__ __forceinline__ __nv_bfloat162 pair_of(uint32_t v) { return *reinterpret_cast<const __nv_bfloat162 *>(&v); }
__device__ __forceinline__ uint32_t word_of(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t *>(&v); }
// Two elements' rotation, y1 = bf16(bf16(x1 c) + bf16(x2 s)) and y2 = bf16(bf16(x1 (-s)) + bf16(x2 c)), in two-wide bf16 arithmetic.  The
// bits of the fp32 operations rounded to bf16 one by one: a product of two bf16 numbers is exact in fp32, so it is rounded once either
// way; a sum that fp32 rounds is of numbers 2^16 apart, and both ways leave the larger one.  Large launches are bound by the
// issue of instructions; with each value widened, multiplied and packed (72 a row's half, now 20) 8 x 2048 tokens of 12 + 12 + 12 heads took
// 82.8 us, now 67.4; 1 x 2048 11.2 / 9.3; 3 x 1531 of 16 + 4 + 4 16.1 / 13.1; one token in 64 rows 2.5 / 2.4.
__device__ __forceinline__ void rotate2(uint32_t x1, uint32_t x2, uint32_t c, uint32_t s, uint32_t &y1, uint32_t &y2) {
    const __nv_bfloat162 a = pair_of(x1), b = pair_of(x2), cc = pair_of(c), ss = pair_of(s);
    y1 = word_of(__hadd2_rn(__hmul2_rn(a, cc), __hmul2_rn(b, ss)));
    y2 = word_of(__hadd2_rn(__hmul2_rn(a, __hneg2(ss)), __hmul2_rn(b, cc)));
}
__device__ __forceinline__ float squares4(const float (&y)[4]) {
    float e = __fmul_rn(y[0], y[0]);
    e = __fmaf_rn(y[1], y[1], e);
    e = __fmaf_rn(y[2], y[2], e);
    return __fmaf_rn(y[3], y[3], e);
}

// RoPE -> rms-norm -> scale on a 128-wide head row held by 16 lanes; all 32 lanes of a warp must call this.
__device__ __forceinline__ void rope_norm_scale(uint2 &lo, uint2 &hi, uint2 c, uint2 s, float qk_scale, float eps) {
    float y1[4], y2[4];
    uint2 r1, r2;
    rotate2(lo.x, hi.x, c.x, s.x, r1.x, r2.x);
    rotate2(lo.y, hi.y, c.y, s.y, r1.y, r2.y);
    unpack4(r1, y1);
    unpack4(r2, y2);
    // Offset 16 of the tree joins lanes that one thread holds here.  Every level adds the same pairs as the
    // shuffle-down does for its lane 0, whichever lane of the butterfly looks at it (a sum of two commutes).
    float e = __fadd_rn(squares4(y1), squares4(y2));
#pragma unroll
    for (int off = 8; off >= 1; off >>= 1) e = __fadd_rn(e, __shfl_xor_sync(0xffffffffu, e, off));
    const float rstd = rsqrtf(__fadd_rn(__fdiv_rn(e, 128.0f), eps));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        y1[i] = __fmul_rn(y1[i], rstd);
        y2[i] = __fmul_rn(y2[i], rstd);
    }
    unpack4(pack4(y1), y1);
    unpack4(pack4(y2), y2);
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // pack4 applies the final bf16 rounding
        y1[i] = __fmul_rn(y1[i], qk_scale);
        y2[i] = __fmul_rn(y2[i], qk_scale);
    }
    lo = pack4(y1);
    hi = pack4(y2);
}

}  // namespace nckv
