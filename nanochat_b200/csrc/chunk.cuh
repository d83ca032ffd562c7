// What a recurrence in chunks of 16 tokens needs (delta_chunk.cu): m16n8k8 tf32 products of fp32 operands in
// two terms each, the sums over channels of pairs of tokens, the order of the operands in the records.
#pragma once

#include "vec_io.cuh"

namespace nckv {

constexpr int CH_T = 16;  // tokens per chunk

// channel c of row t in a record: odd rows' halves of 32 channels are swapped, which keeps 16-byte reads of 8 rows free of conflicts
template <int KP> __device__ __forceinline__ int ch_at(int t, int c) { return t * KP + (c ^ ((t & 1) << 4)); }

// place of token i among the 16 summed positions: the four a lane of a fragment needs lie together
__device__ __forceinline__ int ch_place(int i) { return ((i & 7) >> 1) * 4 + ((i >> 3) << 1) + (i & 1); }

// sums of o[0 .. LEN) over the warp: each level halves what a lane still holds.  Returns the index a lane ends with.
template <int BIT, int LEN> __device__ __forceinline__ int scatter_sum(float *o, int lane) {
    if constexpr (BIT == 0) {
        return 0;
    } else if constexpr (LEN == 1) {
        o[0] += __shfl_xor_sync(0xffffffffu, o[0], BIT);
        return scatter_sum<BIT / 2, 1>(o, lane);
    } else {
        constexpr int HALF = LEN / 2;
        const bool up = (lane & BIT) != 0;
#pragma unroll
        for (int c = 0; c < HALF; ++c) {
            const float keep = up ? o[c + HALF] : o[c], give = up ? o[c] : o[c + HALF];
            o[c] = keep + __shfl_xor_sync(0xffffffffu, give, BIT);
        }
        return (up ? HALF : 0) + scatter_sum<BIT / 2, HALF>(o, lane);
    }
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same from zero
__device__ __forceinline__ void mma_tf32_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// x = hi + lo, hi rounded to the 11 bits that a tf32 operand keeps (the instruction itself drops the others), so that lo has one bit
// more than an operand at most: products of two such sums without lo * lo keep 23 to 24 bits
__device__ __forceinline__ void split_tf32(float x, uint32_t &hi, uint32_t &lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
struct Pair4 {  // the B values of two summed steps (x, y and z, w) in two terms
    uint32_t hi[4], lo[4];
    __device__ __forceinline__ explicit Pair4(const float4 &f) {
        split_tf32(f.x, hi[0], lo[0]);
        split_tf32(f.y, hi[1], lo[1]);
        split_tf32(f.z, hi[2], lo[2]);
        split_tf32(f.w, hi[3], lo[3]);
    }
};
struct LeftFrag {  // an accumulator fragment as left operand
    uint32_t hi[4], lo[4];
    LeftFrag() = default;
    __device__ __forceinline__ void take(const uint32_t (&h)[4], const uint32_t (&l)[4]) {  // its two terms, 16-byte aligned
        const uint4 a = *reinterpret_cast<const uint4 *>(h), b = *reinterpret_cast<const uint4 *>(l);
        hi[0] = a.x; hi[1] = a.z; hi[2] = a.y; hi[3] = a.w;
        lo[0] = b.x; lo[1] = b.z; lo[2] = b.y; lo[3] = b.w;
    }
    __device__ __forceinline__ explicit LeftFrag(const float (&s)[4]) {
        // accumulator (g, 2t) (g, 2t+1) (g+8, 2t) (g+8, 2t+1); operand (g, t) (g+8, t) (g, t+4) (g+8, t+4)
        split_tf32(s[0], hi[0], lo[0]);
        split_tf32(s[2], hi[1], lo[1]);
        split_tf32(s[1], hi[2], lo[2]);
        split_tf32(s[3], hi[3], lo[3]);
    }
};

// A tile of the state's transpose behind a chunk: decayed by the product of the chunk's decays (for the channels of this lane's two
// columns, in two terms, the second `next` floats behind the first) plus the chunk's share d.  Rounded to nearest: matrix instructions round
// their sums towards zero, and a product of decays rounded once is the same factor chunk after chunk where the decay is constant; both would
// pile up in the state.
__device__ __forceinline__ void decay_add(float (&s)[4], const float *decay, int next, const float (&d)[4]) {
    const float2 hi = *reinterpret_cast<const float2 *>(decay), lo = *reinterpret_cast<const float2 *>(decay + next);
    s[0] = fmaf(s[0], hi.x, fmaf(s[0], lo.x, d[0]));
    s[1] = fmaf(s[1], hi.y, fmaf(s[1], lo.y, d[1]));
    s[2] = fmaf(s[2], hi.x, fmaf(s[2], lo.x, d[2]));
    s[3] = fmaf(s[3], hi.y, fmaf(s[3], lo.y, d[3]));
}

// Sums over a warp's 32 channels (one per lane) of x_t k_i w_(i+1) .. w_t for all i < t, x being q (and k: BOTH) of token t; SHIFT: w_(i+1) ..
// w_(t-1).  Pairs whose numbers differ first in the bit of weight b form blocks of b x b; with the decays cut at the block's upper half,
// one factor with the row and one with the column, each at most 1, all eight rows and columns of a b are one matrix product.
// Level l has b = 8 >> l: row r stands for token (r / b) 2 b + b + r % b, column n for (n / b) 2 b + n % b.  acc[l]: rows g (x = k if BOTH,
// else q) and 8 + g (q if BOTH) of columns 2 t, 2 t + 1.  s: CH_PAIR_ROWS x CH_PAIR_STRIDE floats of the warp's own.
constexpr int CH_PAIR_ROWS = 24, CH_PAIR_STRIDE = 36;
template <bool BOTH, bool SHIFT>
__device__ __forceinline__ void pair_products(float *s, int lane, const float (&k)[CH_T], const float (&q)[CH_T], const float (&w)[CH_T],
                                              float4 (&acc)[4]) {
    const int g = lane >> 2, tg = lane & 3;
#pragma unroll
    for (int level = 0; level < 4; ++level) {
        const int b = 8 >> level;
#pragma unroll
        for (int block = 0; block < 8 / b; ++block) {
            const int half = block * 2 * b + b;
            float f = 1.f;
#pragma unroll
            for (int r = 0; r < b; ++r) {
                const int t = half + r, row = block * b + r;
                if (!SHIFT) f *= w[t];
                if (BOTH) s[row * CH_PAIR_STRIDE + lane] = f * k[t];
                s[((BOTH ? 8 : 0) + row) * CH_PAIR_STRIDE + lane] = f * q[t];
                if (SHIFT) f *= w[t];
            }
            f = 1.f;
#pragma unroll
            for (int r = b - 1; r >= 0; --r) {
                const int i = block * 2 * b + r;
                s[(16 + block * b + r) * CH_PAIR_STRIDE + lane] = f * k[i];
                f *= w[i];
            }
        }
        __syncwarp();
        float d[4], c[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // the order of the summed channels is free: a lane takes 8 tg .. 8 tg + 7
            const float *at = s + g * CH_PAIR_STRIDE + 8 * tg + 4 * h;
            const float4 x = *reinterpret_cast<const float4 *>(at);
            const float4 y = BOTH ? *reinterpret_cast<const float4 *>(at + 8 * CH_PAIR_STRIDE) : make_float4(0.f, 0.f, 0.f, 0.f);
            const Pair4 bb(*reinterpret_cast<const float4 *>(at + 16 * CH_PAIR_STRIDE));
            const float first[4] = {x.x, x.y, y.x, y.y}, second[4] = {x.z, x.w, y.z, y.w};
            const LeftFrag a0(first), a1(second);
            if (h == 0) {
                mma_tf32_first(d, a0.hi, bb.hi[0], bb.hi[1]);
                mma_tf32_first(c, a0.hi, bb.lo[0], bb.lo[1]);
            } else {
                mma_tf32(d, a0.hi, bb.hi[0], bb.hi[1]);
                mma_tf32(c, a0.hi, bb.lo[0], bb.lo[1]);
            }
            mma_tf32(d, a1.hi, bb.hi[2], bb.hi[3]);
            mma_tf32(c, a0.lo, bb.hi[0], bb.hi[1]);
            mma_tf32(c, a1.hi, bb.lo[2], bb.lo[3]);
            mma_tf32(c, a1.lo, bb.hi[2], bb.hi[3]);
        }
        acc[level] = make_float4(d[0] + c[0], d[1] + c[1], d[2] + c[2], d[3] + c[3]);
        __syncwarp();
    }
}
// Where pair (t, i), i < t, of kind 0 (rows g) or 1 (rows 8 + g) lies in acc: level, lane, component.
__device__ __forceinline__ void pair_place(int t, int i, int kind, int &level, int &lane, int &part) {
    const int bit = 31 - __clz(t ^ i), b = 1 << bit, block = t >> (bit + 1);
    const int row = block * b + (t & (b - 1)), col = block * b + (i & (b - 1));
    level = 3 - bit;
    lane = row * 4 + (col >> 1);
    part = 2 * kind + (col & 1);
}

__device__ __forceinline__ void bulk_load(void *smem_dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

}  // namespace nckv
