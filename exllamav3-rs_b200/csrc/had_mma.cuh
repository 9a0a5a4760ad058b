// 128-point Hadamard transform of two neighbouring blocks by a warp, with the butterflies on the tensor core.  H128 = H8 (x) H16 on
// the index i = 16 a + b: X[a][b] of both blocks goes through shared memory into transposed MMA fragments (ldmatrix.trans),
// D0 = (H8 (+) H8) X contracts over a with the sign matrix as the A operand, D0 - as an fp16 pair hi + lo, which keeps 22 of its bits -
// becomes the A operand of the second product Y = D0 H16, whose columns are ordered so that a lane ends up with four consecutive
// outputs.  About a quarter of the instructions of the shuffle version (which needs 20 shuffles per 4 values); sums are formed in
// another order than hadamard_inner.cuh:93-147 does, so single results may differ from the shuffle version's by one fp16 step where
// the fp32 value sits on a rounding boundary.
// D0 is a sum of eight fp16 values and may leave fp16's range where the transform, which is 0.088 of such sums, does not.  A pair of
// blocks with such a sum, or with an infinity or a NaN among its values, goes through the shuffles, whose fp32 sums hold every input.
// (What the test costs, us without and with it: four layers of hidden 5120, 28 rows beside 4 x 256, 4334 and 4346; calls of 5120 x 17408
// at 4 bits, 52 rows 28.7 and 28.8, 2048 rows 321 and 320.  Of D0's size, with the shuffles in line: 4248 and 4267, 28.8 and 29.1.)
#pragma once
#include "common.cuh"

namespace exl3 {

// the two blocks of 128 values in the warp's `stage` by shuffles; a call, because the code is seldom needed
static __device__ __noinline__ uint4 had_shuffles(const uint8_t* stage, int lane)
{
    uint2 o[2];
    #pragma unroll
    for (int blk = 0; blk < 2; ++blk) {
        const uint2 v = *reinterpret_cast<const uint2*>(stage + blk * 256 + lane * 8);
        o[blk] = had128_lane(*reinterpret_cast<const half2*>(&v.x), *reinterpret_cast<const half2*>(&v.y), lane);
    }
    __syncwarp();
    return make_uint4(o[0].x, o[0].y, o[1].x, o[1].y);
}

struct HadMma {
    uint32_t h8, hb[2][2];             // H8 (+) H8 as A of the first product, H16 with permuted columns as B of the second

    static __device__ __forceinline__ uint32_t sign_pair(int i, int j0, int j1)
    {
        const uint32_t lo = (__popc(i & j0) & 1) ? 0xBC00u : 0x3C00u, hi = (__popc(i & j1) & 1) ? 0xBC00u : 0x3C00u;
        return lo | (hi << 16);
    }
    __device__ __forceinline__ explicit HadMma(int lane)
    {
        const int g = lane >> 2, t = lane & 3;
        h8 = sign_pair(g, 2 * t, 2 * t + 1);
        #pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            const int bp = 4 * (g >> 1) + 2 * nb + (g & 1);        // output column b' of MMA column g in column block nb
            hb[nb][0] = sign_pair(bp, 2 * t, 2 * t + 1);
            hb[nb][1] = sign_pair(bp, 2 * t + 8, 2 * t + 9);
        }
    }
    static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
    {
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
    // x: the lane's eight consecutive values (signs applied) of the 256; stage: 512 bytes of the warp's, free again on return;
    // out[blk]: four consecutive results of block blk, from offset(lane) on
    __device__ __forceinline__ void operator()(uint4 x, uint8_t* stage, int lane, uint2 (&out)[2]) const
    {
        constexpr float r128 = 0.088388347648f;
        *reinterpret_cast<uint4*>(stage + lane * 16) = x;
        __syncwarp();
        // four 8x8 matrices, transposed on the way out: (block 0, b 0..7), (block 0, b 8..15), (block 1, ...), (block 1, ...)
        uint32_t r0, r1, r2, r3;
        const int mat = lane >> 3, rr = lane & 7;                  // row a = rr of matrix mat
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                     : "r"((uint32_t)__cvta_generic_to_shared(stage + (mat >> 1) * 256 + rr * 32 + (mat & 1) * 16)) : "memory");
        __syncwarp();
        float d0[2][4];
        #pragma unroll
        for (int bh = 0; bh < 2; ++bh) {
            d0[bh][0] = d0[bh][1] = d0[bh][2] = d0[bh][3] = 0.f;
            mma(d0[bh], h8, 0u, 0u, h8, bh ? r1 : r0, bh ? r3 : r2);
        }
        // D0[(block, a')][b] -> A operand of the second product, as hi + lo
        uint32_t ahi[4], alo[4];
        #pragma unroll
        for (int bh = 0; bh < 2; ++bh)
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float p = d0[bh][2 * h], q = d0[bh][2 * h + 1];
                const half2 hi = __floats2half2_rn(p, q);
                const half2 lo = __floats2half2_rn(p - __low2float(hi), q - __high2float(hi));
                ahi[2 * bh + h] = *reinterpret_cast<const uint32_t*>(&hi);
                alo[2 * bh + h] = *reinterpret_cast<const uint32_t*>(&lo);
            }
        float y[2][4];
        #pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
            y[nb][0] = y[nb][1] = y[nb][2] = y[nb][3] = 0.f;
            mma(y[nb], ahi[0], ahi[1], ahi[2], ahi[3], hb[nb][0], hb[nb][1]);
            mma(y[nb], alo[0], alo[1], alo[2], alo[3], hb[nb][0], hb[nb][1]);
        }
        // for row a' = g of block 0 ([0], [1]) and of block 1 ([2], [3]): the outputs b' = 4t .. 4t+3
        #pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
            const half2 p = __floats2half2_rn(y[0][2 * blk] * r128, y[0][2 * blk + 1] * r128);
            const half2 q = __floats2half2_rn(y[1][2 * blk] * r128, y[1][2 * blk + 1] * r128);
            out[blk].x = *reinterpret_cast<const uint32_t*>(&p); out[blk].y = *reinterpret_cast<const uint32_t*>(&q);
        }
        // a hi beyond fp16 is a NaN in all sixteen outputs of its row, of which a lane has y[0][0] or y[0][2] (inf - inf in the products)
        if (__any_sync(0xffffffffu, !(fabsf(y[0][0] + y[0][2]) < INFINITY))) {
            const uint4 o = had_shuffles(stage, lane);
            out[0] = make_uint2(o.x, o.y); out[1] = make_uint2(o.z, o.w);
        }
    }
    static __device__ __forceinline__ int offset(int lane) { return 16 * (lane >> 2) + 4 * (lane & 3); }
};
// the lane's eight values times signs, in fp16
__device__ __forceinline__ uint4 had_signed8(uint4 x, uint4 signs)
{
    half2* h = reinterpret_cast<half2*>(&x);
    const half2* s = reinterpret_cast<const half2*>(&signs);
    #pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __hmul2(h[e], s[e]);
    return x;
}

}  // namespace exl3
