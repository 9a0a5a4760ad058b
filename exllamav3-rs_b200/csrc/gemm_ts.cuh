// EXL3 GEMM up to 128 rows (decoding, verify batches, many users, the ragged end of a prefill): the decoded weights are the
// tensor core's A operand and never leave the SM's tensor memory.
//
// What bounds it: turning codes into fp16 weights, 43 warp instructions per 16 x 16 tile and 47 cycles per scheduler with
// nothing around them (ALU pipe 22 instructions, FMA pipe 18, each at one per two clocks).  Everything else is arranged around
// that.  The product is transposed (weights^T . activations^T): the 128 columns of a block are the 128 lanes of the accumulator
// and the batch rows its N columns, so an MMA costs 27 cycles up to 32 rows, 32 at 64 and 64 at 128 (measured; with the weights
// as the B operand of a 256-row CTA-pair MMA it is 128 whatever the row count, 64 of the 95 cycles a tile took there).  A
// decoder warp hands its tiles over with one tcgen05.st per two tiles, because a tile's trellis order is the 16x128b register
// layout; a st keeps its lane quadrant's port busy for 4.4 cycles per tile, beside the decoding.  Through shared memory it was
// four stores per tile, and the operand reads of the tensor core out of the same 128 B/clk.
//
// The service roles share the schedulers with four busy decoders each, and every instruction of theirs costs about ten cycles:
// with 64-k units, two barriers per unit for the issuer and indices computed per unit they, not the decoders, set the pace
// (5120 x 17408, 4 bits, 52 rows, kernel alone: 43 us; 128-k units 33; lean producer loops and one elected issuer thread 29;
// epilogue warps of their own 26.5).  The loop runs at 55 cycles per tile and scheduler.
//
// A call behind other kernels also waits for its own instructions, every role for its own, at about 0.4 us per KB that it comes to
// first.  So what a CTA runs once is kept short: levels of a transform in a loop, a sign as the factor of an fma, 32-bit indices
// (64-bit divisions are subroutines).  Against everything unrolled, us, with four other instantiations run in front of each call:
// 5120 x 17408 at 4 bits, 1, 8 and 52 rows 22.9 -> 20.2, 25.0 -> 21.8, 27.5 -> 25.2; back to back 25.5 -> 25.4, 27.5 -> 27.2, 29.1
// both; steps of 28 layers of hidden 1024 with 8 rows 1706 -> 1625, six of 5120 with 8 rows 1125 -> 1098.  The decoders' tiles stay
// unrolled: half of them in a loop gives a cold call another 2 us and takes 0.3 us of every warm one.
//
// Whole calls, us, tcgen05 kernel of gemm_tc.cuh -> this one: 5120 x 17408 at 4 bits 45.5 -> 32.8 (32 rows), 45.6 -> 33.1 (52),
// 47.4 -> 35.1 (128); 52 rows at 3 and 8 bits 49.1 -> 36.0, 46.6 -> 34.9; 17408 x 5120 80.3 -> 34.6 (32 rows), 85.6 -> 41.3
// (128); 5120 x 5120 30.9 -> 17.3 and 31.1 -> 22.9; 5120 x 151936, 52 rows, 359 -> 183.
// Up to 16 rows it replaces a kernel that streamed raw codes through mma.sync (50 cycles per tile and scheduler up to 8 rows, more
// than twice that above), us: 5120 x 17408 at 4 bits 27.9 -> 25.6 (1 row), 29.3 -> 27.4 (8), 39.2 -> 27.4 (16); 17408 x 5120 at 3
// bits 37.2 -> 29.8, 39.9 -> 32.0, 58.5 -> 32.5; 5120 x 5120 18.8 -> 15.1, 21.0 -> 15.3, 33.2 -> 15.4.  The weights being rounded
// to fp16 here, as the format has them, the error against 64 bits falls from 4.2e-4 to 3.6e-4.
//
// Work: units of (128-column block, 128 k), column-block-major, in contiguous ranges per CTA (ts_split in gemm.cu); partial sums
// of a block that several CTAs share are added in owner order by the last one to arrive (deterministic).  Roles: warps 0..15
// decode, in four groups that take units in turn (warp w writes lane quadrant w % 4); warps 16..19 take finished accumulators
// out and run the output transform; then a producer of codes, a producer of activations, the MMA issuer (owner of tensor
// memory), and a warp that passes on the arrival of activations.
// Every wait is bounded; a CTA that gives up waits for its copies and MMAs in flight, frees tensor memory and sets the status word.
#pragma once
#include "gemm_tc.cuh"
#include "gemm_decode.cuh"

namespace exl3 {

constexpr int TS_DECODERS = 16;                     // then 4 epilogue warps and 4 service warps
constexpr int TS_SERVICE = TS_DECODERS + 4;
constexpr int TS_THREADS = (TS_DECODERS + 8) * 32;
constexpr int TS_UNIT_K = 128, TS_ROWS = TS_UNIT_K / 16;
constexpr int TS_MAX_N = 128;                       // batch rows = columns of the accumulator
constexpr int TS_SW = 6;                            // units of decoded weights in tensor memory, 64 columns each, behind the accumulator
constexpr int TS_SB = 6;                            // most slots of the activation ring
// Units of codes in shared memory.  A multiple of the four decoder groups, so that a slot always belongs to the same group: a
// group that could come to a slot before the load of another group's earlier unit there has landed would take that earlier
// phase's parity for its own.
constexpr int TS_SR = 8;
constexpr uint32_t TS_POLLS = 1u << 24, TS_NS = 100;   // a wait gives up after about two seconds
constexpr int TS_FEW = 4;                           // most rows that the kernel transforms itself
constexpr int TS_T_ROWS = 64, TS_TSTRIDE = 132;     // output tile: rows at a time, floats per row

// the activation ring takes what the codes leave of a CTA's 227 KB, 96 KB at most
constexpr int ts_b_bytes(int K)
{
    const int room = 225 * 1024 - TS_T_ROWS * TS_TSTRIDE * 4 - TS_SR * 256 * TS_ROWS * K;
    return room < 96 * 1024 ? room : 96 * 1024;
}

template <int K> struct TsSmem {
    static constexpr int RAW = 256 * TS_ROWS * K;                      // codes of a unit: 8 tile rows x 8 tiles
    static constexpr int SR = TS_SR;
    static constexpr int OFF_B = 0;
    static constexpr int OFF_RAW = OFF_B + ts_b_bytes(K);
    static constexpr int OFF_T = OFF_RAW + SR * RAW;
    static_assert(SR % 4 == 0, "a slot of codes belongs to one decoder group");
    static_assert(OFF_T >= TS_MAX_N * TS_TSTRIDE * 4, "the last block's rows fit into the two rings");
    // r_full, r_empty [SR], b_full [SB], w_full, done [SW], acc_full, d_free, t_full, t_free, fin, drain, last
    static constexpr int N_BARS = 2 * SR + TS_SB + 2 * TS_SW + 7;
    static constexpr int OFF_BAR = OFF_T + TS_T_ROWS * TS_TSTRIDE * 4;
    static constexpr int BYTES = OFF_BAR + N_BARS * 8 + 1024;          // + slack to align the base to 1024 bytes
    static_assert(BYTES >= EXL3_TMEM_SMEM, "no other holder of tensor memory beside it");
};

struct GemmTsParams {
    void* C[TC_MAX_SEG];               // [m][n] fp16 or fp32
    const half* svh[TC_MAX_SEG];       // [n] or NULL
    int n[TC_MAX_SEG];
    int blk_end[TC_MAX_SEG];           // running count of 128-column blocks; the last entry is the total
    float* partial;                    // [grid][2][m][128]: a CTA's first and last block when shared
    int* counters;                     // [column blocks] arrival counters, zero on entry and on exit
    int* status;
    int m, k, c_fp32;
    int nb;                            // m rounded up to 16
    int sb;                            // slots of the activation ring
    int aligned;                       // 1: every CTA owns whole column blocks
    // few rows: the activations as they come, [m][k] fp16 with a sign vector per tensor; the kernel transforms them itself
    const half* x;
    const half* suh[TC_MAX_SEG];
    int early;                         // 0: nothing of global memory is touched before the kernels in front are complete
};

// gemm_ts.cu
cudaError_t gemm_ts_launch(int K, int cb, const CUtensorMap* amap, const CUtensorMap* rmap, const GemmTsParams& p, int grid, bool overlap, cudaStream_t st);

__device__ __forceinline__ void ts_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// two tiles one below the other (32 k): lane 4g + t holds columns g, g + 8 and k pairs t, t + 4 of each
__device__ __forceinline__ void ts_st_tiles(uint32_t taddr, const half2 (&w)[8])
{
    const uint32_t* r = reinterpret_cast<const uint32_t*>(w);
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void ts_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

// Output transform of four rows of a 128-column block held by a warp (lane = 4 consecutive columns): 128-point Hadamard,
// signs, store.  Four at a time, because a row's five shuffle levels are one chain; the levels are a loop, which a cold call
// reaches sooner (see above).
__device__ __forceinline__ void ts_store_rows(float4 (&a)[4], int row, int m, int lane, bool transform, uint2 sv, void* Cout, int n, int n0, int c_fp32)
{
    const half2 s0 = *reinterpret_cast<const half2*>(&sv.x), s1 = *reinterpret_cast<const half2*>(&sv.y);
    if (transform) {
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float p = a[i].x + a[i].y, d = a[i].x - a[i].y, q = a[i].z + a[i].w, e = a[i].z - a[i].w;
            a[i].x = p + q; a[i].y = d + e; a[i].z = p - q; a[i].w = d - e;
        }
        #pragma unroll 1
        for (int o = 1; o < 32; o <<= 1) {
            const float sg = lane & o ? -1.0f : 1.0f;
            #pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float p0 = __shfl_xor_sync(0xffffffffu, a[i].x, o), p1 = __shfl_xor_sync(0xffffffffu, a[i].y, o);
                const float p2 = __shfl_xor_sync(0xffffffffu, a[i].z, o), p3 = __shfl_xor_sync(0xffffffffu, a[i].w, o);
                a[i].x = fmaf(a[i].x, sg, p0); a[i].y = fmaf(a[i].y, sg, p1);
                a[i].z = fmaf(a[i].z, sg, p2); a[i].w = fmaf(a[i].w, sg, p3);
            }
        }
    }
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (row + i >= m) break;
        float4 v = a[i];
        if (transform) { v.x *= TC_R128; v.y *= TC_R128; v.z *= TC_R128; v.w *= TC_R128; }
        const size_t off = (size_t)(row + i) * n + n0 + lane * 4;
        if (c_fp32) {
            if (transform) { v.x *= __low2float(s0); v.y *= __high2float(s0); v.z *= __low2float(s1); v.w *= __high2float(s1); }
            *reinterpret_cast<float4*>((float*)Cout + off) = v;
        } else {
            half2 x = __floats2half2_rn(v.x, v.y), y = __floats2half2_rn(v.z, v.w);
            if (transform) { x = __hmul2(x, s0); y = __hmul2(y, s1); }
            uint2 o; o.x = *reinterpret_cast<const uint32_t*>(&x); o.y = *reinterpret_cast<const uint32_t*>(&y);
            *reinterpret_cast<uint2*>((half*)Cout + off) = o;
        }
    }
}

// What finishing a column block takes: where it goes, this lane's four signs, and the CTAs that own parts of it.
struct TsBlock {
    const half* svh; void* C; uint2 sv;
    int n, n0, c_first, c_last, first1;
    __device__ __forceinline__ bool split() const { return c_first != c_last; }
};
__device__ __forceinline__ TsBlock ts_block(const GemmTsParams& p, int nbg, int KS, unsigned total, unsigned G, int lane)
{
    TsBlock b;
    const int seg = (nbg >= p.blk_end[0]) + (nbg >= p.blk_end[1]);
    b.n0 = (nbg - (seg == 0 ? 0 : (seg == 1 ? p.blk_end[0] : p.blk_end[1]))) * 128;
    b.svh = seg == 0 ? p.svh[0] : (seg == 1 ? p.svh[1] : p.svh[2]);
    b.C = seg == 0 ? p.C[0] : (seg == 1 ? p.C[1] : p.C[2]);
    b.n = seg == 0 ? p.n[0] : (seg == 1 ? p.n[1] : p.n[2]);
    b.sv = b.svh ? *reinterpret_cast<const uint2*>(b.svh + b.n0 + lane * 4) : make_uint2(0u, 0u);
    b.c_first = b.c_last = b.first1 = 0;
    if (!p.aligned) {
        const unsigned first = (unsigned)nbg * KS;
        auto owner = [&](unsigned u) -> int { return (int)(((u + 1) * G + total - 1) / total - 1); };
        b.c_first = owner(first); b.c_last = owner(first + KS - 1);
        // slot 0 of a CTA holds the partial sums of the block its range begins in, slot 1 of the one it ends in; only the first of
        // a block's owners can have begun in an earlier block
        b.first1 = (int)((total * b.c_first / G) / KS) != nbg;
    }
    return b;
}
// rows r0 .. rend - 1 of an output tile
__device__ __forceinline__ void ts_finish_tile(const GemmTsParams& p, const TsBlock& b, const float* T, int r0, int rend, int wi, int nw, int lane)
{
    #pragma unroll 1
    for (int row = r0 + wi * 4; row < rend; row += nw * 4) {
        float4 a[4];
        #pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(T + (row + i - r0) * TS_TSTRIDE + lane * 4);
        ts_store_rows(a, row, p.m, lane, b.svh != nullptr, b.sv, b.C, b.n, b.n0, p.c_fp32);
    }
}
// all rows of a shared block: the owners' partial sums in owner order (independent of arrival order)
__device__ __forceinline__ void ts_finish_partials(const GemmTsParams& p, const TsBlock& b, int wi, int nw, int lane)
{
    const size_t slot = (size_t)p.m * 128;
    #pragma unroll 1
    for (int row = wi * 4; row < p.m; row += nw * 4) {
        float4 a[4];
        #pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* src = p.partial + ((size_t)b.c_first * 2 + b.first1) * slot + (size_t)row * 128 + lane * 4;
        const float* next = p.partial + (size_t)(b.c_first + 1) * 2 * slot + (size_t)row * 128 + lane * 4;
        const int rows = p.m - row < 4 ? p.m - row : 4;
        for (int s = b.c_first; s <= b.c_last; s += 2) {
            // two owners' rows are requested before the first is added
            float4 v[2][4];
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                #pragma unroll
                for (int i = 0; i < 4; ++i)
                    v[h][i] = s + h <= b.c_last && i < rows ? __ldcg(reinterpret_cast<const float4*>(src + i * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
                src = next; next += 2 * slot;
            }
            #pragma unroll
            for (int h = 0; h < 2; ++h)
                #pragma unroll
                for (int i = 0; i < 4; ++i) { a[i].x += v[h][i].x; a[i].y += v[h][i].y; a[i].z += v[h][i].z; a[i].w += v[h][i].w; }
        }
        ts_store_rows(a, row, p.m, lane, b.svh != nullptr, b.sv, b.C, b.n, b.n0, p.c_fp32);
    }
}

// 128-point Hadamard transform of (x o signs) for 128 values of R rows, lane = 4 consecutive ones (arithmetic of gd_prologue_row).
// Two rows have a form of their own: with four, two of them repeated, 1024 x 3072 took 9.4 us instead of 8.0 (8.6 before this kernel).
template <int R>
__device__ __forceinline__ void ts_transform(uint2 (&x)[R], uint2 sg, int lane)
{
    float v[R][4];
    #pragma unroll
    for (int r = 0; r < R; ++r) {
        const half2 a = __hmul2(*reinterpret_cast<const half2*>(&x[r].x), *reinterpret_cast<const half2*>(&sg.x));
        const half2 b = __hmul2(*reinterpret_cast<const half2*>(&x[r].y), *reinterpret_cast<const half2*>(&sg.y));
        const float s0 = __low2float(a) + __high2float(a), d0 = __low2float(a) - __high2float(a);
        const float s1 = __low2float(b) + __high2float(b), d1 = __low2float(b) - __high2float(b);
        v[r][0] = s0 + s1; v[r][1] = d0 + d1; v[r][2] = s0 - s1; v[r][3] = d0 - d1;
    }
    #pragma unroll (R <= 2 ? 5 : 1)
    for (int i = 1; i < 32; i <<= 1) {
        const float sgn = lane & i ? -1.0f : 1.0f;
        #pragma unroll
        for (int r = 0; r < R; ++r)
            #pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float o = __shfl_xor_sync(0xffffffffu, v[r][e], i);
                v[r][e] = fmaf(v[r][e], sgn, o);
            }
    }
    #pragma unroll
    for (int r = 0; r < R; ++r) {
        const half2 p = __floats2half2_rn(v[r][0] * TC_R128, v[r][1] * TC_R128), q = __floats2half2_rn(v[r][2] * TC_R128, v[r][3] * TC_R128);
        x[r] = make_uint2(*reinterpret_cast<const uint32_t*>(&p), *reinterpret_cast<const uint32_t*>(&q));
    }
}

// Warp-uniform bounded wait with a short way through when the phase is complete already: one poll and one vote.
__device__ __forceinline__ bool ts_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t now;
    asm volatile("{\n\t.reg .pred p, q;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "vote.sync.all.pred q, p, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(now) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (now) return true;
    bool ok = false;
    for (uint32_t i = 0; i < TS_POLLS && !ok; ++i) ok = __all_sync(0xffffffffu, mbar_try_wait_hint(bar, parity, TS_NS));
    return ok;
}

// Activations of up to R rows, units odd, odd + 2, ... of the CTA: (x o signs), 128-point transform, rows of 128 bytes with the
// 16-byte chunks XORed with row & 7 in slot u % SW; the rows past m stay zero.  False when a wait ran out.
template <int R>
__device__ __forceinline__ bool ts_few_rows(const GemmTsParams& p, uint8_t* ring, uint64_t* done, uint64_t* w_full, int nbg, int ks, int KS, int nst, int odd, int lane)
{
    for (int i = lane; i < 3 * 256; i += 32)
        *reinterpret_cast<uint4*>(ring + (2 * (i >> 8) + odd) * 4096 + (i & 255) * 16) = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    pdl_wait();
    ks += odd;
    int sw = odd;
    uint32_t par = 1;
    uint2 x[R], sg = make_uint2(0u, 0u);
    bool sign = false;
    auto fetch = [&]() {
        while (ks >= KS) { ks -= KS; ++nbg; }
        const int seg = (nbg >= p.blk_end[0]) + (nbg >= p.blk_end[1]);
        const half* suh = seg == 0 ? p.suh[0] : (seg == 1 ? p.suh[1] : p.suh[2]);
        sign = suh != nullptr;
        if (sign) sg = reinterpret_cast<const uint2*>(suh + ks * TS_UNIT_K)[lane];
        #pragma unroll
        for (int r = 0; r < R; ++r)                                   // (rows past m repeat the last one and are not written)
            x[r] = reinterpret_cast<const uint2*>(p.x + (size_t)(r < p.m ? r : p.m - 1) * p.k + ks * TS_UNIT_K)[lane];
    };
    if (odd < nst) fetch();
    for (int s = odd; s < nst; s += 2) {
        uint2 h[R];
        #pragma unroll
        for (int r = 0; r < R; ++r) h[r] = x[r];
        if (sign) ts_transform<R>(h, sg, lane);
        ks += 2;
        if (s + 2 < nst) fetch();                                      // the next unit's, under the wait
        if (!ts_wait(&done[sw], par)) return false;
        uint8_t* dst = ring + sw * 4096 + (lane >> 4) * 2048 + (lane & 1) * 8;
        #pragma unroll
        for (int r = 0; r < R; ++r)
            if (r < p.m) *reinterpret_cast<uint2*>(dst + r * 128 + ((((lane & 15) >> 1) ^ r) << 4)) = h[r];
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_full[sw]);
        __syncwarp();
        sw += 2; if (sw >= TS_SW) { sw -= TS_SW; par ^= 1; }
    }
    return true;
}

// the same wait for one thread
__device__ __forceinline__ bool ts_wait1(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    for (uint32_t i = 0; i < TS_POLLS; ++i) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(TS_NS) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void ts_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    gd_tma_load_2d(dst, map, x, y, bar);
}

// grid = CTAs of the split (at most one per SM).  amap*: transformed activations [m][k] fp16, box 64 x nb, 128-byte swizzle;
// rmap*: the trellis of each tensor as a matrix of 64-bit words [k/16][n/16 * 4K], box 4 rows x 8 tiles.
template <int K, int CB>
__global__ void __launch_bounds__(TS_THREADS, 1) gemm_ts_kernel(const __grid_constant__ CUtensorMap amap0,
                                                               const __grid_constant__ CUtensorMap amap1,
                                                               const __grid_constant__ CUtensorMap amap2,
                                                               const __grid_constant__ CUtensorMap rmap0,
                                                               const __grid_constant__ CUtensorMap rmap1,
                                                               const __grid_constant__ CUtensorMap rmap2, const GemmTsParams p)
{
    using SM = TsSmem<K>;
    extern __shared__ uint8_t ts_smem_unaligned[];
    uint8_t* smem = ts_smem_unaligned + ((1024u - (smem_u32(ts_smem_unaligned) & 1023u)) & 1023u);
    uint64_t* r_full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
    uint64_t* r_empty = r_full + SM::SR;
    uint64_t* b_full = r_empty + SM::SR;
    uint64_t* w_full = b_full + TS_SB;        uint64_t* done = w_full + TS_SW;
    uint64_t* acc_full = done + TS_SW;        uint64_t* d_free = acc_full + 1;
    uint64_t* t_full = d_free + 1;            uint64_t* t_free = t_full + 1;
    uint64_t* fin_bar = t_free + 1;           uint64_t* drain = fin_bar + 1;
    uint64_t* last_bar = drain + 1;
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed, s_fin, s_last;

    if (p.early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int KS = p.k / TS_UNIT_K;                                    // units per column block
    const int blocks = p.blk_end[TC_MAX_SEG - 1];
    const unsigned total = (unsigned)blocks * KS, G = gridDim.x;
    const unsigned u0 = p.aligned ? (unsigned)(blocks * (unsigned)blockIdx.x / G) * KS : total * blockIdx.x / G;
    const unsigned u1 = p.aligned ? (unsigned)(blocks * (unsigned)(blockIdx.x + 1) / G) * KS : total * (blockIdx.x + 1) / G;
    const int nst = (int)(u1 - u0);
    const int nbg0 = (int)(u0 / KS), ks0 = (int)(u0 - (unsigned)nbg0 * KS);
    auto seg_of = [&](int nbg) -> int { return (nbg >= p.blk_end[0]) + (nbg >= p.blk_end[1]); };
    auto col0_of = [&](int nbg, int seg) -> int { return (nbg - (seg == 0 ? 0 : (seg == 1 ? p.blk_end[0] : p.blk_end[1]))) * 128; };

    if (tid == 0) {
        s_failed = 0;
        for (int i = 0; i < SM::SR; ++i) { mbar_init(&r_full[i], 1); mbar_init(&r_empty[i], 4); }
        for (int i = 0; i < TS_SB; ++i) mbar_init(&b_full[i], 1);
        for (int i = 0; i < TS_SW; ++i) { mbar_init(&w_full[i], 5); mbar_init(&done[i], 1); }
        mbar_init(acc_full, 1); mbar_init(d_free, 4);
        mbar_init(t_full, 4); mbar_init(t_free, 4); mbar_init(fin_bar, 1); mbar_init(drain, 1); mbar_init(last_bar, 1);
        mbar_fence_init();
    }
    if (warp == TS_SERVICE + 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!p.early) pdl_enter_first(0);
    const uint32_t tmem = s_tmem;
    bool failed = false;
    int issued = 0;                                                    // copies requested by a producer

    if (p.x && (warp == TS_SERVICE + 1 || warp == TS_SERVICE + 3)) {
        // ===== few rows: two warps take units in turn, transform their activations and write them where the TMA would
        const int odd = warp == TS_SERVICE + 3;
        failed = !(p.m == 1 ? ts_few_rows<1>(p, smem + SM::OFF_B, done, w_full, nbg0, ks0, KS, nst, odd, lane)
                 : p.m == 2 ? ts_few_rows<2>(p, smem + SM::OFF_B, done, w_full, nbg0, ks0, KS, nst, odd, lane)
                            : ts_few_rows<TS_FEW>(p, smem + SM::OFF_B, done, w_full, nbg0, ks0, KS, nst, odd, lane));
    } else if (warp == TS_SERVICE) {
        // ===== codes: one box of 8 tile rows x 8 tiles per unit
        if (lane == 0) {
            const uint32_t bars = smem_u32(r_full), ring = smem_u32(smem + SM::OFF_RAW);
            uint32_t slot = 0, par = 1;                               // the first round waits for nothing
            for (int nbg = nbg0, ks = ks0; issued < nst && !failed; ++nbg, ks = 0) {
                const int seg = seg_of(nbg), send = issued + KS - ks < nst ? issued + KS - ks : nst;
                const CUtensorMap* map = seg == 0 ? &rmap0 : (seg == 1 ? &rmap1 : &rmap2);
                const int x = (col0_of(nbg, seg) >> 4) * 4 * K;
                for (int y = ks * TS_ROWS; issued < send; ++issued, y += TS_ROWS) {
                    if (issued == SM::SR) pdl_wait();                 // from here on it waits for what depends on the activations
                    const uint32_t bar = bars + 8 * slot;
                    if (!ts_wait1(bar + 8 * SM::SR, par)) { failed = true; break; }
                    ts_load(ring + slot * SM::RAW, map, x, y, bar, SM::RAW);
                    if (++slot == SM::SR) { slot = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == TS_SERVICE + 1) {
        // ===== activations: two boxes of 64 k x nb rows per unit
        if (lane == 0) {
            pdl_wait();
            const uint32_t box = (uint32_t)p.nb * 128, bars = smem_u32(b_full), ring = smem_u32(smem + SM::OFF_B), dn = smem_u32(done);
            uint32_t slot = 0, prev = 0, par = 0;                     // prev: the weight slot of the unit that had this slot before
            for (int nbg = nbg0, ks = ks0; issued < nst && !failed; ++nbg, ks = 0) {
                const int seg = seg_of(nbg), send = issued + KS - ks < nst ? issued + KS - ks : nst;
                const CUtensorMap* map = seg == 0 ? &amap0 : (seg == 1 ? &amap1 : &amap2);
                for (int x = ks * TS_UNIT_K; issued < send; ++issued, x += TS_UNIT_K) {
                    if (issued >= p.sb) {
                        if (!ts_wait1(dn + 8 * prev, par)) { failed = true; break; }
                        if (++prev == TS_SW) { prev = 0; par ^= 1; }
                    }
                    const uint32_t bar = bars + 8 * slot, dst = ring + slot * 2 * box;
                    ts_load(dst, map, x, 0, bar, 2 * box);
                    gd_tma_load_2d(dst + box, map, x + 64, 0, bar);
                    if (++slot == (uint32_t)p.sb) slot = 0;
                }
            }
        }
    } else if (warp == TS_SERVICE + 3) {
        // ===== tells the issuer, on the barrier of a unit's weights, that its activations have landed: the issuer shares its
        // scheduler with four decoders, every instruction that it does not execute shortens the chain through the tensor core
        if (lane == 0) {
            int sb = 0, sw = 0;
            uint32_t par = 0;
            pdl_wait();
            for (int s = 0; s < nst; ++s) {
                if (!ts_wait1(smem_u32(b_full) + 8 * sb, par)) { failed = true; break; }
                mbar_arrive(&w_full[sw]);
                if (++sb == p.sb) { sb = 0; par ^= 1; }
                if (++sw == TS_SW) sw = 0;
            }
        }
    } else if (warp == TS_SERVICE + 2) {
        // ===== MMA issuer: one elected thread
        if (elect_one()) {
            constexpr uint32_t HI = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);     // SBO 1024, version 1, SWIZZLE_128B
            const uint32_t idesc = tc_idesc(p.nb, 128);
            const uint32_t b_lo = (smem_u32(smem + SM::OFF_B) >> 4) | (1u << 16), half = p.nb * 8;
            const uint32_t wf = smem_u32(w_full), dn = smem_u32(done);
            uint32_t s = 0, sb = 0, sw = 0, par_w = 0;
            pdl_wait();
            for (int ev = 0; s < (uint32_t)nst && !failed; ++ev) {     // column blocks
                const uint32_t part = ev == 0 ? KS - ks0 : KS, send = nst - s < part ? nst : s + part;
                if (ev > 0 && !ts_wait1(smem_u32(d_free), (ev & 1) ^ 1)) { failed = true; break; }
                uint32_t acc = 0;
                for (; s < send; ++s) {
                    if (!ts_wait1(wf + 8 * sw, par_w)) { failed = true; break; }
                    tc_fence_after();
                    const uint32_t a = tmem + TS_MAX_N + sw * (TS_UNIT_K / 2), b = b_lo + sb * (2 * half);
                    #pragma unroll
                    for (int kk = 0; kk < TS_UNIT_K / 16; ++kk)
                        ts_mma(tmem, a + kk * 8, ((uint64_t)HI << 32) | (b + (kk >> 2) * half + 2 * (kk & 3)), idesc, kk > 0 ? 1u : acc);
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(dn + 8 * sw) : "memory");
                    acc = 1;
                    if (++sb == (uint32_t)p.sb) sb = 0;
                    if (++sw == TS_SW) { sw = 0; par_w ^= 1; }
                }
                if (!failed) tc_commit(acc_full);
            }
            if (failed) { tc_commit(drain); mbar_wait(drain, 0); }     // leave no MMA in flight behind
        }
        __syncwarp();
    } else if (warp < TS_DECODERS) {
        // ===== decoders: four groups of four warps take units in turn; a warp decodes its quadrant's two tile columns
        const int q = warp & 3, grp = warp >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        const int lane_prev = (lane + 31) & 31;
        bool waited = false;
        int sr = grp % SM::SR, sw = grp;
        uint32_t par_r = 0, par_w = 1;
        #pragma unroll 1
        for (int s = grp; s < nst; s += 4) {
            if (!waited && s >= TS_SW) { pdl_wait(); waited = true; }      // in front of the waits, which then count from here
            if (!ts_wait(&r_full[sr], par_r)) { failed = true; break; }
            if (!ts_wait(&done[sw], par_w)) { failed = true; break; }      // at once in the first round
            tc_fence_after();
            const uint32_t* raw = reinterpret_cast<const uint32_t*>(smem + SM::OFF_RAW + sr * SM::RAW) + 2 * q * 8 * K;
            const uint32_t ta = lanes + TS_MAX_N + sw * (TS_UNIT_K / 2);
            #pragma unroll
            for (int c = 0; c < 2; ++c)
                #pragma unroll
                for (int r = 0; r < TS_ROWS; r += 2) {
                    half2 w[8];
                    #pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t* tile = raw + ((r + i) * 8 + c) * 8 * K;
                        uint32_t st[8];
                        if constexpr (K == 4) lane_states4(tile, lane, lane_prev, st);
                        else lane_states<K>(tile, lane, st);
                        w[4 * i + 0] = tc_decode_pair<CB>(st[0], st[1]);      // column g,     k 2t, 2t+1
                        w[4 * i + 2] = tc_decode_pair<CB>(st[2], st[3]);      // column g,     k 2t+8, 2t+9
                        w[4 * i + 1] = tc_decode_pair<CB>(st[4], st[5]);      // column g + 8, k 2t, 2t+1
                        w[4 * i + 3] = tc_decode_pair<CB>(st[6], st[7]);      // column g + 8, k 2t+8, 2t+9
                    }
                    ts_st_tiles(ta + ((uint32_t)(c * 16) << 16) + r * 8, w);
                }
            tc_wait_st_acc();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(&w_full[sw]); mbar_arrive(&r_empty[sr]); }
            __syncwarp();
            sr += 4; if (sr >= SM::SR) { sr -= SM::SR; par_r ^= 1; }
            sw += 4; if (sw >= TS_SW) { sw -= TS_SW; par_w ^= 1; }
        }
    } else {
        // ===== epilogue: one warp per lane quadrant takes the accumulators out whenever a block, or this CTA's part of it, is
        // complete, while the decoders go on with the next
        const int q = warp & 3;
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        uint32_t t_phase = 0, f_phase = 1, fin_phase = 0;
        pdl_wait();
        #pragma unroll 1
        for (int ev = 0, sbeg = 0, nbg = nbg0; sbeg < nst && !failed; ++ev, ++nbg) {
            const int part = ev == 0 ? KS - ks0 : KS;
            sbeg = nst - sbeg < part ? nst : sbeg + part;
            const bool last = sbeg == nst;
            const TsBlock blk = ts_block(p, nbg, KS, total, G, lane);
            if (!ts_wait(acc_full, ev & 1)) { failed = true; break; }
            tc_fence_after();
            // lane = column q * 32 + lane, register = batch row.  The last block goes out through the two rings, which are
            // idle by then and take all its rows, others through the output tile, 64 rows at a time.
            float* T = reinterpret_cast<float*>(smem + (last ? SM::OFF_B : SM::OFF_T));
            const bool tiled = !blk.split() && !last;
            const int step = tiled ? TS_T_ROWS : p.nb;
            for (int r0 = 0; r0 < p.m; r0 += step) {
                const int rend = p.m < r0 + step ? p.m : r0 + step;
                if (tiled) {
                    if (!ts_wait(t_free, f_phase)) { failed = true; break; }       // at once the first time
                    f_phase ^= 1;
                }
                if (blk.split()) {
                    float* dst = p.partial + ((size_t)blockIdx.x * 2 + (nbg != nbg0)) * p.m * 128 + q * 32 + lane;
                    #pragma unroll 1
                    for (int c0 = 0; c0 < rend; c0 += 16, dst += 16 * 128) {
                        float v[16];
                        ts_ld16(lanes + c0, v);
                        tc_wait_ld();
                        #pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c0 + i < rend) dst[i * 128] = v[i];
                    }
                } else {
                    float* dst = T + q * 32 + lane;
                    #pragma unroll 1
                    for (int c0 = r0; c0 < rend; c0 += 16, dst += 16 * TS_TSTRIDE) {
                        float v[16];
                        ts_ld16(lanes + c0, v);
                        tc_wait_ld();
                        #pragma unroll
                        for (int i = 0; i < 16; ++i) dst[i * TS_TSTRIDE] = v[i];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (rend == p.m) mbar_arrive(d_free);
                    mbar_arrive(t_full);
                }
                __syncwarp();
                if (!ts_wait(t_full, t_phase)) { failed = true; break; }
                t_phase ^= 1;
                if (!tiled) break;
                ts_finish_tile(p, blk, T, r0, rend, q, 4, lane);
                __syncwarp();
                if (lane == 0) mbar_arrive(t_free);
                __syncwarp();
            }
            if (failed) break;
            if (tiled) continue;
            // one arrival per CTA of a shared block: its release half publishes the partial sums of all warps (ordered before it
            // by the barrier above), its acquire half makes the other owners' visible here
            if (q == 0 && lane == 0) {
                int fin = 1;
                if (blk.split()) {
                    int old;
                    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(p.counters + nbg) : "memory");
                    fin = old == blk.c_last - blk.c_first;
                    if (fin) p.counters[nbg] = 0;
                }
                if (last) { s_last = fin; mbar_arrive(last_bar); }
                else { s_fin = fin; mbar_arrive(fin_bar); }
            }
            __syncwarp();             // no lane polls for the arrival before lane 0 has made it (a poll can suspend the warp)
            if (last) break;                                                     // all warps finish it, below
            if (!ts_wait(fin_bar, fin_phase)) { failed = true; break; }
            fin_phase ^= 1;
            if (*(volatile int*)&s_fin) ts_finish_partials(p, blk, q, 4, lane);
        }
    }
    // ===== the CTA's last block: the decoders have nothing left to do either
    if (warp < TS_SERVICE && !failed) {
        pdl_wait();
        const int nbg = (int)((u1 - 1) / KS);
        const TsBlock blk = ts_block(p, nbg, KS, total, G, lane);
        if (!ts_wait(last_bar, 0)) failed = true;
        else if (*(volatile int*)&s_last) {
            if (blk.split()) ts_finish_partials(p, blk, warp, TS_SERVICE, lane);
            else ts_finish_tile(p, blk, reinterpret_cast<const float*>(smem + SM::OFF_B), 0, p.m, warp, TS_SERVICE, lane);
        }
    }

    // ===== tear-down
    if (failed) s_failed = 1;
    tc_fence_before();
    __syncthreads();
    if (s_failed && lane == 0 && (warp == TS_SERVICE || warp == TS_SERVICE + 1)) {
        // copies requested and perhaps not landed: the CTA may not leave before they have
        const bool codes = warp == TS_SERVICE;
        const int depth = codes ? SM::SR : p.sb;
        for (int i = issued > depth ? issued - depth : 0; i < issued; ++i) mbar_wait(codes ? &r_full[i % depth] : &b_full[i % depth], (i / depth) & 1);
    }
    __syncthreads();
    if (warp == TS_SERVICE + 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
    if (tid == 0 && s_failed) atomicExch(p.status, 2);
}

}  // namespace exl3
