// Decode-class paged attention over 4-bit and 8-bit quantised KV pools (k_bits = v_bits, head_dim 128; one row block of a
// work item holds 8 * NB packed (query, head) rows): the kernel behind exl3_bighead_attn_paged_q for decode and short
// verify batches: up to 48 packed rows, but for 33 to 40 at 4 bits where a batch has work for all SMs and few sequences of fewer rows
// (attn_impl in attn.cu has both sides; else attn_qt.cuh).
// Reference semantics: kernels/attention.cu:97-269,1716-1870 with the cache codec of
// kernels/cache/q_cache_kernels.cuh:61-236 (a code c of a group of 32 rotated values stands for
// (c - (2^(B-1) - 1/2)) * scale / 2^(B-1)).
//
// What bounds it: instruction issue, not the pool's bytes, so everything is arranged around the instructions per key.
//  * Both products are transposed: S^T = K Q^T and O^T = V^T P^T put the keys and the output dims on the 16 rows of the
//    MMA and the packed rows on its 8 columns.  A decode row with 1..8 sibling heads then costs 8 + 8 MMAs per 16 keys
//    and 4 exponentials per lane instead of 16 + 16 and 8, and the output takes 32 registers instead of 64.
//  * A tile of 64 keys (codes and scales of one kv head) arrives by four tiled TMA copies issued by one thread, the codes
//    in the copy's swizzle of their row width, which makes every load below free of bank conflicts.
//  * K operands are the codes with an exponent put on them (one logic op or permute per pair).  An MMA pair covers one
//    group of 32 dims, so the group's scale is applied to the fp32 sum afterwards (one FMA per group and score instead of
//    one multiplication per code pair).  4-bit codes get an exponent fine enough to be centred exactly in fp16, once for
//    all rows; what the exponents add to a sum of 8-bit ones, -off * sum(q), is taken out of the fp32 sum.
//  * V operands are pairs of one dim over two neighbouring keys, built in registers from the two keys' words (a permute
//    pairs the bytes); V never goes through shared memory a second time.  Its scales are multiplied into the softmax
//    weights, per group.  The 4-bit offset 23.5 * sum(P s) comes from one MMA per group against a row of ones; 8-bit codes
//    are centred exactly in fp16 instead, where the offset would cost precision in the sums.
//  * A row's running maximum is reduced over the warp only in tiles where some score passes it.
//  * Warps are coupled by a full and an empty mbarrier per stage, not by a CTA barrier per tile, and take turns requesting
//    tiles.
// Per 16 keys and warp, 4 bits, row blocks of 8: 437 instructions, 204 of them on the ALU pipe, whose rate is the bound (65 %
// of the issue slots under ncu); 8 bits: 417 and 188.  Whole calls, 40 / 8 heads, before (4 bits: an arrangement with keys
// on the columns, 8 bits: the generic kernel) and now: 64 sequences, contexts 128 .. 32768, 5 rows each, 222 -> 144 us and
// 607 -> 160 us; 24 sequences, contexts 512 .. 16384, 4 / 8 bits: 5 rows 95 -> 68 and 221 -> 68 us, 15 rows 102 -> 93 and
// 223 -> 95, 25 rows 155 -> 144 and 287 -> 147, 45 rows 207 -> 193 and 285 -> 198.
// Error against 64 bits, value scales 0.01 .. 0.06: 4 bits 3.0e-4 -> 2.8e-4, 8 bits 3.4e-4 -> 3.1e-4.  Softmax weight x value
// scale is formed in fp16: under scores with a deviation of 6 the error at 8 bits is 6e-4 at value scales of 1, 0.01 and
// 1e-3 and 7e-4 at 1e-4, where the generic kernel, which rounds scale / 128 to fp16, has 8e-4, 8e-4, 2.2e-3 and 2.0e-2.
// Queries are rotated by H32 once per work unit (q . H(c) = H(q) . c; those near the end of fp16 are packed at an eighth),
// output rows once when the warps' parts are merged.
// Work distribution, split-KV partials and the combine kernel are those of attn_paged.cuh.
#pragma once
#include <cuda.h>
#include "attn_paged.cuh"
#include "async_copy.cuh"

namespace exl3 {

constexpr int QD_TK = 64;                 // keys per tile, 16 per warp
constexpr int QD_THREADS = 128;

template <int B, int NB> struct QdSmem {
    static constexpr int ROWB = 16 * B;                    // bytes of codes per key, head and plane
    static constexpr int CODES = QD_TK * ROWB;
    static constexpr int SCALES = QD_TK * 16;              // scales of two neighbouring heads per key (the copy is 16 bytes wide)
    static constexpr int STAGE = 2 * CODES + 2 * SCALES;   // a multiple of 1024: stages keep the swizzle's alignment
    static constexpr int STAGES = B == 4 && NB == 1 ? 5 : 4;
    static constexpr int AHEAD = STAGES - 2;               // tiles requested ahead: a warp may run two tiles behind the fastest
    static constexpr int PIPE = STAGES * STAGE;
    static constexpr int MERGE = 4 * 8 * NB * (128 + 4) * 4;
    static_assert(MERGE <= PIPE && STAGE % 1024 == 0, "stage layout");
    static constexpr int OFF_BAR = PIPE;                   // full[STAGES], empty[STAGES]
    static constexpr int BYTES = PIPE + 128 + 1024;        // barriers, slack to align the base to 1024 bytes
};

__device__ __forceinline__ void qd_tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ float qd_ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t qd_transpose(uint32_t x)
{
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
__device__ __forceinline__ uint32_t qd_hmul2(uint32_t a, uint32_t b)
{
    const half2 r = __hmul2(*reinterpret_cast<const half2*>(&a), *reinterpret_cast<const half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
// d = a . b
__device__ __forceinline__ void qd_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t qd_lds32(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 qd_lds64(uint32_t a)
{
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
// A constant that stays in a register, so that (x & M) | E is one logic operation with one immediate.
__device__ __forceinline__ uint32_t qd_reg(uint32_t x)
{
    asm volatile("mov.b32 %0, %0;" : "+r"(x));
    return x;
}
// (x & m) | e
__device__ __forceinline__ uint32_t qd_field(uint32_t x, uint32_t m, uint32_t e)
{
    uint32_t y;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(y) : "r"(x), "r"(m), "r"(e));
    return y;
}
struct QdConst { uint32_t e16, e256, e512, e1024, x64, x4, x2; };

// K, 4 bits: the four fp16 pairs (n_i - 7.5, n_{i+4} - 7.5) of a word: 256 + n for even i, 16 + n for odd i, whose fp16 steps
// are fine enough to take the centre out exactly.  Both words come from one shift and one multiplication.
__device__ __forceinline__ void qd_pairs4_k(uint32_t w, uint32_t (&x)[4], const QdConst& c)
{
    const uint32_t l = w * c.x4, h = w >> 6;
    x[0] = qd_field(l, 0x003C003Cu, c.e256);
    x[1] = qd_field(l, 0x03C003C0u, c.e16);
    x[2] = qd_field(h, 0x003C003Cu, c.e256);
    x[3] = qd_field(h, 0x03C003C0u, c.e16);
    const half2 o256 = __float2half2_rn(263.5f), o16 = __float2half2_rn(23.5f);
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const half2 a = __hsub2(*reinterpret_cast<const half2*>(&x[i]), (i & 1) ? o16 : o256);
        x[i] = *reinterpret_cast<const uint32_t*>(&a);
    }
}
// V, 4 bits: fp16 pairs 16 + n of four dims over two keys, from the keys' words (the selectors pick the two bytes that hold
// the dims).  The left shifts are multiplications, which run beside the logic operations on another pipe.
__device__ __forceinline__ void qd_pairs4_v(uint32_t w0, uint32_t w1, uint32_t sel_lo, uint32_t sel_hi, uint32_t (&x)[4], const QdConst& c)
{
    const uint32_t lo = __byte_perm(w0, w1, sel_lo), hi = __byte_perm(w0, w1, sel_hi);
    x[0] = qd_field(lo * c.x64, 0x03C003C0u, c.e16);
    x[1] = qd_field(lo * c.x4, 0x03C003C0u, c.e16);
    x[2] = qd_field(hi * c.x64, 0x03C003C0u, c.e16);
    x[3] = qd_field(hi * c.x4, 0x03C003C0u, c.e16);
}
// K, 8 bits: the fp16 pairs of the bytes (0, 2) and (1, 3) of a word, 1024 + n: one permute each.
__device__ __forceinline__ void qd_pairs8_k(uint32_t w, uint32_t& x0, uint32_t& x1, const QdConst& c)
{
    x0 = __byte_perm(w, c.e1024, 0x5250);
    x1 = __byte_perm(w, c.e1024, 0x5351);
}
// V, 8 bits: the fp16 pairs of the bytes (0, 2) and (1, 3) of a word, 512 + n (which can be centred exactly in fp16).
__device__ __forceinline__ void qd_pairs8_v(uint32_t w, uint32_t& x0, uint32_t& x1, const QdConst& c)
{
    x0 = qd_field(w * c.x2, 0x01FE01FEu, c.e512);
    x1 = qd_field(w >> 7, 0x01FE01FEu, c.e512);
}

// Resident CTAs per SM the kernel is compiled for and launched with: four where a stage is 10 KB and a CTA has one column
// block (128 registers), else three.
constexpr int qd_ctas(int b, int nb) { return b == 4 && nb == 1 ? 4 : 3; }

template <int B, int NB>
__global__ void __launch_bounds__(QD_THREADS, qd_ctas(B, NB))
attn_qdec_kernel(const __grid_constant__ CUtensorMap map_qk, const __grid_constant__ CUtensorMap map_qv,
                 const __grid_constant__ CUtensorMap map_sk, const __grid_constant__ CUtensorMap map_sv, const AttnParams p)
{
    pdl_enter_late();
    using SM = QdSmem<B, NB>;
    constexpr int D = 128, ROWS = 8 * NB;
    extern __shared__ uint8_t qd_smem_unaligned[];
    uint8_t* smem = qd_smem_unaligned + ((1024u - (smem_u32(qd_smem_unaligned) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
    uint64_t* empty = full + SM::STAGES;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int G = p.nq / p.nkv;
    const int n_items = p.plan->n_items, chunk = p.plan->chunk;
    __shared__ uint32_t s_asked[SM::STAGES];               // parity of the last copy requested into a stage, 2 = none yet
    if (tid == 0) {
        #pragma unroll
        for (int s = 0; s < SM::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 4); s_asked[s] = 2; }
        mbar_fence_init();
    }
    // stage and parity of the next tile to consume and of the next to request (the same in every thread)
    int c_stage = 0, i_stage = 0;
    uint32_t c_par = 0, i_par = 1;                         // a stage is waited for from its second use on
    const QdConst cst = {qd_reg(0x4C004C00u), qd_reg(0x5C005C00u), qd_reg(0x60006000u), qd_reg(0x64006400u), qd_reg(64u), qd_reg(4u), qd_reg(2u)};
    // Byte offsets in a stage of this lane's first word of K and of V.  The chunk index of the copies' swizzle sits in
    // address bits 4.. of a 1024-byte aligned stage, so that chunk c of a row is reached by XOR with c << 4:
    //   K, 4 bits: chunk j ^ (key / 2 % 4), word t; 8 bits: chunk (2 j + h) ^ (key % 8), word t;  keys g and g + 8
    //   V, 4 bits: chunk j ^ (key / 2 % 4), word g / 2; 8 bits: chunk (2 j + g / 4) ^ (key % 8), word g % 4;  keys 2t, 2t+1, +8, +9
    const uint32_t base = smem_u32(smem);
    const uint32_t k_off = (warp * 16 + g) * SM::ROWB + ((B == 4 ? g >> 1 : g) << 4) + 4 * t;
    const uint32_t v_off = SM::CODES + (warp * 16 + 2 * t) * SM::ROWB +
                           (B == 4 ? (t << 4) + 4 * (g >> 1) : (((g >> 2) ^ (2 * t)) << 4) + 4 * (g & 3));
    const uint32_t sel_lo = (g & 1) ? 0x3632u : 0x1410u, sel_hi = (g & 1) ? 0x2723u : 0x0501u;

    __shared__ int s_unit;
    const int n_units = n_items * p.nkv;
    for (;;) {
        __syncthreads();                                   // the previous unit's merge buffer and s_unit are free
        if (tid == 0) s_unit = atomicAdd(const_cast<int*>(&p.plan->next), 1);
        __syncthreads();
        const int unit = s_unit;
        if (unit >= n_units) break;
        const AttnItem item = p.items[unit / p.nkv];
        const int item_idx = item.idx, kvh = unit % p.nkv;
        const int b = item.b, row_base = item.row_base, ql = item.ql, total_k = item.total_k, splits = item.splits;
        const int r0 = item.rb * ROWS;
        const int i_last = min(ql - 1, (r0 + ROWS - 1) / G);
        const int vis_max = p.causal ? min(total_k, total_k - ql + i_last + 1) : total_k;
        const int k_begin = item.split * chunk;
        const int k_end = min(min(k_begin + chunk, total_k), vis_max);
        const int32_t* bt = p.block_table + (size_t)b * p.pps;
        const int n_tiles = k_end > k_begin ? (k_end - k_begin + QD_TK - 1) / QD_TK : 0;
        const bool both = NB > 1 && ql * G - r0 > 8;       // the second column block of the MMAs holds rows

        // ---- tile loads: one thread, four tiled copies per tile (a tile of 64 keys lies inside one 256-token page).  The
        // warps take turns, so that none of them waits for every block-table entry.
        bool failed = false;
        auto issue = [&](int tile) {
            if (warp == (tile & 3) && lane == 0) {
                const int k0 = k_begin + tile * QD_TK;
                const int tok0 = bt[k0 >> 8] * EXL3_PAGE + (k0 & 255);
                if (!mbar_wait(&empty[i_stage], i_par)) failed = true;
                else {
                    const uint32_t dst = smem_u32(smem + i_stage * SM::STAGE), bar = smem_u32(&full[i_stage]);
                    s_asked[i_stage] = i_par ^ 1u;
                    mbar_expect_tx(&full[i_stage], SM::STAGE);
                    qd_tma_2d(dst, &map_qk, kvh * 4 * B, tok0, bar);
                    qd_tma_2d(dst + SM::CODES, &map_qv, kvh * 4 * B, tok0, bar);
                    qd_tma_2d(dst + 2 * SM::CODES, &map_sk, (kvh >> 1) * 8, tok0, bar);
                    qd_tma_2d(dst + 2 * SM::CODES + SM::SCALES, &map_sv, (kvh >> 1) * 8, tok0, bar);
                }
            }
            if (++i_stage == SM::STAGES) { i_stage = 0; i_par ^= 1; }
        };
        // the stages were last written and read through the generic proxy (merge buffer of the previous unit, zeroed scales)
        if (lane == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        #pragma unroll 1
        for (int pre = 0; pre < SM::AHEAD; ++pre)
            if (pre < n_tiles) issue(pre);

        // ---- Q as B operands.  Lane (g, t) holds row g of a column block at the eight dims of every group whose codes it
        // unpacks from a key: 4 bits: dims 8t .. 8t+7 (word t of the group), 8 bits: dims 4t .. 4t+3 and 16 + 4t .. (word t
        // of either half).  H32 runs over the lane's eight values and the quad.  cini (8 bits): minus the exponents' share of a sum.
        uint32_t w[NB][4][4];
        half2 qmax = __float2half2_rn(0.f);
        #pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            const int row = r0 + nb * 8 + g;
            const int qidx = row / G, head = kvh * G + (row - qidx * G);
            const half* qp = p.q + ((size_t)(row_base + qidx) * p.nq + head) * D;
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint4 raw = make_uint4(0u, 0u, 0u, 0u);
                if (row < ql * G) {
                    if constexpr (B == 4) raw = *reinterpret_cast<const uint4*>(qp + 32 * j + 8 * t);
                    else {
                        const uint2 lo = *reinterpret_cast<const uint2*>(qp + 32 * j + 4 * t);
                        const uint2 hi = *reinterpret_cast<const uint2*>(qp + 32 * j + 16 + 4 * t);
                        raw = make_uint4(lo.x, lo.y, hi.x, hi.y);
                    }
                }
                w[nb][j][0] = raw.x; w[nb][j][1] = raw.y; w[nb][j][2] = raw.z; w[nb][j][3] = raw.w;
                #pragma unroll
                for (int e = 0; e < 4; ++e) qmax = __hmax2(qmax, __habs2(*reinterpret_cast<const half2*>(&w[nb][j][e])));
            }
        }
        // A group that lines up with a row of the transform grows by sqrt(32) and would leave fp16 from 11580 on.  Such queries
        // are packed at an eighth, which keeps every finite one in range (46 318), and the scores are taken up again.  (Every
        // warp holds all rows of the block, so the CTA's warps agree.)
        const bool big = __any_sync(0xffffffffu, fmaxf(__low2float(qmax), __high2float(qmax)) > 11576.f);
        const float q_mul = big ? 0.125f * R32 : R32;
        const float s_mul = p.scale_log2 * (big ? 8.f / (float)(1 << (B - 1)) : 1.f / (float)(1 << (B - 1)));
        uint32_t qf[NB][8][2];
        float cini[NB][4][2];
        int lim[NB][2];                                    // keys visible to rows 2t, 2t+1 of the column block
        int wlim = 0x7fffffff;
        #pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                float v[8];
                #pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const half2 x = *reinterpret_cast<const half2*>(&w[nb][j][e]);
                    v[2 * e] = __low2float(x); v[2 * e + 1] = __high2float(x);
                }
                #pragma unroll
                for (int st = 1; st < 8; st <<= 1) {
                    #pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if ((e & st) == 0) { const float a = v[e], c = v[e | st]; v[e] = a + c; v[e | st] = a - c; }
                }
                #pragma unroll
                for (int st = 1; st < 4; st <<= 1) {
                    #pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float o = __shfl_xor_sync(0xffffffffu, v[e], st);
                        v[e] = ((t & st) ? -v[e] : v[e]) + o;
                    }
                }
                #pragma unroll
                for (int e = 0; e < 8; ++e) v[e] *= q_mul;
                if constexpr (B == 4) {                    // pair i of a word: codes i, i + 4
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) qf[nb][2 * j + (i >> 1)][i & 1] = pack_h2(v[i], v[i + 4]);
                } else {                                   // pairs of a word: codes (0, 2) and (1, 3)
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) qf[nb][2 * j + (i >> 1)][i & 1] = pack_h2(v[4 * (i >> 1) + (i & 1)], v[4 * (i >> 1) + (i & 1) + 2]);
                }
                if constexpr (B == 8) {
                    // what the exponents put on the codes adds to the products (of the rounded values, which the MMA multiplies)
                    float sum = 0.f;
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const half2 x = *reinterpret_cast<const half2*>(&qf[nb][2 * j + (i >> 1)][i & 1]);
                        sum = fmaf(1151.5f, __low2float(x) + __high2float(x), sum);
                    }
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    cini[nb][j][0] = -__shfl_sync(0xffffffffu, sum, 8 * t);
                    cini[nb][j][1] = -__shfl_sync(0xffffffffu, sum, 8 * t + 4);
                }
            }
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + nb * 8 + 2 * t + h;
                const bool rv = r < ql * G;
                lim[nb][h] = rv ? min(k_end, p.causal ? total_k - ql + r / G + 1 : total_k) : 0;
                if (rv) wlim = min(wlim, lim[nb][h]);
            }
        }
        wlim = min(wlim, __shfl_xor_sync(0xffffffffu, wlim, 1));
        wlim = min(min(wlim, __shfl_xor_sync(0xffffffffu, wlim, 2)), k_end);

        float o_acc[NB][8][4];                             // [m block]: dims 32 (mb / 2) + 4 g + 2 (mb % 2) + {0, 1}, rows 2t, 2t+1
        float cs[NB][4];                                   // row j (lanes g = j): sum over keys of P * scale of group j (4 bits only)
        float m_run[NB][2], l_run[NB][2];
        #pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            #pragma unroll
            for (int i = 0; i < 8; ++i) o_acc[nb][i][0] = o_acc[nb][i][1] = o_acc[nb][i][2] = o_acc[nb][i][3] = 0.f;
            cs[nb][0] = cs[nb][1] = cs[nb][2] = cs[nb][3] = 0.f;
            m_run[nb][0] = m_run[nb][1] = -INFINITY;
            l_run[nb][0] = l_run[nb][1] = 0.f;
        }
        const uint32_t s_off = 2 * SM::CODES + warp * 256 + (kvh & 1) * 8;      // this head's 4 scales inside a key's 16-byte pair

        for (int tile = 0; tile < n_tiles; ++tile) {
            if (tile + SM::AHEAD < n_tiles) issue(tile + SM::AHEAD);
            if (!mbar_wait(&full[c_stage], c_par)) failed = true;
            if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
            const uint32_t sb = base + c_stage * SM::STAGE;
            uint64_t* done = &empty[c_stage];
            if (++c_stage == SM::STAGES) { c_stage = 0; c_par ^= 1; }
            const int kbase = k_begin + tile * QD_TK + warp * 16;      // first key of this warp's 16
            if (kbase + 16 > k_end) {                                  // warp-uniform: the end of the range
                if (kbase >= k_end) {
                    if (lane == 0) mbar_arrive(done);
                    continue;
                }
                // rows of the page past the sequence hold any bits: their scales become zero
                if (lane < 16 && kbase + lane >= k_end) {
                    const uint32_t z = sb + s_off + lane * 16;
                    asm volatile("st.shared.v2.b32 [%0], {%1, %1};" ::"r"(z), "r"(0u) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1, %1};" ::"r"(z + SM::SCALES), "r"(0u) : "memory");
                }
                __syncwarp();
            }

            // ---- S^T = K Q^T, group by group (two MMAs each); keys g and g + 8 of the warp's 16
            float s_acc[NB][4];
            {
                const uint32_t ka = sb + k_off;
                const uint2 sca = qd_lds64(sb + s_off + g * 16), scb = qd_lds64(sb + s_off + g * 16 + 128);
                #pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t xa[4], xb[4];
                    if constexpr (B == 4) {
                        const uint32_t a = ka ^ (j << 4);
                        qd_pairs4_k(qd_lds32(a), xa, cst);
                        qd_pairs4_k(qd_lds32(a + 8 * SM::ROWB), xb, cst);
                    } else {
                        #pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t a = ka ^ ((2 * j + h) << 4);
                            qd_pairs8_k(qd_lds32(a), xa[2 * h], xa[2 * h + 1], cst);
                            qd_pairs8_k(qd_lds32(a + 8 * SM::ROWB), xb[2 * h], xb[2 * h + 1], cst);
                        }
                    }
                    const half2 ha = *reinterpret_cast<const half2*>(j < 2 ? &sca.x : &sca.y);
                    const half2 hb = *reinterpret_cast<const half2*>(j < 2 ? &scb.x : &scb.y);
                    const float fa = (j & 1) ? __high2float(ha) : __low2float(ha), fb = (j & 1) ? __high2float(hb) : __low2float(hb);
                    #pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        if (nb > 0 && !both) continue;
                        float d[4];
                        qd_mma0(d, xa[0], xb[0], xa[1], xb[1], qf[nb][2 * j][0], qf[nb][2 * j][1]);
                        mma_f16(d, xa[2], xb[2], xa[3], xb[3], qf[nb][2 * j + 1][0], qf[nb][2 * j + 1][1]);
                        #pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float v = B == 4 ? d[e] : d[e] + cini[nb][j][e & 1];
                            s_acc[nb][e] = j == 0 ? v * (e < 2 ? fa : fb) : fmaf(v, e < 2 ? fa : fb, s_acc[nb][e]);
                        }
                    }
                }
            }

            // ---- softmax in base 2 over the warp's keys
            uint32_t pb[NB][2];
            #pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                pb[nb][0] = pb[nb][1] = 0u;
                if (nb > 0 && !both) continue;
                float (&s)[4] = s_acc[nb];
                #pragma unroll
                for (int e = 0; e < 4; ++e) s[e] *= s_mul;
                if (kbase + 16 > wlim) {                               // warp-uniform
                    #pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (kbase + g + 8 * (e >> 1) >= lim[nb][e & 1]) s[e] = -INFINITY;
                }
                float mx[2] = {fmaxf(s[0], s[2]), fmaxf(s[1], s[3])};
                if (__any_sync(0xffffffffu, mx[0] > m_run[nb][0] || mx[1] > m_run[nb][1])) {
                    float corr[2];
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        #pragma unroll
                        for (int o = 4; o < 32; o <<= 1) mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], o));
                        corr[h] = 1.0f;
                        if (mx[h] > m_run[nb][h]) {
                            corr[h] = qd_ex2(m_run[nb][h] - mx[h]);
                            m_run[nb][h] = mx[h];
                        }
                        l_run[nb][h] *= corr[h];
                    }
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        o_acc[nb][i][0] *= corr[0]; o_acc[nb][i][2] *= corr[0];
                        o_acc[nb][i][1] *= corr[1]; o_acc[nb][i][3] *= corr[1];
                    }
                    cs[nb][0] *= corr[0]; cs[nb][1] *= corr[1];
                }
                const float r0m = m_run[nb][0] == -INFINITY ? 0.f : m_run[nb][0], r1m = m_run[nb][1] == -INFINITY ? 0.f : m_run[nb][1];
                const float e0 = qd_ex2(s[0] - r0m), e1 = qd_ex2(s[1] - r1m), e2 = qd_ex2(s[2] - r0m), e3 = qd_ex2(s[3] - r1m);
                l_run[nb][0] += e0 + e2; l_run[nb][1] += e1 + e3;
                // weights of (key g | g + 8, rows 2t, 2t+1), turned into the B operand (keys 2t, 2t+1 | + 8, row g)
                pb[nb][0] = qd_transpose(pack_h2(e0, e1));
                pb[nb][1] = qd_transpose(pack_h2(e2, e3));
            }

            // ---- the V scales of this lane's four keys (2t, 2t+1, 2t+8, 2t+9 of the warp's 16)
            uint2 sv4[4];
            #pragma unroll
            for (int i = 0; i < 4; ++i) sv4[i] = qd_lds64(sb + s_off + SM::SCALES + t * 32 + (i & 1) * 16 + (i >> 1) * 128);

            // ---- O^T += V^T (P^T * scale of the group), group by group
            const uint32_t va = sb + v_off;
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t x01[4], x89[4];                                // dims 32 j + 4 g + 0 .. 3, keys (2t, 2t+1) and (2t+8, 2t+9)
                if constexpr (B == 4) {
                    const uint32_t a = va ^ (j << 4);
                    const uint32_t w0 = qd_lds32(a), w1 = qd_lds32(a + SM::ROWB), w8 = qd_lds32(a + 8 * SM::ROWB), w9 = qd_lds32(a + 9 * SM::ROWB);
                    qd_pairs4_v(w0, w1, sel_lo, sel_hi, x01, cst);
                    qd_pairs4_v(w8, w9, sel_lo, sel_hi, x89, cst);
                } else {
                    const uint32_t a0 = va ^ (j << 5), a1 = va ^ (j << 5) ^ 16;
                    const uint32_t w0 = qd_lds32(a0), w1 = qd_lds32(a1 + SM::ROWB), w8 = qd_lds32(a0 + 8 * SM::ROWB), w9 = qd_lds32(a1 + 9 * SM::ROWB);
                    qd_pairs8_v(__byte_perm(w0, w1, 0x5410), x01[0], x01[1], cst);
                    qd_pairs8_v(__byte_perm(w0, w1, 0x7632), x01[2], x01[3], cst);
                    qd_pairs8_v(__byte_perm(w8, w9, 0x5410), x89[0], x89[1], cst);
                    qd_pairs8_v(__byte_perm(w8, w9, 0x7632), x89[2], x89[3], cst);
                    const half2 off = __float2half2_rn(639.5f);
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) {                       // 512 + n - 639.5 = n - 127.5, exact
                        const half2 a = __hsub2(*reinterpret_cast<const half2*>(&x01[i]), off), c2 = __hsub2(*reinterpret_cast<const half2*>(&x89[i]), off);
                        x01[i] = *reinterpret_cast<const uint32_t*>(&a); x89[i] = *reinterpret_cast<const uint32_t*>(&c2);
                    }
                }
                const uint32_t s01 = __byte_perm((j & 2) ? sv4[0].y : sv4[0].x, (j & 2) ? sv4[1].y : sv4[1].x, (j & 1) ? 0x7632 : 0x5410);
                const uint32_t s89 = __byte_perm((j & 2) ? sv4[2].y : sv4[2].x, (j & 2) ? sv4[3].y : sv4[3].x, (j & 1) ? 0x7632 : 0x5410);
                const uint32_t ones = g == j ? 0x3C003C00u : 0u;
                #pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    if (nb > 0 && !both) continue;
                    const uint32_t b0 = qd_hmul2(pb[nb][0], s01), b1 = qd_hmul2(pb[nb][1], s89);
                    mma_f16(o_acc[nb][2 * j], x01[0], x01[1], x89[0], x89[1], b0, b1);
                    mma_f16(o_acc[nb][2 * j + 1], x01[2], x01[3], x89[2], x89[3], b0, b1);
                    if constexpr (B == 4) mma_f16(cs[nb], ones, 0u, ones, 0u, b0, b1);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(done);
        }
        // all warps are done with the stages: the merge buffer may overwrite them
        if (__syncthreads_or(failed)) {
            if (tid == 0) atomicCAS(p.status, 0, 4);
            // no copy may land after the CTA has given its shared memory back (a wait for a phase that has passed returns)
            if (tid < SM::STAGES && s_asked[tid] < 2u) mbar_wait(&full[tid], s_asked[tid]);
            return;                                                    // uniform: every thread saw the same barrier result
        }

        // ---- merge the four key slices through shared memory: [warp][row][D + 4] fp32, columns D, D+1 = m, l
        float* ms = reinterpret_cast<float*>(smem);
        constexpr int MS = D + 4;
        #pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            float* mine = ms + (warp * ROWS + nb * 8 + 2 * t) * MS;
            #pragma unroll
            for (int j = 0; j < 4; ++j) {
                float c0 = 0.f, c1 = 0.f;
                if constexpr (B == 4) {                                // take the offset out
                    c0 = 23.5f * __shfl_sync(0xffffffffu, cs[nb][0], 4 * j + t);
                    c1 = 23.5f * __shfl_sync(0xffffffffu, cs[nb][1], 4 * j + t);
                }
                const float (&x)[4] = o_acc[nb][2 * j];
                const float (&y)[4] = o_acc[nb][2 * j + 1];
                *reinterpret_cast<float4*>(mine + 32 * j + 4 * g) = make_float4(x[0] - c0, x[2] - c0, y[0] - c0, y[2] - c0);
                *reinterpret_cast<float4*>(mine + MS + 32 * j + 4 * g) = make_float4(x[1] - c1, x[3] - c1, y[1] - c1, y[3] - c1);
            }
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                float l = l_run[nb][h];
                #pragma unroll
                for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
                if (g == 0) { mine[h * MS + D] = m_run[nb][h]; mine[h * MS + D + 1] = l; }
            }
        }
        __syncthreads();
        // one warp per output row; lane = (group lane / 8, values 4 (lane % 8) .. + 3) as in the cache codec
        for (int lr = warp; lr < ROWS; lr += 4) {
            const int row = r0 + lr;
            if (row >= ql * G) break;
            float mm = -INFINITY;
            #pragma unroll
            for (int w = 0; w < 4; ++w) mm = fmaxf(mm, ms[(w * ROWS + lr) * MS + D]);
            float ll = 0.f;
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            #pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float* src = ms + (w * ROWS + lr) * MS;
                const float mw = src[D];
                const float sc = (mw == -INFINITY) ? 0.f : qd_ex2(mw - mm);
                ll += src[D + 1] * sc;
                const float4 v = *reinterpret_cast<const float4*>(src + 4 * lane);
                acc[0] += v.x * sc; acc[1] += v.y * sc; acc[2] += v.z * sc; acc[3] += v.w * sc;
            }
            h4(acc[0], acc[1], acc[2], acc[3]);
            h8_lanes(acc[0], acc[1], acc[2], acc[3], lane);
            #pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] *= R32 / (float)(1 << (B - 1));
            const int qidx = row / G, head = kvh * G + (row - qidx * G);
            if (splits == 1) {
                const float inv = ll > 0.f ? 1.0f / ll : 0.f;
                half* op = p.o + ((size_t)(row_base + qidx) * p.nq + head) * D + lane * 4;
                *reinterpret_cast<uint2*>(op) = make_uint2(pack_h2(acc[0] * inv, acc[1] * inv), pack_h2(acc[2] * inv, acc[3] * inv));
            } else {
                float* pp = p.partial + (((size_t)item_idx * p.nkv + kvh) * ROWS + lr) * (D + 2);
                *reinterpret_cast<float2*>(pp + lane * 4) = make_float2(acc[0], acc[1]);
                *reinterpret_cast<float2*>(pp + lane * 4 + 2) = make_float2(acc[2], acc[3]);
                if (lane == 0) { pp[D] = mm; pp[D + 1] = ll; }
            }
        }
    }
}

}  // namespace exl3
