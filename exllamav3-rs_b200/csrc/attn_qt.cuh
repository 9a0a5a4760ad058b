// Paged attention over 4-bit and 8-bit quantised KV pools on tcgen05 (k_bits = v_bits, head_dim 128): the kernel behind
// exl3_bighead_attn_paged_q for verify batches and prefill rows (attn_impl in attn.cu says which).
// Reference semantics: kernels/attention.cu:97-269,1716-1870 with the cache codec of
// kernels/cache/q_cache_kernels.cuh:61-236 (a code c of a group of 32 rotated values stands for
// (c - (2^(B-1) - 1/2)) * scale / 2^(B-1)).
//
// A CTA works on tiles of 128 keys of one kv head for up to 40 packed (query, head) rows; two threads per key.
//  * S^T = K Q^T: a thread unpacks half of its key's codes, centred exactly in fp16, into its lane of tensor memory, where they are
//    the A operand; the rotated queries are the B operand.  One product per group of 32 dims, so that the group's scale is applied
//    to the fp32 sum by the thread that owns the key.
//  * Scores come back with the key on the lane: every lane works whatever the number of rows, and the key's scales are the
//    thread's own.  A row's maximum is looked for only when a score has left its reference behind (one barrier with a vote).
//  * O^T = V^T P^T: values (code x scale as an fp16 and what that rounding left over as another, so that a value is exact to 22
//    bits) and softmax weights (fp16) go to shared memory, with the key outermost, as a thread has them: no transposition.
// Codes are unpacked once for all rows of a block, where fragments of mma.sync operands were built again for every 16 rows
// (attn_qdec.cuh) or fp16 tiles for every 64 (attn_paged.cuh).  Two CTAs per SM hide each other's barriers and waits; a producer
// thread draws work units ahead and keeps the ring of code tiles full across units.
//
// What bounds it: latency.  Twelve sequences of 40 rows over contexts of 1024 .. 32768, profiled: 23 tiles per CTA, some 6600 cycles each
// with start and end, issue slots 57 % busy, 28 % of the warps an SM can hold, tensor pipe 18 %, DRAM 16 %; stalls of a warp per issued
// instruction: shared memory 1.5, fixed latencies 1.3, branches 0.7, tensor memory and global loads 0.6, barriers 0.5, instruction
// fetch 0.4.  On the way, us, 4 sequences of 40 rows, contexts 1024 .. 32768, whole call behind a work list of 8.7: one thread per
// key with products issued by a warp of keys 82, with an issuer 75, two threads per key 61, references left alone up to a factor of
// sqrt(2) 50, values to 22 bits 54 (the mma.sync kernel: 72).  Scales applied to the weights per group instead, which keeps codes exact
// with one rounding less, need four copies of the output: for up to 8 rows, three CTAs per SM, 64 sequences of 5 rows took 176 to 202 us
// (the mma.sync kernel: 142): not kept.
// Whole calls now, 4 bits, us: these 72 -> 43, 32 such sequences 435 -> 248, 4 of 500 rows 428 -> 366, at 8 bits 632 -> 565.
// Error against 64 bits: 40 rows, 4 bits 3.0e-4 -> 2.6e-4; 500 rows 4.8e-4 -> 4.2e-4, 8 bits 3.9e-4 -> 3.1e-4.  (With values rounded to
// one fp16 and weights to another it was 3.4e-4: the largest weight is exact, its value was not.)
// Every wait is bounded; a wait that runs out lets the others run out at once and sets the status word.
#pragma once
#include <cuda.h>
#include "attn_paged.cuh"
#include "attn_tc.cuh"

namespace exl3 {

constexpr int QT_TK = 128;                                 // keys per tile
constexpr int QT_WARPS = 8;                                // warps of keys: two threads per key
constexpr int QT_THREADS = (QT_WARPS + 2) * 32;            // then the producer of tiles and the issuer of products
// A row's weights are taken relative to a reference (base 2): the maximum of its first tile, moved to the maximum so far when a
// score exceeds it by this.  (Moved at once, it costs a fifth of the time.  From 2 on the error shows that the largest weights
// are no longer powers of two, which are exact.)
constexpr float QT_LAG = 0.5f;
constexpr uint32_t QT_POLLS = 1u << 22, QT_NS = 500;       // a wait gives up after about two seconds
constexpr int QT_ROWS = 40;                                // packed rows of a block (the products have 48 columns)
template <int B> struct QtSmem {
    static constexpr int NR = QT_ROWS;
    static constexpr int ROWB = 16 * B;                    // bytes of codes per key, head and plane
    static constexpr int CODES = QT_TK * ROWB;
    static constexpr int SLOT = CODES + QT_TK * 16;        // codes and scales (of two neighbouring heads) of the keys or the values of a tile
    static constexpr int SLOTS = B == 4 ? 2 : 1;           // what the other tiles leave room for
    static constexpr int VALUES = QT_TK * 256;             // two blocks of 64 dims: [key][128 bytes], 128-byte swizzle
    static constexpr int PROBS = QT_TK * 128;              // [key][rows], 128-byte swizzle
    static constexpr int QUERIES = NR * 256;               // two blocks of 64 dims: [row][128 bytes], 128-byte swizzle
    static constexpr int OFF_V = 0;
    static constexpr int OFF_P = OFF_V + 2 * VALUES;    // values, and what their rounding left over
    static constexpr int OFF_Q = OFF_P + PROBS;
    static constexpr int OFF_RING = OFF_Q + QUERIES;
    static constexpr int OFF_M = OFF_RING + SLOTS * SLOT;  // per row: minus its reference, the reference's last step, its correction
    static constexpr int OFF_UNIT = OFF_M + 3 * NR * 4;    // two work units
    static constexpr int OFF_BAR = OFF_UNIT + 2 * 64;
    static constexpr int N_BARS = 2 * SLOTS + 4 + 5;       // ring full / empty, unit full / empty [2], k_ready, s_full, p_ready, pv_done, drain
    static constexpr int BYTES = OFF_BAR + N_BARS * 8 + 1024;
    static_assert(BYTES + EXL3_TMEM_SMEM > EXL3_SM_SMEM, "not beside a GEMM that has yet to take tensor memory");
    static constexpr int OSTRIDE = 132;                    // floats per row of the output stage, in the value tile's place
    static_assert(NR * OSTRIDE * 4 <= VALUES && NR * 64 * 4 <= PROBS && SLOT % 512 == 0, "stage layout");
    // Tensor memory: codes 0..63, sums of the groups, output.  The sums of the last group take the place of the codes of the first
    // three, whose products the tensor core has executed by then.
    static constexpr int T_COLS = 256;
    static constexpr int t_s(int g) { return g < 3 ? 64 + g * 48 : 0; }
    static constexpr int T_O = 64 + 3 * 48;
    static_assert(T_O + 48 <= T_COLS && NR <= 48, "tensor memory");
};

// Bounded wait of one thread; one that runs out is seen by all others, which then stop waiting.
__device__ __forceinline__ bool qt_wait(uint64_t* bar, uint32_t parity, volatile int* failed)
{
    if (mbar_try_wait(bar, parity)) return true;
    for (uint32_t i = 0; i < QT_POLLS; ++i) {
        if (mbar_try_wait_hint(bar, parity, QT_NS)) return true;
        if (*failed) return false;
    }
    *failed = 1;
    return false;
}
// the same for a warp: one lane polls (32 lanes that poll take the barrier's port 32 times)
__device__ __forceinline__ void qt_wait_warp(uint64_t* bar, uint32_t parity, volatile int* failed)
{
    if ((threadIdx.x & 31) == 0) qt_wait(bar, parity, failed);
    __syncwarp();
}
__device__ __forceinline__ uint4 qt_lds128(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 qt_lds64(uint32_t a)
{
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
template <int OFF>
__device__ __forceinline__ void qt_sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    asm volatile("st.shared.v4.b32 [%0+%5], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w), "n"(OFF) : "memory");
}
__device__ __forceinline__ float qt_ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// maxima of eight rows over the warp: lane i holds that of row i % 8
__device__ __forceinline__ float qt_max8(const float* x, int lane)
{
    float y[8];
    #pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = x[i];
    #pragma unroll
    for (int s = 1; s < 8; s <<= 1)
        #pragma unroll
        for (int i = 0; i < 4 / s; ++i) {
            const float o = __shfl_xor_sync(0xffffffffu, (lane & s) ? y[2 * i] : y[2 * i + 1], s);
            y[i] = fmaxf((lane & s) ? y[2 * i + 1] : y[2 * i], o);
        }
    const float m = fmaxf(y[0], __shfl_xor_sync(0xffffffffu, y[0], 8));
    return fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
}
// eight columns of a lane of tensor memory
__device__ __forceinline__ void qt_ld8(uint32_t taddr, float* v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(taddr));
}
__device__ __forceinline__ void qt_st8(uint32_t taddr, const float* v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
}
// the warps of keys
__device__ __forceinline__ void qt_bar() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ bool qt_bar_or(bool x)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.aligned.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((uint32_t)x) : "memory");
    return r != 0;
}
__device__ __forceinline__ void qt_tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// A constant that stays in a register, so that (x & M) | E is one logic operation with one immediate.
__device__ __forceinline__ uint32_t qt_reg(uint32_t x)
{
    asm volatile("mov.b32 %0, %0;" : "+r"(x));
    return x;
}
__device__ __forceinline__ uint32_t qt_field(uint32_t x, uint32_t m, uint32_t e)      // (x & m) | e
{
    uint32_t y;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(y) : "r"(x), "r"(m), "r"(e));
    return y;
}
struct QtConst { uint32_t e16, e256, e512, x4, x2; };

// The fp16 pairs of a word of codes, centred exactly.  4 bits: (n_i - 7.5, n_{i+4} - 7.5), from 256 + n for even i and 16 + n for
// odd i, whose fp16 steps are fine enough; 8 bits: bytes (0, 2) and (1, 3) less 127.5, from 512 + n.  Left shifts are
// multiplications, which run beside the logic operations on another pipe.
template <int B>
__device__ __forceinline__ void qt_pairs(uint32_t w, uint32_t (&x)[B == 4 ? 4 : 2], const QtConst& c)
{
    if constexpr (B == 4) {
        const uint32_t l = w * c.x4, h = w >> 6;
        x[0] = qt_field(l, 0x003C003Cu, c.e256);
        x[1] = qt_field(l, 0x03C003C0u, c.e16);
        x[2] = qt_field(h, 0x003C003Cu, c.e256);
        x[3] = qt_field(h, 0x03C003C0u, c.e16);
        const half2 o256 = __float2half2_rn(263.5f), o16 = __float2half2_rn(23.5f);
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const half2 a = __hsub2(*reinterpret_cast<const half2*>(&x[i]), (i & 1) ? o16 : o256);
            x[i] = *reinterpret_cast<const uint32_t*>(&a);
        }
    } else {
        x[0] = qt_field(w * c.x2, 0x01FE01FEu, c.e512);
        x[1] = qt_field(w >> 7, 0x01FE01FEu, c.e512);
        const half2 off = __float2half2_rn(639.5f);
        #pragma unroll
        for (int i = 0; i < 2; ++i) {
            const half2 a = __hsub2(*reinterpret_cast<const half2*>(&x[i]), off);
            x[i] = *reinterpret_cast<const uint32_t*>(&a);
        }
    }
}
// the eight centred codes of chunk c (8 dims, 4 registers) of a key
template <int B>
__device__ __forceinline__ void qt_unpack(const uint32_t* w, uint32_t (&x)[4], const QtConst& cst)
{
    if constexpr (B == 4) qt_pairs<4>(w[0], x, cst);
    else {
        uint32_t a[2], b[2];
        qt_pairs<8>(w[0], a, cst);
        qt_pairs<8>(w[1], b, cst);
        x[0] = a[0]; x[1] = a[1]; x[2] = b[0]; x[3] = b[1];
    }
}
// dim that stands at position `pos` of a row of unpacked codes
template <int B>
__device__ __forceinline__ int qt_dim(int pos)
{
    return B == 4 ? (pos & ~7) + ((pos & 7) >> 1) + 4 * (pos & 1) : (pos & ~3) + ((pos & 3) >> 1) + 2 * (pos & 1);
}
__device__ __forceinline__ uint32_t qt_hmul2(uint32_t a, half2 b)
{
    const half2 r = __hmul2(*reinterpret_cast<const half2*>(&a), b);
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t qt_hfms2(uint32_t a, half2 b, uint32_t c)      // a b - c
{
    const half2 r = __hfma2(*reinterpret_cast<const half2*>(&a), b, __hneg2(*reinterpret_cast<const half2*>(&c)));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void qt_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]));
}

// a work unit, which the producer works out for all
struct QtUnit {
    int item, kvh, splits, row_base, r0, rows;             // item < 0: no more
    int k_begin, k_end, n_tiles;
    int lim0;                                              // keys that the block's first row sees
    int rem0;                                              // its head among its query's
    int b;
};
static_assert(sizeof(QtUnit) <= 64, "unit slots");
__device__ __forceinline__ QtUnit qt_unit(const AttnParams& p, int unit, int chunk, int G)
{
    QtUnit u;
    const AttnItem it = p.items[unit / p.nkv];
    const int ql = it.ql, total_k = it.total_k;
    u.item = it.idx; u.kvh = unit % p.nkv; u.b = it.b; u.row_base = it.row_base; u.splits = it.splits;
    u.r0 = it.rb * QT_ROWS;
    u.rows = min(QT_ROWS, ql * G - u.r0);
    const int q0 = u.r0 / G, i_last = min(ql - 1, (u.r0 + QT_ROWS - 1) / G);
    const int vis = p.causal ? min(total_k, total_k - ql + i_last + 1) : total_k;
    u.lim0 = p.causal ? total_k - ql + q0 + 1 : total_k; u.rem0 = u.r0 - q0 * G;
    u.k_begin = it.split * chunk;
    u.k_end = min(min(u.k_begin + chunk, total_k), vis);
    u.n_tiles = u.k_end > u.k_begin ? (u.k_end - u.k_begin + QT_TK - 1) / QT_TK : 0;
    return u;
}

template <int B>
__global__ void __launch_bounds__(QT_THREADS, 2)
attn_qt_kernel(const __grid_constant__ CUtensorMap map_qk, const __grid_constant__ CUtensorMap map_qv,
               const __grid_constant__ CUtensorMap map_sk, const __grid_constant__ CUtensorMap map_sv, const AttnParams p)
{
    using SM = QtSmem<B>;
    constexpr int D = 128, NR = SM::NR;
    extern __shared__ uint8_t qt_smem_unaligned[];
    uint8_t* smem = qt_smem_unaligned + ((1024u - (smem_u32(qt_smem_unaligned) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
    uint64_t* empty = full + SM::SLOTS;
    uint64_t* u_full = empty + SM::SLOTS;                  // [2]
    uint64_t* u_empty = u_full + 2;                        // [2]
    uint64_t* k_ready = u_empty + 2;
    uint64_t* s_full = k_ready + 1;
    uint64_t* p_ready = s_full + 1;
    uint64_t* pv_done = p_ready + 1;
    uint64_t* drain = pv_done + 1;
    float* s_nm = reinterpret_cast<float*>(smem + SM::OFF_M);                 // [NR] each
    float* s_step = s_nm + NR;
    float* s_corr = s_step + NR;
    uint8_t* s_unit = smem + SM::OFF_UNIT;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_failed;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_failed = 0;
        for (int i = 0; i < SM::SLOTS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], QT_WARPS); }
        for (int i = 0; i < 2; ++i) { mbar_init(&u_full[i], 1); mbar_init(&u_empty[i], QT_WARPS + 1); }
        mbar_init(k_ready, QT_WARPS); mbar_init(s_full, 1); mbar_init(p_ready, QT_WARPS); mbar_init(pv_done, 1); mbar_init(drain, 1);
        mbar_fence_init();
    }
    if (warp == QT_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(SM::T_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // behind the allocation: a kernel let go before it could take the tensor memory that this one waits for; and behind the wait, so
    // that the merge kernel finds the work list complete
    pdl_wait();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const int G = p.nq / p.nkv;
    volatile int* failed = &s_failed;
    int loads = 0;                                         // copies requested

    if (warp == QT_WARPS) {
        // ===== producer: draws units, one ahead of the keys' warps, and requests their tiles, keys and values in turn
        if (lane == 0) {
            const int chunk = p.plan->chunk, n_units = p.plan->n_items * p.nkv;
            uint32_t us = 0, upar = 1, slot = 0, par = 1;
            bool ok = true;
            for (int unit = blockIdx.y * gridDim.x + blockIdx.x; ok;) {
                QtUnit u;
                u.item = -1;
                if (unit < n_units) u = qt_unit(p, unit, chunk, G);
                if (!qt_wait(&u_empty[us], upar, failed)) break;
                *reinterpret_cast<QtUnit*>(s_unit + us * 64) = u;
                mbar_arrive(&u_full[us]);
                if (u.item < 0) break;
                if ((us ^= 1) == 0) upar ^= 1;
                const int32_t* bt = p.block_table + (size_t)u.b * p.pps;
                unit = gridDim.x * gridDim.y + atomicAdd(const_cast<int*>(&p.plan->next), 1);
                #pragma unroll 1
                for (int t = 0; t < 2 * u.n_tiles; ++t) {
                    const int k0 = u.k_begin + (t >> 1) * QT_TK;
                    const int tok = bt[k0 >> 8] * EXL3_PAGE + (k0 & 255);
                    if (!qt_wait(&empty[slot], par, failed)) { ok = false; break; }
                    const uint32_t dst = smem_u32(smem + SM::OFF_RING + slot * SM::SLOT), bar = smem_u32(&full[slot]);
                    mbar_expect_tx(&full[slot], SM::SLOT);
                    qt_tma_2d(dst, (t & 1) ? &map_qv : &map_qk, u.kvh * 4 * B, tok, bar);
                    qt_tma_2d(dst + SM::CODES, (t & 1) ? &map_sv : &map_sk, (u.kvh >> 1) * 8, tok, bar);
                    ++loads;
                    if (++slot == SM::SLOTS) { slot = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == QT_WARPS + 1) {
        // ===== issuer of the products (a thread that issues eight waits some hundred cycles for the last to be taken)
        if (lane == 0) {
            constexpr uint32_t HI = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);       // SBO 1024, version 1, SWIZZLE_128B
            const uint32_t base = smem_u32(smem), q_lo = ((base + SM::OFF_Q) >> 4) | (1u << 16);
            const uint32_t a_lo = ((base + SM::OFF_V) >> 4) | ((uint32_t)((QT_TK * 128) >> 4) << 16), b_lo = ((base + SM::OFF_P) >> 4) | (1u << 16);
            uint32_t us = 0, upar = 0, par = 0;
            bool ok = true;
            while (ok) {
                if (!qt_wait(&u_full[us], upar, failed)) break;
                const volatile QtUnit* u = reinterpret_cast<const volatile QtUnit*>(s_unit + us * 64);
                if (u->item < 0) break;
                const int n_tiles = u->n_tiles;
                const uint32_t n16 = (u->rows + 15) & ~15;
                mbar_arrive(&u_empty[us]);
                if ((us ^= 1) == 0) upar ^= 1;
                const uint32_t idesc_s = tc_idesc(n16, 128), idesc_o = idesc_s | (1u << 15) | (1u << 16);      // both operands with the key outermost
                #pragma unroll 1
                for (int t = 0; t < n_tiles; ++t, par ^= 1) {
                    if (!qt_wait(k_ready, par, failed)) { ok = false; break; }
                    tc_fence_after();
                    #pragma unroll
                    for (int g = 0; g < 4; ++g)
                        #pragma unroll
                        for (int h = 0; h < 2; ++h)
                            tc_mma_f16_ts(tmem + SM::t_s(g), tmem + g * 16 + h * 8,
                                          ((uint64_t)HI << 32) | (q_lo + (g >> 1) * (NR * 8) + (g & 1) * 4 + h * 2), idesc_s, h);
                    tc_commit(s_full);
                    if (!qt_wait(p_ready, par, failed)) { ok = false; break; }
                    tc_fence_after();
                    #pragma unroll
                    for (int kk = 0; kk < QT_TK / 16; ++kk)
                        tc_mma_f16(tmem + SM::T_O, ((uint64_t)HI << 32) | (a_lo + kk * (2048 >> 4)), ((uint64_t)HI << 32) | (b_lo + kk * (2048 >> 4)),
                                   idesc_o, t > 0 || kk > 0 ? 1u : 0u);
                    #pragma unroll
                    for (int kk = 0; kk < QT_TK / 16; ++kk)
                        tc_mma_f16(tmem + SM::T_O, ((uint64_t)HI << 32) | (a_lo + (SM::VALUES >> 4) + kk * (2048 >> 4)),
                                   ((uint64_t)HI << 32) | (b_lo + kk * (2048 >> 4)), idesc_o, 1u);
                    tc_commit(pv_done);
                }
            }
            if (*failed) { tc_commit(drain); mbar_wait(drain, 0); }
        }
        __syncwarp();
    } else {
        // ===== keys: thread = (key, half): two of the four groups of its codes, half of the rows of its scores
        const int quad = warp & 3, half_id = warp >> 2, key = quad * 32 + lane;
        constexpr int RT = 24;
        const int row0 = half_id * RT;                     // first of the thread's rows: 24, and what is left
        const uint32_t base = smem_u32(smem), lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const QtConst cst = {qt_reg(0x4C004C00u), qt_reg(0x5C005C00u), qt_reg(0x60006000u), qt_reg(4u), qt_reg(2u)};
        // this key's codes: chunk c of 16 bytes stands at c ^ swizzle
        const uint32_t k_off = base + SM::OFF_RING + key * SM::ROWB + (((B == 4 ? (key >> 1) & 3 : key & 7) ^ (half_id * (B / 2))) << 4);
        // rows of the value and weight tiles, likewise: chunk c at row ^ (c << 4); a thread's values are one block of 64 dims
        const uint32_t k_row = base + key * 128 + ((key & 7) << 4), v_row = k_row + SM::OFF_V + half_id * (QT_TK * 128), p_row = k_row + SM::OFF_P;
        uint32_t us = 0, upar = 0, slot = 0, par = 0, s_par = 0, pv_par = 0;
        for (;;) {
            qt_wait_warp(&u_full[us], upar, failed);
            if (qt_bar_or(*failed != 0)) break;            // all warps or none
            const volatile QtUnit& u = *reinterpret_cast<const volatile QtUnit*>(s_unit + us * 64);
            if (u.item < 0) break;
            const int n_tiles = u.n_tiles;
            const int rows = u.rows - row0;                // of this thread; may be none
            const half* q_base = p.q + ((size_t)u.row_base * p.nq + u.kvh * G) * D + lane * 4;
            const int r0 = u.r0;
            float l[RT];
            #pragma unroll
            for (int r = 0; r < RT; ++r) l[r] = 0.f;

            // ---- queries, rotated by H32 (q . H(c) = H(q) . c), are the B operand of the scores.  A group that lines up with a row of
            // the transform grows by sqrt(32) and would leave fp16 from 11580 on; a block that holds one over 11576 is packed at
            // an eighth, which keeps every finite one in range (46 318), and the scores are taken up again.
            float s_mul;
            {
                constexpr int RW = NR / QT_WARPS;          // rows warp, warp + 8, ...
                uint2 qx[RW];
                half2 qmax = __float2half2_rn(0.f);
                #pragma unroll
                for (int i = 0; i < RW; ++i) {
                    const int r = warp + QT_WARPS * i, row = r0 + r, qi = row / G;
                    qx[i] = make_uint2(0u, 0u);
                    if (r < rows + row0) qx[i] = *reinterpret_cast<const uint2*>(q_base + ((size_t)qi * (p.nq - G) + row) * D);
                }
                #pragma unroll
                for (int i = 0; i < RW; ++i)
                    qmax = __hmax2(qmax, __hmax2(__habs2(*reinterpret_cast<const half2*>(&qx[i].x)), __habs2(*reinterpret_cast<const half2*>(&qx[i].y))));
                const bool big = qt_bar_or(fmaxf(__low2float(qmax), __high2float(qmax)) > 11576.f);
                const float q_mul = big ? 0.125f * R32 : R32;
                s_mul = p.scale_log2 * (big ? 8.f / (float)(1 << (B - 1)) : 1.f / (float)(1 << (B - 1)));
                // dims 4 lane .. + 3 go to their positions among the unpacked codes: 16-byte chunk lane / 2 of the row
                uint8_t* dst = smem + SM::OFF_Q + (lane >> 4) * (NR * 128) + warp * 128 + ((((lane >> 1) & 7) ^ (warp & 7)) << 4) + (lane & 1) * 8;
                #pragma unroll 1
                for (int i = 0; i < RW; ++i, dst += QT_WARPS * 128) {
                    const half2 a = *reinterpret_cast<const half2*>(&qx[0].x), b = *reinterpret_cast<const half2*>(&qx[0].y);
                    #pragma unroll
                    for (int j = 0; j + 1 < RW; ++j) qx[j] = qx[j + 1];
                    float v0 = __low2float(a), v1 = __high2float(a), v2 = __low2float(b), v3 = __high2float(b);
                    h4(v0, v1, v2, v3);
                    h8_lanes(v0, v1, v2, v3, lane);
                    v0 *= q_mul; v1 *= q_mul; v2 *= q_mul; v3 *= q_mul;
                    uint2 o;
                    if constexpr (B == 4) {                // pairs (n_i, n_{i+4}) of dims 8 w .. + 7: two lanes make two each
                        const uint32_t lo = pack_h2(v0, v1), hi = pack_h2(v2, v3);
                        const uint32_t other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? lo : hi, 1);
                        const uint32_t first = (lane & 1) ? other : lo, second = (lane & 1) ? hi : other;
                        o = make_uint2(__byte_perm(first, second, 0x5410), __byte_perm(first, second, 0x7632));
                    } else o = make_uint2(pack_h2(v0, v2), pack_h2(v1, v3));
                    *reinterpret_cast<uint2*>(dst) = o;
                }
                fence_proxy_async();
            }

            #pragma unroll 1
            for (int t = 0, kbase = u.k_begin; t < n_tiles; ++t, kbase += QT_TK) {
                constexpr int NW = B / 2;                  // 16-byte chunks of codes per thread
                float ks[4];
                uint32_t w[4 * NW];
                auto fetch = [&]() -> uint2 {              // the thread's codes and its key's scales from the next slot
                    qt_wait_warp(&full[slot], par, failed);
                    const uint32_t row = k_off + slot * SM::SLOT;
                    #pragma unroll
                    for (int c = 0; c < NW; ++c) {
                        const uint4 v = qt_lds128(row ^ (c << 4));
                        w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
                    }
                    return qt_lds64(base + SM::OFF_RING + slot * SM::SLOT + SM::CODES + key * 16 + (u.kvh & 1) * 8);
                };
                auto release = [&]() { if (++slot == SM::SLOTS) { slot = 0; par ^= 1; } };
                // ---- keys -> tensor memory
                {
                    const uint2 sc = fetch();
                    #pragma unroll
                    for (int j = 0; j < 2; ++j) {          // a group: 32 codes, 16 columns
                        uint32_t x[16];
                        #pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            uint32_t y[4];
                            qt_unpack<B>(w + (4 * j + c) * (B / 4), y, cst);
                            x[4 * c] = y[0]; x[4 * c + 1] = y[1]; x[4 * c + 2] = y[2]; x[4 * c + 3] = y[3];
                        }
                        qt_st16(lanes + (half_id * 2 + j) * 16, x);
                    }
                    const half2 s01 = *reinterpret_cast<const half2*>(&sc.x), s23 = *reinterpret_cast<const half2*>(&sc.y);
                    ks[0] = __low2float(s01) * s_mul; ks[1] = __high2float(s01) * s_mul;
                    ks[2] = __low2float(s23) * s_mul; ks[3] = __high2float(s23) * s_mul;
                    tc_wait_st_acc();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) { mbar_arrive(k_ready); mbar_arrive(&empty[slot]); }
                    release();
                }
                // ---- values -> shared memory, under the products of the scores.  Large scales are taken down by a power of two, the
                // key's weights up by it, so that no value leaves fp16.
                bool down;
                {
                    uint2 sc = fetch();
                    if (kbase + key >= u.k_end) sc = make_uint2(0u, 0u);               // rows of the page past the sequence hold any bits
                    half2 sv[2] = {*reinterpret_cast<const half2*>(&sc.x), *reinterpret_cast<const half2*>(&sc.y)};
                    const half2 top = __hmax2(__habs2(sv[0]), __habs2(sv[1]));
                    down = __hmax(__low2half(top), __high2half(top)) > __float2half(B == 4 ? 4096.f : 256.f);
                    half2 mine = half_id ? sv[1] : sv[0];
                    if (down) mine = __hmul2(mine, __float2half2_rn(B == 4 ? 0.125f : 1.f / 256.f));
                    if (t > 0) { qt_wait_warp(pv_done, pv_par, failed); pv_par ^= 1; }         // the last tile's product has read its operands
                    #pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const half2 s = j ? __high2half2(mine) : __low2half2(mine);
                        #pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            uint32_t y[4];
                            qt_unpack<B>(w + (4 * j + c) * (B / 4), y, cst);
                            uint32_t v[4];
                            #pragma unroll
                            for (int i = 0; i < 4; ++i) v[i] = qt_hmul2(y[i], s);
                            qt_sts128<0>(v_row ^ ((j * 4 + c) << 4), v[0], v[1], v[2], v[3]);
                            #pragma unroll
                            for (int i = 0; i < 4; ++i) v[i] = qt_hfms2(y[i], s, v[i]);
                            qt_sts128<SM::VALUES>(v_row ^ ((j * 4 + c) << 4), v[0], v[1], v[2], v[3]);
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[slot]);
                    release();
                }
                // ---- scores less the rows' references, base 2
                float x[RT], top = -INFINITY;
                qt_wait_warp(s_full, s_par, failed);
                s_par ^= 1;
                tc_fence_after();
                const bool masked = kbase + QT_TK > min(u.lim0, u.k_end);          // the same for all threads
                #pragma unroll
                for (int r = 0; r < RT; r += 8) {
                    if (r < rows) {
                        #pragma unroll
                        for (int i = 0; i < 8; i += 4) {
                            const float4 m = t > 0 ? *reinterpret_cast<const float4*>(s_nm + row0 + r + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                            x[r + i] = m.x; x[r + i + 1] = m.y; x[r + i + 2] = m.z; x[r + i + 3] = m.w;
                        }
                        #pragma unroll
                        for (int g = 0; g < 4; g += 2) {
                            float s[2][8];
                            qt_ld8(lanes + SM::t_s(g) + row0 + r, s[0]);
                            qt_ld8(lanes + SM::t_s(g + 1) + row0 + r, s[1]);
                            tc_wait_ld();
                            #pragma unroll
                            for (int h = 0; h < 2; ++h)
                                #pragma unroll
                                for (int i = 0; i < 8; ++i) x[r + i] = fmaf(s[h][i], ks[g + h], x[r + i]);
                        }
                        if (masked) {
                            const int left = u.lim0 - (kbase + key), rem = u.rem0 + row0 + r;  // left > 0: the block's first row sees the key
                            const bool valid = kbase + key < u.k_end;
                            #pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                // rows of one query see the same keys; (rem0 + row) / G for sums below 64
                                const int qd = p.causal ? ((rem + i) * ((65536 + G - 1) / G)) >> 16 : 0;
                                if (!valid || left + qd <= 0) x[r + i] = -INFINITY;
                            }
                        }
                        // (rows behind the block's last have queries of zeros and never exceed their reference of 0)
                        #pragma unroll
                        for (int i = 0; i < 8; i += 2) top = fmaxf(top, fmaxf(x[r + i], x[r + i + 1]));
                    }
                }
                if (qt_bar_or(t == 0 || top > QT_LAG)) {
                    // the first tile, or some row's reference has been left behind.  Maxima of the quadrants' keys per row, where the
                    // weights of this tile will stand
                    float* s_max = reinterpret_cast<float*>(smem + SM::OFF_P);         // [NR][4]
                    #pragma unroll
                    for (int r = 0; r < RT; r += 8)
                        if (r < rows) {
                            const float m = qt_max8(&x[r], lane);
                            if (lane < 8) s_max[(row0 + r + lane) * 4 + quad] = m;
                        }
                    qt_bar();
                    if (tid < NR) {                                            // a thread per row
                        const float4 v = reinterpret_cast<const float4*>(s_max)[tid];
                        float d = fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w));
                        // the first tile sets the reference, which is 0 for a row that sees none of its keys (and none behind it)
                        d = t == 0 ? (d == -INFINITY ? 0.f : d) : fmaxf(d, 0.f);
                        s_nm[tid] = (t == 0 ? 0.f : s_nm[tid]) - d;
                        s_step[tid] = d;
                        s_corr[tid] = qt_ex2(-d);
                    }
                    qt_bar();
                    #pragma unroll
                    for (int r = 0; r < RT; r += 8)
                        if (r < rows) {
                            #pragma unroll
                            for (int i = 0; i < 8; ++i) x[r + i] -= s_step[row0 + r + i];
                            if (t > 0) {
                                float o[8];
                                qt_ld8(lanes + SM::T_O + row0 + r, o);
                                tc_wait_ld();
                                #pragma unroll
                                for (int i = 0; i < 8; ++i) { const float c = s_corr[row0 + r + i]; o[i] *= c; l[r + i] *= c; }
                                qt_st8(lanes + SM::T_O + row0 + r, o);
                            }
                        }
                    if (t > 0) tc_wait_st_acc();
                }
                // ---- weights -> shared memory
                const float up = down ? (B == 4 ? 8.f : 256.f) : 1.f;
                const bool any_down = __any_sync(0xffffffffu, down);
                #pragma unroll
                for (int r = 0; r < RT; r += 8) {
                    if (r < rows) {
                        float e[8];
                        #pragma unroll
                        for (int i = 0; i < 8; ++i) { e[i] = qt_ex2(x[r + i]); l[r + i] += e[i]; }
                        if (any_down) {
                            #pragma unroll
                            for (int i = 0; i < 8; ++i) e[i] *= up;
                        }
                        qt_sts128<0>(p_row ^ (((row0 + r) >> 3) << 4), pack_h2(e[0], e[1]), pack_h2(e[2], e[3]), pack_h2(e[4], e[5]), pack_h2(e[6], e[7]));
                    }
                }
                fence_proxy_async();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready);
            }
            // ===== end of the unit: output and sums through shared memory, then a warp per row
            float* stage = reinterpret_cast<float*>(smem + SM::OFF_V);          // [row][OSTRIDE], dims in order
            float* sums = reinterpret_cast<float*>(smem + SM::OFF_P);           // [row][64]
            if (n_tiles > 0) { qt_wait_warp(pv_done, pv_par, failed); pv_par ^= 1; }
            tc_fence_after();
            const int dim = qt_dim<B>(key);
            #pragma unroll
            for (int r = 0; r < RT; r += 8) {
                if (r < rows) {
                    float o[8];
                    qt_ld8(lanes + SM::T_O + row0 + r, o);
                    tc_wait_ld();
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        stage[(row0 + r + i) * SM::OSTRIDE + dim] = n_tiles > 0 ? o[i] : 0.f;
                        l[r + i] += __shfl_xor_sync(0xffffffffu, l[r + i], 16);
                        if (lane < 16) sums[(row0 + r + i) * 64 + quad * 16 + lane] = l[r + i];
                    }
                }
            }
            tc_fence_before();
            qt_bar();
            #pragma unroll 1
            for (int lr = warp; lr < rows + row0; lr += QT_WARPS) {
                const float2 ls = *reinterpret_cast<const float2*>(sums + lr * 64 + 2 * lane);
                const float4 v = *reinterpret_cast<const float4*>(stage + lr * SM::OSTRIDE + 4 * lane);
                float ll = ls.x + ls.y, a0 = v.x, a1 = v.y, a2 = v.z, a3 = v.w;
                #pragma unroll
                for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, o);
                h4(a0, a1, a2, a3);
                h8_lanes(a0, a1, a2, a3, lane);
                constexpr float f = R32 / (float)(1 << (B - 1));
                if (u.splits == 1) {
                    const int row = r0 + lr, qi = row / G;
                    const float inv = (ll > 0.f ? 1.0f / ll : 0.f) * f;
                    half* op = p.o + ((size_t)u.row_base * p.nq + u.kvh * G + (size_t)qi * (p.nq - G) + row) * D + lane * 4;
                    *reinterpret_cast<uint2*>(op) = make_uint2(pack_h2(a0 * inv, a1 * inv), pack_h2(a2 * inv, a3 * inv));
                } else {
                    float* pp = p.partial + (((size_t)u.item * p.nkv + u.kvh) * NR + lr) * (D + 2);
                    *reinterpret_cast<float2*>(pp + lane * 4) = make_float2(a0 * f, a1 * f);
                    *reinterpret_cast<float2*>(pp + lane * 4 + 2) = make_float2(a2 * f, a3 * f);
                    if (lane == 0) { pp[D] = ll > 0.f ? -s_nm[lr] : -INFINITY; pp[D + 1] = ll; }
                }
            }
            // (the next unit's first barrier stands between these reads and what overwrites them)
            __syncwarp();
            if (lane == 0) mbar_arrive(&u_empty[us]);
            if ((us ^= 1) == 0) upar ^= 1;
        }
    }

    // ===== tear-down.  A CTA that gave up waits, within a bound, for its copies in flight (a wait for a phase that has passed
    // returns at once); the issuer has waited for its products.
    tc_fence_before();
    __syncthreads();
    if (s_failed && tid == QT_WARPS * 32)
        for (int i = loads > SM::SLOTS ? loads - SM::SLOTS : 0; i < loads; ++i) mbar_wait(&full[i % SM::SLOTS], (i / SM::SLOTS) & 1);
    __syncthreads();
    if (warp == QT_WARPS + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(SM::T_COLS) : "memory");
    }
    if (tid == 0 && s_failed) atomicCAS(p.status, 0, 4);
}

}  // namespace exl3
