// What stands in front of an attention kernel: the work list, and the append of the call's new keys and values to the pools.  Neither
// needs the other, so they are one launch: block 0 plans while the other blocks append.
//
// What bounds it: latency.  The list is one block's work on a few hundred numbers, so every load that waits for another and every
// barrier counts.  A sequence's numbers are loaded once and kept in shared memory, sums are shuffles and one barrier, an item is
// found by a search over the sequences' first items and written once, in its final place, with all that a kernel needs to begin
// (attn_paged.cuh).  Against a list built by one thread per sequence, sorted through global memory, behind an append of its own, us
// per call: 24 sequences over 8-bit pools 64.1 -> 57.8, 64 over 4-bit ones 141.5 -> 136.5, over fp16 281.2 -> 279.6, 4 x 256 rows
// over fp16 136.2 -> 133.8 (the last with the attention kernel a programmatic dependent too).
#pragma once
#include "attn_paged.cuh"

namespace exl3 {

constexpr int AP_THREADS = 1024;

struct AttnPlanArgs {
    const int32_t* seqlens; const int32_t* cu_q;
    AttnPlan* plan; AttnItem* items; int* seq_base; int* seq_splits; int* status;
    int bsz, q_len, kv_append, G, rows_per_cta;
    int rows_lo, rows_hi;              // only sequences with packed row counts in (rows_lo, rows_hi] get work items
    int chunk_mult, target_items, max_items;
    int causal;                        // < 0: A/B switch, the list stays in plan order
    int slots;
};
// new keys and values of a call: fp16 pools, or codes and scales (bits > 0)
struct AttnAppendArgs {
    const half* k; const half* v;
    half* kc; half* vc;
    uint32_t* qk; half* sk; uint32_t* qv; half* sv;
    const int32_t* block_table; const int32_t* seqlens; const int32_t* cu_q;
    int bsz, seq, rows, nkv, pages, pps, k_bits, v_bits;     // rows: packed rows, or bsz * seq
};

// sum of v over the block; buf: 32 entries of its own per use
__device__ __forceinline__ long long ap_sum(long long v, long long* buf)
{
    const int lane = threadIdx.x & 31;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) buf[threadIdx.x >> 5] = v;
    __syncthreads();
    v = buf[lane];
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// exclusive scan over the block and its total; buf: 32 entries of its own per use
__device__ __forceinline__ int ap_scan(int v, int* buf, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, own = v;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
    if (lane == 31) buf[warp] = v;
    __syncthreads();
    int w = buf[lane];
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += u; }
    total = __shfl_sync(0xffffffffu, w, 31);
    const int before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    return v - own + (warp > 0 ? before : 0);
}

// Builds the split-KV work list from the REAL sequence lengths (one block; bsz is small next to the KV walk).
// Each sequence gets ceil(total_k / chunk) splits per row block, with chunk sized so that the list has about
// `target_items` entries; the reference sizes its splits from the padded block-table width instead
// (kernels/attention.cu:1805), which launches empty CTAs for the short sequences of a ragged batch.
__device__ __forceinline__ void attn_plan_block(const AttnPlanArgs& a)
{
    __shared__ long long s_sum[2][32];
    __shared__ int s_warp[3][32];
    __shared__ int s_bin[1024], s_cursor[1024];
    __shared__ int s_base[1024], s_sp[1024], s_ql[1024], s_tk[1024], s_row[1024];
    const int tid = threadIdx.x;
    s_bin[tid] = 0; s_cursor[tid] = 0;

    struct Seq { int ql, tk, row, rb; };
    auto load = [&](int b) -> Seq {
        Seq s;
        s.row = a.cu_q ? a.cu_q[b] : b * a.q_len;
        s.ql = a.cu_q ? a.cu_q[b + 1] - s.row : a.q_len;
        s.tk = (a.seqlens ? a.seqlens[b] : 0) + (a.cu_q ? s.ql : a.kv_append);
        const int pr = s.ql * a.G;
        s.rb = (pr > a.rows_lo && pr <= a.rows_hi) ? (pr + a.rows_per_cta - 1) / a.rows_per_cta : 0;
        return s;
    };
    Seq mine = {0, 0, 0, 0};                               // of sequence tid
    if (tid < a.bsz) mine = load(tid);
    long long local = (long long)mine.tk * mine.rb;
    for (int b = tid + 1024; b < a.bsz; b += 1024) { const Seq s = load(b); local += (long long)s.tk * s.rb; }
    const long long total = ap_sum(local, s_sum[0]);
    // Keys per split: total work / target_items.  slots > 0 (kernels whose CTAs are whole items, target_items = two per CTA
    // slot): one item per slot instead when that already gives two or more items per slot, because every row block and
    // every sequence rounds its split count up.  Then the longest-first order balances the slots and fewer items save the
    // fixed cost of a CTA and the partials (four 256-row chunks: 125 us at one item per slot, 135 at two, 150 at three; 32
    // x 8 verify rows: 125 against 133 us), while a batch of few long items (one 256-row chunk over 32768 keys: 20 items
    // on 18 slots) keeps the finer split.
    auto chunk_for = [&](int t) -> int {
        long long c = total < (1LL << 31) - t ? (long long)(((unsigned)total + t - 1) / (unsigned)t) : (total + t - 1) / t;
        if (c > (1 << 30)) return 1 << 30;
        const int r = ((int)c + a.chunk_mult - 1) / a.chunk_mult * a.chunk_mult;      // splits start on a key-tile boundary of the kernel
        return r < 256 ? 256 : r;
    };
    int chunk = chunk_for(a.slots > 0 ? a.slots : a.target_items);
    auto splits = [&](const Seq& s) -> int { return (s.rb > 0 && s.tk > 0) ? (s.tk + chunk - 1) / chunk : 1; };
    if (a.slots > 0) {
        long long cnt = (long long)mine.rb * splits(mine);
        for (int b = tid + 1024; b < a.bsz; b += 1024) { const Seq s = load(b); cnt += (long long)s.rb * splits(s); }
        if (ap_sum(cnt, s_sum[1]) < 2LL * a.slots) chunk = chunk_for(a.target_items);
    }
    int n = 0;                                             // items so far
    for (int b0 = 0; b0 < a.bsz; b0 += 1024) {
        const int b = b0 + tid;
        Seq s = mine;
        if (b0 > 0) { s = {0, 0, 0, 0}; if (b < a.bsz) s = load(b); }
        const int sp = b < a.bsz ? splits(s) : 1;
        int sum;
        const int base = n + ap_scan(s.rb * sp, s_warp[(b0 >> 10) & 1], sum);
        if (b < a.bsz) { a.seq_base[b] = base; a.seq_splits[b] = sp; }
        if (b0 == 0) { s_base[tid] = base; s_sp[tid] = sp; s_ql[tid] = s.ql; s_tk[tid] = s.tk; s_row[tid] = s.row; }
        n += sum;
    }
    __syncthreads();
    // Launch order: longest items first (counting sort by key tiles, most first).  Items differ in length - last splits,
    // causal cuts, short sequences - and a long one started late leaves the other SMs idle at the end of the kernel
    // (four 256-row chunks: a quarter of the SM time).
    const int n_items = n < a.max_items ? n : a.max_items;
    const bool small = a.bsz <= 1024;
    auto item = [&](int i, int& key) -> AttnItem {
        int lo = 0, hi = a.bsz - 1;                        // last sequence whose first item is not behind i
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((small ? s_base[mid] : a.seq_base[mid]) <= i) lo = mid; else hi = mid - 1;
        }
        AttnItem it;
        it.b = lo; it.idx = i;
        if (small) { it.ql = s_ql[lo]; it.total_k = s_tk[lo]; it.row_base = s_row[lo]; it.splits = s_sp[lo]; i -= s_base[lo]; }
        else { const Seq s = load(lo); it.ql = s.ql; it.total_k = s.tk; it.row_base = s.row; it.splits = a.seq_splits[lo]; i -= a.seq_base[lo]; }
        it.rb = i / it.splits; it.split = i - it.rb * it.splits;
        const int i_last = min(it.ql - 1, (it.rb * a.rows_per_cta + a.rows_per_cta - 1) / a.G);
        const int vis = a.causal > 0 ? min(it.total_k, it.total_k - it.ql + i_last + 1) : it.total_k;
        const int k_begin = it.split * chunk, k_end = min(min(k_begin + chunk, it.total_k), vis);
        key = k_end > k_begin ? (k_end - k_begin + a.chunk_mult - 1) / a.chunk_mult : 0;
        key = 1023 - min(key, 1023);                       // bin 0 = longest
        return it;
    };
    AttnItem first;                                        // item tid; others are worked out twice
    int first_key = 0;
    for (int i = tid; i < n_items; i += 1024) {
        int key;
        const AttnItem it = item(i, key);
        if (i == tid) { first = it; first_key = key; }
        atomicAdd(&s_bin[key], 1);
    }
    __syncthreads();
    int all;
    const int before = ap_scan(s_bin[tid], s_warp[2], all);
    s_bin[tid] = before;                                   // first position of bin tid (every thread has read its own count)
    __syncthreads();
    for (int i = tid; i < n_items; i += 1024) {
        int key = first_key;
        const AttnItem it = i == tid ? first : item(i, key);
        a.items[a.causal < 0 ? i : s_bin[key] + atomicAdd(&s_cursor[key], 1)] = it;
    }
    if (tid == 0) {
        a.plan->n_items = n_items;
        a.plan->next = 0;
        a.plan->chunk = chunk;
        // the host sizes the list from bounds on the batch; a list that does not fit would silently drop work, so it is
        // reported through the status word like a device-side wait that ran out
        if (n > a.max_items) atomicExch(a.status, 3);
    }
}

// A warp appends a token's row: of fp16 pools all of it, of quantised ones 4 groups of 32 values.
__device__ __forceinline__ void attn_append_warp(const AttnAppendArgs& a, long long w)
{
    const int lane = threadIdx.x & 31, groups = a.nkv * 4, quads = a.k_bits ? (groups + 3) >> 2 : 1;
    const long long r64 = w / quads;
    if (r64 >= a.rows) return;
    const int row = (int)r64, g0 = (int)(w - r64 * quads) * 4;
    int b, s;
    if (a.cu_q) {
        // cu_q[b] <= row < cu_q[b + 1]: the lanes probe the range side by side
        int lo = 0, hi = a.bsz;
        while (hi - lo > 1) {
            const int step = (hi - lo + 31) >> 5, at = lo + lane * step;
            const unsigned below = __ballot_sync(0xffffffffu, at < hi && a.cu_q[at] <= row);
            if (below == 0) return;                        // in front of the first sequence
            lo += (31 - __clz(below)) * step;
            hi = min(hi, lo + step);
        }
        b = lo; s = row - a.cu_q[b];
        if (s < 0 || row >= a.cu_q[b + 1]) return;         // rows behind the last sequence go nowhere
    } else { b = row / a.seq; s = row - b * a.seq; }
    if (s >= a.seq) return;
    const int pos = a.seqlens[b] + s, lp = pos >> 8;
    if (lp >= a.pps) return;
    const int page = a.block_table[(size_t)b * a.pps + lp];
    if (page < 0 || page >= a.pages) return;
    const size_t tok = (size_t)page * EXL3_PAGE + (pos & 255);
    if (a.k_bits == 0) {
        const int chunks = a.nkv * 16;
        const uint4 *k = reinterpret_cast<const uint4*>(a.k) + (size_t)row * chunks, *v = reinterpret_cast<const uint4*>(a.v) + (size_t)row * chunks;
        uint4 *kc = reinterpret_cast<uint4*>(a.kc) + tok * chunks, *vc = reinterpret_cast<uint4*>(a.vc) + tok * chunks;
        #pragma unroll 4
        for (int c = lane; c < chunks; c += 32) { kc[c] = k[c]; vc[c] = v[c]; }
    } else {
        const int active = min(4, groups - g0);
        const size_t base = tok * groups + g0, in = ((size_t)row * groups + g0) * 32;
        quant_x4(a.k + in, a.qk + base * a.k_bits, a.sk + base, active, a.k_bits);
        quant_x4(a.v + in, a.qv + base * a.v_bits, a.sv + base, active, a.v_bits);
    }
}

// the list alone
__global__ void __launch_bounds__(AP_THREADS) attn_plan_kernel(const AttnPlanArgs a)
{
    pdl_enter();
    attn_plan_block(a);
}
// the first kernel of a call (exl3_launch_first): block 0 plans, the others append, a warp per row or per 4 groups of one
__global__ void __launch_bounds__(AP_THREADS) attn_front_kernel(const AttnPlanArgs a, const AttnAppendArgs ap, int early)
{
    pdl_enter_first(early);
    if (blockIdx.x == 0) attn_plan_block(a);
    else attn_append_warp(ap, (long long)(blockIdx.x - 1) * (AP_THREADS / 32) + (threadIdx.x >> 5));
}

}  // namespace exl3
