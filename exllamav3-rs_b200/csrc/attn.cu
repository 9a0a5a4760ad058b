// exl3_bighead_attn_paged / exl3_bighead_attn_paged_q: planning, launch and split-KV combine.
#include <algorithm>
#include "attn_front.cuh"
#include "attn_tc.cuh"
#include "attn_tc2.cuh"
#include "attn_qdec.cuh"
#include "attn_qt.cuh"

namespace {

using namespace exl3;

// Merges the split-KV partials of one output row (b, query, head); one warp per row, lane = D/32 dims.
// HAD: also writes the 128-point transform of (output o signs).  (A form of its own: with the test at run time in every call 24
// sequences over 8-bit pools took 67.3 us instead of 65.4.)
template <int D, bool HAD>
__global__ void __launch_bounds__(256) attn_combine_kernel(const AttnParams p, int rows_per_cta, int total_rows, const half* had_suh, half* had_out)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    uint2 sg = make_uint2(0u, 0u);                             // signs do not depend on the kernels in front
    if constexpr (HAD) sg = reinterpret_cast<const uint2*>(had_suh)[(int)(w % p.nq) * 32 + lane];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // the attention kernel in front has handed out all its units: the work list is ready for the next layer's
    if (blockIdx.x == 0 && threadIdx.x == 0) const_cast<AttnPlan*>(p.plan)->next = 0;
    if (w >= (long long)total_rows * p.nq) return;
    const int row = (int)(w / p.nq), head = (int)(w % p.nq);
    int b;
    if (p.cu_q) {                                              // binary search: cu_q[b] <= row < cu_q[b+1]
        int lo = 0, hi = p.bsz - 1;
        while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (p.cu_q[mid] <= row) lo = mid; else hi = mid - 1; }
        b = lo;
        if (row >= p.cu_q[b + 1]) return;                      // rows behind the last sequence have no partials
    } else b = row / p.q_len;
    const int splits = p.seq_splits[b];
    // the input transform of the projection behind the attention: a head is one 128-block of its k
    auto transform = [&](uint2 v) {
        reinterpret_cast<uint2*>(had_out)[((size_t)row * p.nq + head) * 32 + lane] =
            had128_signed_lane(*reinterpret_cast<const half2*>(&v.x), *reinterpret_cast<const half2*>(&v.y), sg, lane);
    };
    if (splits <= 1) {                                         // the attention kernel wrote the final value itself
        if constexpr (HAD) transform(*reinterpret_cast<const uint2*>(p.o + ((size_t)row * p.nq + head) * D + lane * (D / 32)));
        return;
    }
    const int row_base = p.cu_q ? p.cu_q[b] : b * p.q_len;
    const int G = p.nq / p.nkv, kvh = head / G;
    const int packed = (row - row_base) * G + (head - kvh * G);
    const int rb = packed / rows_per_cta, lr = packed - rb * rows_per_cta;
    const int item0 = p.seq_base[b] + rb * splits;
    // A sequence of a small batch can have dozens of splits; walked one after the other by every lane their loads form
    // one long dependent chain (53 us per launch on 4 verify sequences).  So the lanes take the splits' maxima and sums
    // side by side, and the rows themselves are fetched four splits at a time.
    static_assert(D == 128, "a lane covers 4 dims as two 8-byte loads");
    const size_t stride = (size_t)p.nkv * rows_per_cta * (D + 2);             // floats between consecutive splits
    const float* base = p.partial + (((size_t)item0 * p.nkv + kvh) * rows_per_cta + lr) * (D + 2);
    float mm = -INFINITY;
    for (int s0 = 0; s0 < splits; s0 += 32) {
        const int s = s0 + lane;
        if (s < splits) mm = fmaxf(mm, base[(size_t)s * stride + D]);
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    float acc[D / 32], ll = 0.f;
    #pragma unroll
    for (int e = 0; e < D / 32; ++e) acc[e] = 0.f;
    for (int s0 = 0; s0 < splits; s0 += 32) {
        const int s = s0 + lane;
        float sc_l = 0.f;
        if (s < splits) {
            const float ms = base[(size_t)s * stride + D];
            sc_l = (ms == -INFINITY) ? 0.f : exp2f(ms - mm);
            ll += base[(size_t)s * stride + D + 1] * sc_l;
        }
        const int cnt = min(32, splits - s0);
        #pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const float sc = __shfl_sync(0xffffffffu, sc_l, j);
            const float* pp = base + (size_t)(s0 + j) * stride + lane * (D / 32);
            const float2 v0 = *reinterpret_cast<const float2*>(pp), v1 = *reinterpret_cast<const float2*>(pp + 2);
            acc[0] += v0.x * sc; acc[1] += v0.y * sc; acc[2] += v1.x * sc; acc[3] += v1.y * sc;
        }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, o);
    const float inv = ll > 0.f ? 1.0f / ll : 0.f;
    half* op = p.o + ((size_t)row * p.nq + head) * D + lane * (D / 32);
    #pragma unroll
    for (int e = 0; e < D / 32; e += 2) *reinterpret_cast<uint32_t*>(op + e) = pack_h2(acc[e] * inv, acc[e + 1] * inv);
    if constexpr (HAD) transform(make_uint2(pack_h2(acc[0] * inv, acc[1] * inv), pack_h2(acc[2] * inv, acc[3] * inv)));
}

// The same for few rows, where the kernel is bounded by its chain of dependent loads.  The attention kernels let it go behind their own
// wait, so a row's sequence, split count and place among the partials, which come from kernels in front of those, are found before the
// wait; behind it the splits' maxima and sums and the first eight rows are requested together.  (us, together with the later release:
// 24 sequences over 8-bit pools 58.2 -> 55.7, 4 x 8 rows over fp16 36.6 -> 31; as the last of a 27B-class verify layer, 32 rows and up to
// 37 splits, 11.2 -> 5.0.)  Its 80 registers against 40 cost more than they give where there are many rows.
template <int D, bool HAD>
__global__ void __launch_bounds__(256) attn_combine_few_kernel(const AttnParams p, int rows_per_cta, int total_rows, const half* had_suh, half* had_out)
{
    static_assert(D == 128, "a lane covers 4 dims as two 8-byte loads");
    constexpr int AHEAD = 8;                           // rows in flight per warp
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    uint2 sg = make_uint2(0u, 0u);                             // signs do not depend on the kernels in front
    int row = 0, head = 0, splits = 0;
    const float* base = nullptr;
    const size_t stride = (size_t)p.nkv * rows_per_cta * (D + 2);             // floats between consecutive splits
    bool mine = w < (long long)total_rows * p.nq;
    if (mine) {
        row = (int)(w / p.nq); head = (int)(w % p.nq);
        if constexpr (HAD) sg = reinterpret_cast<const uint2*>(had_suh)[head * 32 + lane];
        int b, row_base;
        if (p.cu_q) {                                          // binary search: cu_q[b] <= row < cu_q[b+1]
            int lo = 0, hi = p.bsz - 1;
            while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (__ldcg(p.cu_q + mid) <= row) lo = mid; else hi = mid - 1; }
            b = lo;
            row_base = __ldcg(p.cu_q + b);
            mine = row < __ldcg(p.cu_q + b + 1);                  // rows behind the last sequence have no partials
        } else { b = row / p.q_len; row_base = b * p.q_len; }
        splits = __ldcg(p.seq_splits + b);
        const int G = p.nq / p.nkv, kvh = head / G;
        const int packed = (row - row_base) * G + (head - kvh * G);
        const int rb = packed / rows_per_cta, lr = packed - rb * rows_per_cta;
        const int item0 = __ldcg(p.seq_base + b) + rb * splits;
        base = p.partial + (((size_t)item0 * p.nkv + kvh) * rows_per_cta + lr) * (D + 2);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // the attention kernel in front has handed out all its units: the work list is ready for the next layer's
    if (blockIdx.x == 0 && threadIdx.x == 0) const_cast<AttnPlan*>(p.plan)->next = 0;
    if (!mine) return;
    // the input transform of the projection behind the attention: a head is one 128-block of its k
    auto transform = [&](uint2 v) {
        reinterpret_cast<uint2*>(had_out)[((size_t)row * p.nq + head) * 32 + lane] =
            had128_signed_lane(*reinterpret_cast<const half2*>(&v.x), *reinterpret_cast<const half2*>(&v.y), sg, lane);
    };
    if (splits <= 1) {                                         // the attention kernel wrote the final value itself
        if constexpr (HAD) transform(*reinterpret_cast<const uint2*>(p.o + ((size_t)row * p.nq + head) * D + lane * (D / 32)));
        return;
    }
    float2 v0[AHEAD], v1[AHEAD];
    auto fetch = [&](int s0) {
        #pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            v0[j] = v1[j] = make_float2(0.f, 0.f);
            if (s0 + j < splits) {
                const float* pp = base + (size_t)(s0 + j) * stride + lane * (D / 32);
                v0[j] = *reinterpret_cast<const float2*>(pp); v1[j] = *reinterpret_cast<const float2*>(pp + 2);
            }
        }
    };
    auto max_sum = [&](int s) { return s < splits ? *reinterpret_cast<const float2*>(base + (size_t)s * stride + D) : make_float2(-INFINITY, 0.f); };
    float2 ms = max_sum(lane);
    fetch(0);
    float mm = ms.x;
    for (int s = lane + 32; s < splits; s += 32) mm = fmaxf(mm, max_sum(s).x);
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    float acc[D / 32], ll = 0.f;
    #pragma unroll
    for (int e = 0; e < D / 32; ++e) acc[e] = 0.f;
    for (int s0 = 0; s0 < splits; s0 += 32) {
        if (s0 > 0) ms = max_sum(s0 + lane);
        const float sc_l = ms.x == -INFINITY ? 0.f : exp2f(ms.x - mm);
        ll += ms.y * sc_l;
        const int cnt = min(32, splits - s0);
        for (int j0 = 0; j0 < cnt; j0 += AHEAD) {
            #pragma unroll
            for (int j = 0; j < AHEAD; ++j) {           // rows behind the last split count as zeros
                const float sc = __shfl_sync(0xffffffffu, sc_l, j0 + j);
                acc[0] += v0[j].x * sc; acc[1] += v0[j].y * sc; acc[2] += v1[j].x * sc; acc[3] += v1[j].y * sc;
            }
            if (s0 + j0 + AHEAD < splits) fetch(s0 + j0 + AHEAD);
        }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, o);
    const float inv = ll > 0.f ? 1.0f / ll : 0.f;
    half* op = p.o + ((size_t)row * p.nq + head) * D + lane * (D / 32);
    #pragma unroll
    for (int e = 0; e < D / 32; e += 2) *reinterpret_cast<uint32_t*>(op + e) = pack_h2(acc[e] * inv, acc[e + 1] * inv);
    if constexpr (HAD) transform(make_uint2(pack_h2(acc[0] * inv, acc[1] * inv), pack_h2(acc[2] * inv, acc[3] * inv)));
}

template <int D, int WM, int WN, int QB>
cudaError_t launch_attn(exl3_ctx* ctx, const AttnParams& p, dim3 grid, cudaStream_t st)
{
    constexpr int bytes = AttnSmem<D, QB>::BYTES;
    auto kern = attn_paged_kernel<D, WM, WN, QB>;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    return exl3_launch(ctx, kern, grid, AT_THREADS, bytes, st, p);
}

// the cluster form: `parts` CTAs per sequence and kv head
template <int QB>
cudaError_t launch_attn_cluster(exl3_ctx* ctx, const AttnParams& p, int parts, cudaStream_t st)
{
    constexpr int bytes = AttnSmem<128, QB, AT_CL_STAGES>::BYTES;
    auto kern = attn_paged_kernel<128, 1, 4, QB, true>;
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(parts, p.nkv, p.bsz); cfg.blockDim = dim3(AT_THREADS); cfg.dynamicSmemBytes = bytes; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = parts; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = exl3_chained(ctx) ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn attn_encode_tiled()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
        else
            cudaGetLastError();
    }
    return fn;
}

// tcgen05 attention: one CTA per work item and kv head; K/V tiles come through 4-D tensor maps of the pools
cudaError_t launch_attn_tc(exl3_ctx* ctx, const AttnParams& p, int max_items, cudaStream_t st)
{
    EncodeTiledFn enc = attn_encode_tiled();
    if (!enc) return cudaErrorNotSupported;
    CUtensorMap maps[2];
    const void* pools[2] = {p.kc, p.vc};
    for (int i = 0; i < 2; ++i) {
        cuuint64_t dims[4] = {(cuuint64_t)ATC_D, (cuuint64_t)p.nkv, 256, (cuuint64_t)p.pages};
        cuuint64_t strides[3] = {(cuuint64_t)ATC_D * 2, (cuuint64_t)p.nkv * ATC_D * 2, (cuuint64_t)256 * p.nkv * ATC_D * 2};
        cuuint32_t box[4] = {64, 1, (cuuint32_t)ATC_TN, 1};           // 128 tokens of one page, one 64-wide d block
        cuuint32_t estr[4] = {1, 1, 1, 1};
        if (enc(&maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(pools[i]), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATC_SMEM);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    (void)ctx;
    attn_tc_kernel<<<dim3((unsigned)max_items * p.nkv), ATC_THREADS, ATC_SMEM, st>>>(maps[0], maps[1], p);
    return cudaPeekAtLastError();
}

cudaError_t launch_attn_tc2(exl3_ctx* ctx, const AttnParams& p, int max_items, cudaStream_t st)
{
    EncodeTiledFn enc = attn_encode_tiled();
    if (!enc) return cudaErrorNotSupported;
    CUtensorMap maps[2];
    const void* pools[2] = {p.kc, p.vc};
    for (int i = 0; i < 2; ++i) {
        cuuint64_t dims[4] = {(cuuint64_t)ATC_D, (cuuint64_t)p.nkv, 256, (cuuint64_t)p.pages};
        cuuint64_t strides[3] = {(cuuint64_t)ATC_D * 2, (cuuint64_t)p.nkv * ATC_D * 2, (cuuint64_t)256 * p.nkv * ATC_D * 2};
        cuuint32_t box[4] = {64, 1, (cuuint32_t)ATC_TN, 1};           // 128 tokens of one page, one 64-wide d block
        cuuint32_t estr[4] = {1, 1, 1, 1};
        if (enc(&maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(pools[i]), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    static bool configured[64] = {};
    static const int tune_h = getenv("EXL3_TUNE_TC_H") ? atoi(getenv("EXL3_TUNE_TC_H")) : 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(attn_tc2_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, A2_SMEM);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_tc2_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, A2_SMEM);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const dim3 grid((unsigned)max_items * p.nkv);
    return tune_h == 4 ? exl3_launch(ctx, attn_tc2_kernel<4>, grid, a2_threads(4), A2_SMEM, st, maps[0], maps[1], p)
                       : exl3_launch(ctx, attn_tc2_kernel<2>, grid, a2_threads(2), A2_SMEM, st, maps[0], maps[1], p);
}

// kernels over 4-bit and 8-bit pools: tensor maps over the code planes ([tokens][nkv * 4 * bits] words, copied in
// the swizzle of a head's 64 or 128 bytes) and the scale planes ([tokens][nkv * 4] halves, copied in 16-byte pairs of heads)
template <int B>
cudaError_t quant_maps(const AttnParams& p, int tile_keys, CUtensorMap (&maps)[4])
{
    EncodeTiledFn enc = attn_encode_tiled();
    if (!enc) return cudaErrorNotSupported;
    const void* planes[4] = {p.qk, p.qv, p.sk, p.sv};
    const cuuint64_t tokens = (cuuint64_t)p.pages * EXL3_PAGE;
    for (int i = 0; i < 4; ++i) {
        const bool codes = i < 2;
        cuuint64_t dims[2] = {(cuuint64_t)p.nkv * (codes ? 4 * B : 4), tokens};
        cuuint64_t strides[1] = {(cuuint64_t)p.nkv * (codes ? 16 * B : 8)};
        cuuint32_t box[2] = {codes ? 4u * B : 8u, (cuuint32_t)tile_keys};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&maps[i], codes ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(planes[i]),
                dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                !codes ? CU_TENSOR_MAP_SWIZZLE_NONE : (B == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B),
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

// launch of a kernel over quantised pools with `bytes` of dynamic shared memory
template <int B, typename Kern>
cudaError_t launch_quant(exl3_ctx* ctx, Kern kern, bool (&configured)[64], int bytes, int threads, int tile_keys, const AttnParams& p, dim3 grid, cudaStream_t st)
{
    CUtensorMap maps[4];
    cudaError_t e = quant_maps<B>(p, tile_keys, maps);
    if (e != cudaSuccess) return e;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    return exl3_launch(ctx, kern, grid, threads, bytes, st, maps[0], maps[1], maps[2], maps[3], p);
}
template <int B, int NB>
cudaError_t launch_attn_qdec(exl3_ctx* ctx, const AttnParams& p, dim3 grid, cudaStream_t st)
{
    static bool configured[64] = {};
    return launch_quant<B>(ctx, attn_qdec_kernel<B, NB>, configured, QdSmem<B, NB>::BYTES, QD_THREADS, QD_TK, p, grid, st);
}
template <int B>
cudaError_t launch_attn_qt(exl3_ctx* ctx, const AttnParams& p, dim3 grid, cudaStream_t st)
{
    static bool configured[64] = {};
    return launch_quant<B>(ctx, attn_qt_kernel<B>, configured, QtSmem<B>::BYTES, QT_THREADS, QT_TK, p, grid, st);
}

bool qdec_kernel_applies(const AttnParams& p, bool quant);

// at least so many sequences of a batch have more than one row
int min_long(int total_rows, int bsz, int max_q_len)
{
    return max_q_len > 1 ? (int)std::max(0LL, ((long long)total_rows - bsz + max_q_len - 2) / (max_q_len - 1)) : 0;
}

// Which kernels a pass runs: those for few packed rows, those for more, or (4-bit and 8-bit pools) the tcgen05 kernel over codes.
enum AttnClass { ATTN_FEW, ATTN_MANY, ATTN_CODES };

// One pass = plan + attention + combine over the sequences whose packed row count lies in (rows_lo, rows_hi].
int attn_pass(exl3_ctx* ctx, cudaStream_t st, AttnParams p, int total_rows, int max_rows, int rows_lo, int rows_hi,
              AttnClass kind, bool quant, size_t* ws_off, const AttnAppendArgs* append, bool had = false)
{
    const int D = 128;
    const int G = p.nq / p.nkv;
    const bool decode_shape = kind == ATTN_FEW, use_qt = kind == ATTN_CODES;
    const bool q4 = quant && p.k_bits == 4 && p.v_bits == 4;       // the common cache format has its own, smaller staging
    // long class on fp16 pools: tcgen05 kernel (256-row items) unless the context was switched to the mma.sync kernels
    // (its row maximum is taken on the raw scores, which needs a positive scale)
    // (sequences with 17..128 packed rows - speculative verify - stay on it too: on 32 sequences x 8 query rows x 5 heads
    // the 64-row mma.sync kernel measured 228 us against 224 us, at 16 and 24 query rows 373 / 383 us against 233 / 241 us)
    const bool use_tc = !decode_shape && !quant && ctx->mma_attn != 0 && p.scale_log2 > 0.f && !p.contig_kv;
    // two arrangements of the tcgen05 kernel: 128-row items with two softmax threads per row (default), 256-row items
    static const bool tc_256 = getenv("EXL3_B200_ATTN_TC256") != nullptr;
    // 4-bit and 8-bit pools, decode class: the kernel that builds its operands from the codes (its scale copies are 16 bytes
    // wide = two heads, so the kv head count must be even and the planes 16-byte aligned).  Row blocks of 8 where no
    // sequence has more rows (a decode batch), else of 16, whose second half costs nothing where it is empty.
    const bool use_qdec = decode_shape && qdec_kernel_applies(p, quant);
    const int rows_per_cta = use_qt ? QT_ROWS : decode_shape ? (use_qdec && max_rows <= 8 ? 8 : 16) : (use_tc ? (tc_256 ? ATC_CTA_ROWS : A2_ROWS) : 64);
    const int rb_max = (max_rows + rows_per_cta - 1) / rows_per_cta;
    // resident CTAs per SM over all kv heads: about 3 for the mma.sync kernels, 1 for the tcgen05 kernel (all of TMEM)
    // (rounded down: one CTA more than fits would run alone in a second wave after all the others have finished)
    int per_sm = 1;
    if (use_qt) per_sm = 2;
    else if (use_qdec) per_sm = qd_ctas(p.k_bits, rows_per_cta / 8);
    else if (!use_tc) {
        // CTAs of the mma.sync kernel that fit on an SM (bounded by shared memory: stages x 34.8 KB for fp16 pools)
        const size_t smem = quant ? (q4 ? AttnSmem<128, 4>::BYTES : AttnSmem<128, 8>::BYTES) : AttnSmem<128, 0>::BYTES;
        per_sm = std::max(1, std::min(q4 ? 4 : 3, (int)((227 * 1024) / (smem + 1024))));
    }
    const int grid_x = std::max(1, ctx->num_sms * per_sm / p.nkv);
    // tcgen05 kernels: two items per CTA slot: more items shorten the tail of the last wave but every extra KV split costs
    // a partial per kv head written and read back (128-row kernel on 4 x 256 query rows: 154 / 168 / 171 / 188 / 205 us at
    // 2 / 3 / 4 / 6 / 8 per slot).
    // mma.sync kernels (units handed out dynamically, 8 KB partials): see below.
    static const int tc_items = getenv("EXL3_TUNE_TC_ITEMS") ? atoi(getenv("EXL3_TUNE_TC_ITEMS")) : 0;
    // With the units handed out longest first, fewer and longer items win on the mma.sync kernels too (64 decode
    // sequences over fp16 pools at 1 / 2 / 3 / 4 items per slot: 242 / 234 / 237 / 242 us): two, and one for the kernel over
    // quantised pools, whose units start with the rotation of their queries (24 sequences, contexts 512 .. 16384, 40 / 8
    // heads, one and two items: 4 bits, 5 rows 68 and 72 us, 40 rows 188 and 193; 8 bits 68 and 75, 188 and 196).
    static const int dec_items = getenv("EXL3_TUNE_DEC_ITEMS") ? atoi(getenv("EXL3_TUNE_DEC_ITEMS")) : 0;
    // The tcgen05 kernel over codes: one item per slot; two, which balance the blocks, where these are not few and contexts may be long; and
    // where they are few less half of them, because each rounds its count up and items beyond the slots are a second wave (us, one and two:
    // 4 sequences of 65 rows, 512 .. 4096, 35 and 37, of 100, 512 .. 4096, 32 and 44, 1024 .. 32768 110 and 98, of 500 506 and 368; one of
    // 250 rows, 512 .. 4096, 25 and 35, of 500, 1024 .. 32768, 110 and 83; 16 of 250, 1024 .. 32768, 830 and 717; 5 of a row and 2 of 640,
    // 109 .. 218, 27 and 39; 3 of 410, 377 .. 1919, at 8 bits 86 and 92; without and with the half: 3 of 125, 512 .. 2048, 34 and 28, one of 300
    // 31 and 25, 5 of 40, 1024 .. 32768, 63 and 52, but 2 of 205, 600 and 2000, 29 and 32).
    const int n_long = min_long(total_rows, p.bsz, max_rows / G);
    const long long qt_blocks = (long long)n_long * rb_max + (rows_lo == 0 ? p.bsz - n_long : 0);
    const bool qt_few = use_qt && 3 * qt_blocks <= grid_x, one_item = use_qdec || (use_qt && p.pps <= 8);
    const int target_items = dec_items && !use_tc ? grid_x * dec_items : qt_few ? grid_x - (int)qt_blocks / 2
                             : grid_x * (use_tc ? (tc_items ? tc_items : 2) : (one_item ? 1 : 2));
    // items <= target + sum of row blocks (every (sequence, row block) rounds its split count up once); the row blocks are
    // bounded by bsz * rb_max and, usually much tighter for ragged batches, by total_rows * G / rows_per_cta + bsz
    const long long rb_sum = std::min((long long)p.bsz * rb_max, ((long long)total_rows * G + rows_per_cta - 1) / rows_per_cta + p.bsz);
    const int max_items = target_items + (int)std::min(rb_sum, (long long)(1 << 24)) + 1;

    // The work list depends on the batch's lengths, not on the layer: inside exl3_step_forward it is built by the first
    // layer's call into the context's slot for this class and reused by the other layers.
    const int cls = decode_shape ? 0 : 1;
    const size_t list_bytes = 256 + (((size_t)max_items * sizeof(AttnItem) + 255) & ~(size_t)255) + 2 * (((size_t)p.bsz * 4 + 255) & ~(size_t)255);
    const bool keep = ctx->plan_keep && list_bytes <= ctx->plan_slot_bytes;
    size_t off = *ws_off;                                // scratch of an earlier pass that may still be running
    AttnPlan* plan; AttnItem* items; int* seq_base; int* seq_splits;
    if (keep) {
        uint8_t* slot = ctx->plan_slots + cls * ctx->plan_slot_bytes;
        plan = (AttnPlan*)slot;
        items = (AttnItem*)(slot + 256);
        seq_base = (int*)(slot + 256 + (((size_t)max_items * sizeof(AttnItem) + 255) & ~(size_t)255));
        seq_splits = (int*)((uint8_t*)seq_base + (((size_t)p.bsz * 4 + 255) & ~(size_t)255));
    } else {
        plan = (AttnPlan*)exl3_ws_take(ctx, &off, sizeof(AttnPlan));
        items = (AttnItem*)exl3_ws_take(ctx, &off, (size_t)max_items * sizeof(AttnItem));
        seq_base = (int*)exl3_ws_take(ctx, &off, (size_t)p.bsz * 4);
        seq_splits = (int*)exl3_ws_take(ctx, &off, (size_t)p.bsz * 4);
    }
    float* partial = (float*)exl3_ws_take(ctx, &off, (size_t)max_items * p.nkv * rows_per_cta * (D + 2) * 4);
    if (!plan || !items || !seq_base || !seq_splits || !partial)
        return exl3_fail(ctx, EXL3_ERR_WORKSPACE, "attention: context scratch too small for the split-KV partials");
    p.plan = plan; p.items = items; p.seq_base = seq_base; p.seq_splits = seq_splits; p.partial = partial;
    p.status = ctx->status;
    *ws_off = off;

    static const bool no_lpt = getenv("EXL3_TUNE_NO_LPT") != nullptr;
    const int chunk_mult = use_tc ? ATC_TN : use_qt ? QT_TK : AT_TK;
    const unsigned long long shape = (unsigned long long)target_items << 36 | (unsigned long long)std::min(rows_hi, 255) << 28 | (unsigned long long)rows_lo << 20 | chunk_mult << 10 | rows_per_cta;
    if (!(keep && ctx->plan_shape[cls] == shape)) {
        const AttnPlanArgs a = {p.seqlens, p.cu_q, plan, items, seq_base, seq_splits, ctx->status, p.bsz, p.q_len, p.kv_append, G, rows_per_cta, rows_lo, rows_hi,
                                chunk_mult, target_items, max_items, no_lpt ? -1 : (p.causal ? 1 : 0), (use_tc && !tc_items) ? grid_x : 0};
        if (append) {
            const long long warps = (long long)append->rows * (append->k_bits ? append->nkv : 1);
            exl3_launch_first(ctx, attn_front_kernel, 1 + (unsigned)((warps + AP_THREADS / 32 - 1) / (AP_THREADS / 32)), AP_THREADS, 0, st, a, *append);
        } else
            exl3_launch(ctx, attn_plan_kernel, 1, AP_THREADS, 0, st, a);
        ctx->launches++;
        if (keep) ctx->plan_shape[cls] = shape;
    }
    exl3_chain_scope chain(ctx);
    dim3 grid(grid_x, p.nkv);
    cudaError_t e;
    if (use_tc) e = tc_256 ? launch_attn_tc(ctx, p, max_items, st) : launch_attn_tc2(ctx, p, max_items, st);
    else if (use_qt) e = q4 ? launch_attn_qt<4>(ctx, p, grid, st) : launch_attn_qt<8>(ctx, p, grid, st);
    else if (use_qdec)
        e = q4 ? (rows_per_cta == 8 ? launch_attn_qdec<4, 1>(ctx, p, grid, st) : launch_attn_qdec<4, 2>(ctx, p, grid, st))
               : (rows_per_cta == 8 ? launch_attn_qdec<8, 1>(ctx, p, grid, st) : launch_attn_qdec<8, 2>(ctx, p, grid, st));
    else if (q4)    e = decode_shape ? launch_attn<128, 1, 4, 4>(ctx, p, grid, st) : launch_attn<128, 4, 1, 4>(ctx, p, grid, st);
    else if (quant) e = decode_shape ? launch_attn<128, 1, 4, 8>(ctx, p, grid, st) : launch_attn<128, 4, 1, 8>(ctx, p, grid, st);
    else            e = decode_shape ? launch_attn<128, 1, 4, 0>(ctx, p, grid, st) : launch_attn<128, 4, 1, 0>(ctx, p, grid, st);
    ctx->launches++;
    if (e != cudaSuccess) { cudaGetLastError(); return exl3_fail(ctx, EXL3_ERR_CUDA, cudaGetErrorString(e)); }
    const long long warps = (long long)total_rows * p.nq;
    // The merge of few rows up to six blocks per SM (us, that of many and that of few: fp16, 24 rows of 40 heads 65.6 and 61.2, 4 x 32
    // rows 48.0 and 43.2, 256 rows 451 and 452, a prefill chunk of 512 53.7 and 55.5; 4 bits, 64 rows 74.5 and 72.5, 256 rows 223.5
    // and 225.1).  In a batch of two passes up to one: its blocks wait, with twice the registers, on SMs that the other pass could use
    // (fp16, 40 heads, 8 of a row and one of 16, 120 blocks, 64.8 and 59.6; one of 40, 240, 24.9 and 23.2; 28 and one of 40, 340, 21.6 and
    // 26.2; 64 and four of 16, 640, 28.4 and 42.0; 100 and one of 40 over 1000 .. 16000 keys 366 and 372).
    const bool pair = rows_lo > 0 || st == ctx->aux_stream;
    const bool few = (warps + 7) / 8 <= (pair ? 1LL : 6LL) * ctx->num_sms;
    auto merge = had ? (few ? attn_combine_few_kernel<128, true> : attn_combine_kernel<128, true>)
                     : (few ? attn_combine_few_kernel<128, false> : attn_combine_kernel<128, false>);
    exl3_launch(ctx, merge, (unsigned)((warps + 7) / 8), 256, 0, st, p, rows_per_cta, total_rows, had ? ctx->had_suh : (const half*)nullptr,
                had ? ctx->had_out : (half*)nullptr);
    ctx->launches++;
    return exl3_check_launch(ctx, "attention");
}

// Sequences with at most 16 packed (query, head) rows (decode, short verify) take the kernel that spreads the keys of a
// tile over the four warps; longer ones (verify with many heads, prefill chunks) the one with a 16-row tile per warp.
// A ragged batch that holds both kinds runs one pass for each.
// true when attn_pass will take the decode-class kernel for quantised pools (attn_qdec.cuh)
bool qdec_kernel_applies(const AttnParams& p, bool quant)
{
    static const bool no_q4 = getenv("EXL3_B200_NO_Q4_ATTN") != nullptr;
    return quant && (p.k_bits == 4 || p.k_bits == 8) && p.v_bits == p.k_bits && !no_q4 && p.nkv % 2 == 0 && aligned16(p.qk) && aligned16(p.qv) &&
           aligned16(p.sk) && aligned16(p.sv);
}

// Appends a call's keys and values ahead of the attention, as the public operators do.
int attn_append(exl3_ctx* ctx, cudaStream_t st, const AttnAppendArgs& a)
{
    return a.k_bits ? exl3_quant_cache_paged(ctx, st, a.k, a.qk, a.sk, a.v, a.qv, a.sv, a.seqlens, a.block_table, a.cu_q, a.bsz, a.seq, a.nkv * 128, a.pages, a.pps,
                                             a.k_bits, a.v_bits, EXL3_PAGE, 0.0f, 1)
                    : exl3_paged_kv_cache_update(ctx, st, a.k, a.v, a.kc, a.vc, a.block_table, a.seqlens, a.cu_q, a.bsz, a.seq, a.nkv, 128, a.pages, a.pps);
}

// `append`: the call's keys and values, which go to the pools in front of the attention, or NULL
int attn_impl(exl3_ctx* ctx, cudaStream_t st, AttnParams p, int total_rows, int max_q_len, bool quant, const AttnAppendArgs* append)
{
    const int G = p.nq / p.nkv;
    const int max_rows = max_q_len * G;
    // Decode class = sequences with at most 16 packed rows.  Over 4-bit and 8-bit pools it also takes up to 48 rows
    // (speculative verify: 8 query rows x 5 heads) as row blocks of 16 that each walk the codes again: the kernel that
    // builds its operands from the codes is that much cheaper per key than the generic one.  Against the generic kernel, us,
    // 40 / 8 heads, 15 / 25 / 40 / 45 rows: 24 sequences, contexts 512 .. 16384, 4 bits 93 / 144 / 188 / 193 against 130 /
    // 196 / 197 / 197, 8 bits 95 / 148 / 188 / 198 against 216 / 282 / 289 / 280; 64 sequences, contexts 128 .. 4096, 40 and 45
    // rows, 4 bits 146 / 155 against 158 / 162, 8 bits 149 / 158 against 216 / 221; 4 sequences, contexts 1024 .. 32768, 45
    // rows, 99 against 126 and 104 against 156.  Behind only on one sequence of 8192 with 40 or more rows at 4 bits (51
    // against 46).  A ragged batch with longer sequences runs all its decode rows in blocks of 16 (28 of 1 row beside 4 of 64
    // rows: 4 bits 221 us, 252 with everything on the generic kernel; 8 bits 286 and 374).
    // (Sending the decode rows of a ragged fp16 batch through the tcgen05 kernel as well, as items of 128 rows with 5 in
    // use, was measured on the benchmark step: the attention stage takes the same 28.0 ms of the step's 83.)
    const int dec_rows = qdec_kernel_applies(p, quant) ? 48 : 16;
    // The tcgen05 kernel over codes unpacks them once for 40 rows; its blocks cost the same however few of those they hold, and a unit
    // some 10 us before and behind its tiles.  So, us, the other kernels and it (40 / 8 heads unless said, contexts spread evenly over
    // the logarithm of a range, calls replayed):
    //  * one block per sequence, 33 to 40 rows, at 4 bits, where the pages of the block table leave room for work for all SMs: 4 of 40
    //    rows, 1024 .. 32768, 72 and 43; 12, 512 .. 4096, 50 and 41; 32, 128 .. 1024, 45 and 42; but 6, 128 .. 1024, 20.7 and 21.2, one,
    //    128 .. 8192, 20 and 21.  Beside sequences of few rows, up to half as many: 8 of a row beside 16 of 40, 1024 .. 32768, 268 and
    //    185, 512 .. 4096 69 and 62, 128 .. 1024 36 and 41; 8 beside 4, 128 .. 8192, 41 and 41, 128 .. 1024 21 and 23; 28 beside 4 51 and
    //    70; 64 beside one 70 and 107; and with half the kv heads and so half the work 4 beside 12, 512 .. 4096, 32 and 38, 128 .. 8192 37
    //    and 31.  Two blocks, 41 to 48 rows: 12 of 44, 128 .. 8192, 57 and 63, 32 of 48 with four kv heads 67 and 74.  At 8 bits, where the
    //    ring of codes has one slot, 4 of 45, 1024 .. 32768, 82 and 117.
    //  * more rows: 4 of 65 rows, 512 .. 4096, 43 and 35, of 120 47 and 33, of 500 124 and 109; 16 of 640, 1024 .. 32768, 1945 and 1531; at 8
    //    bits 58 and 43, 63 and 42, 166 and 148, 3013 and 2361.  The other kernel's block has 64 rows: up to that many, 4 of 50, 512 .. 4096,
    //    28 and 33, 16, 1024 .. 32768, 232 and 232, at 8 bits 334 and 361; one alone 26 and 20, 35 and 23, and of a ragged
    //    batch, where the other kernel is a pass beside that of few rows, 8 of a row and 3 of 50 46 and 43, 58 and 52.  (8 bits with more
    //    than 800 rows stay where they were.)
    //    Where contexts are short a unit is little more than its start and end, and a second wave of them costs as much as the first: by the
    //    block table, one page and more than a wave (6 of 300 rows without a context 20 and 29, 24 of 640 133 and 156, 4 of 300, one wave,
    //    20 and 19; with contexts of 64 .. 128 26 and 34, 161 and 187, 26 and 24), or up to five pages, more blocks than the other kernel has, and
    //    a second or third wave that it does not need (128 .. 512, one of 800 rows 29 and 34, 5 of 300 34 and 42, 12 of 125 33 and 43; but 5 of
    //    800 86 and 71, 12 of 300 72 and 68, 24 of 65, as many blocks in either, 48 and 42; with eight pages 3 of 410 92 and 85; beside
    //    sequences of few rows, for which the other kernel needs a pass more, 5 of a row and 2 of 640 47 and 27, 40 and 2 of 240 without a
    //    context 26 and 32, 0.87 in the mean of 700 such batches).
    //  * a ragged batch of both kinds in one pass instead of two, as long as the short ones have few keys, by the width of the block table:
    //    8 of a row and one of 100, two passes and one, 128 .. 1024 (5 pages) 25 and 20, 512 .. 4096 (17) 42 and 33, 1024 .. 32768 (129) 80 and
    //    94; 32 and one 39 and 30, 63 and 64, 168 and 223; at 8 bits 29 and 23, 47 and 43, 89 and 142; 44 and 38, 71 and 96, 171 and 359.
    const bool codes = qdec_kernel_applies(p, quant);
    const int n_long = min_long(total_rows, p.bsz, max_q_len);
    const long long table = (long long)p.bsz * p.pps;
    auto waves = [&](int rows, int per_sm) -> long long {          // of units, at two splits per block where a context can have more than a page
        const long long slots = (long long)per_sm * ctx->num_sms;
        return ((long long)n_long * ((max_rows + rows - 1) / rows) * p.nkv * (p.pps == 1 ? 1 : 2) + slots - 1) / slots;
    };
    const long long wq = waves(QT_ROWS, 2), w64 = waves(64, 3);
    const bool cheap = n_long >= p.bsz && (p.pps == 1 ? wq > 1 : p.pps <= 5 && (max_rows + QT_ROWS - 1) / QT_ROWS > (max_rows + 63) / 64 && wq > w64 && wq <= 3);
    const bool long_codes = codes && max_rows > dec_rows && (p.k_bits == 4 || max_rows <= 800) && (max_rows > 64 || p.cu_q || p.bsz == 1) && !cheap;
    const bool codes_alone = long_codes ? (long long)(p.bsz - n_long) * p.pps <= (p.k_bits == 4 ? 300 : 200)
                                        : codes && p.k_bits == 4 && max_rows > 32 && max_rows <= QT_ROWS && table >= 200 &&
                                          (n_long >= p.bsz || (3 * n_long >= 2 * p.bsz && table * p.nkv >= 1600));
    // One pass.  (The transform behind the attention is left to its own launch where the scratch does not hold it beside the
    // partials; attn_pass refuses before it launches anything.)  The list and the append are one launch unless the list is another
    // layer's already.
    const bool one = append && !ctx->plan_keep;
    auto single = [&](AttnClass kind, int rows_hi) -> int {
        int rc = EXL3_ERR_WORKSPACE;
        if (ctx->had_out) {
            size_t off = ctx->had_bytes;
            rc = attn_pass(ctx, st, p, total_rows, max_rows, 0, rows_hi, kind, quant, &off, one ? append : nullptr, true);
            ctx->had_done = rc == EXL3_OK;
        }
        size_t off = 0;
        if (rc == EXL3_ERR_WORKSPACE) rc = attn_pass(ctx, st, p, total_rows, max_rows, 0, rows_hi, kind, quant, &off, one ? append : nullptr);
        return rc;
    };
    const bool general_single = max_rows <= dec_rows || !p.cu_q;
    // A small batch in clusters (attn_paged.cuh): at most two CTAs per SM with as many parts per sequence and kv head as that allows, and
    // at most 512 keys per part, by the width of the block table: a longer sequence among short ones would hold up the others'
    // SMs, which the work list shares out.  Us, list and clusters: step of 28 layers of hidden 1024, 8 sequences of up to 1024 tokens,
    // 1409 and 1332; calls of 16 / 8 heads over fp16 pools, replayed, 8 sequences of 1000 keys 15.8 and 13.7, of 2000 24.9 and 20.0, one
    // of 2000 among seven of 64 14.4 and 13.6, but one of 4000 15.7 and 21.5; one of 4000 among three of 64 (eight parts) 15.7 and 13.9,
    // among fifteen (two parts) 16.0 and 37.4; one sequence of 64 9.8 and 5.4, of 4000 15.2 and 13.0, of 8000 17.6 and 21.0.  Twice the
    // parts, four CTAs per SM: 8 of 1000 17.6, 16 of 500 16.8 against 13.9 in two parts; 32 of 500 in two parts 23.4 and by the list 25.3,
    // 32 of 250 16.5 and 15.3.
    // In a step, where the list is built once for all layers: us a layer of hidden 1024, 16 / 8 heads, list and clusters, 8 of 2000 keys 54.8
    // and 51.1, 16 of 1000 54.9 and 50.9, one of 2000 among seven of 64 45.2 and 46.6; with fewer CTAs at most 448 keys per part, 4 of 2000 in
    // four parts 45.2 and 48.3, one of 4000 in eight 45.1 and 47.5, of 3000 among three of 64 45.5 and 43.9; and clusters of eight only
    // where they leave room, because one waits for eight places at a time: 32 of them (4 of 1000) 46.1, of four CTAs 42.7, list 45.0; 4 of
    // 4000 in eight parts 63.5 and 55.2; 24 (3 of 3000) 46.0 and 46.2; 16 (2 of 2000) 41.8 and 44.4.
    // Codes, whose tiles take longer, at most 320 keys per part there (6 bits: one of 2000 among seven of 64 63.4 and 73.2, 3 of 3000 in
    // eight parts 60.5 and 68.6, 4 of 2000 62.5 and 80.4; but one of 1000 among seven 62.5 and 56.5; a call of its own, with its list, one of
    // 2000 among seven 29.7 and 36.3, 36 before list and append were one launch).
    int parts = 0;
    if (max_rows <= 16 && !codes && !p.contig_kv)
        for (int c = 8; c >= 2 && parts == 0; c >>= 1) {
            const long long ctas = (long long)p.bsz * p.nkv * c;
            const bool full = 2 * ctas > 3LL * ctx->num_sms, step = ctx->plan_keep;
            const int most = !step ? 512 : quant ? 320 : full ? 512 : 448;       // keys per part
            if (ctas <= 2LL * ctx->num_sms && (long long)p.pps * EXL3_PAGE <= (long long)most * c && !(step && full && c == 8)) parts = c;
        }
    if (parts) {
        if (append) {
            const int rc = attn_append(ctx, st, *append);
            if (rc != EXL3_OK) return rc;
        }
        exl3_chain_scope chain(ctx, append != nullptr);
        if (ctx->had_out) { p.had_suh = ctx->had_suh; p.had_out = ctx->had_out; }
        const cudaError_t e = !quant ? launch_attn_cluster<0>(ctx, p, parts, st) : launch_attn_cluster<8>(ctx, p, parts, st);
        ctx->launches++;
        if (e != cudaSuccess) { cudaGetLastError(); return exl3_fail(ctx, EXL3_ERR_CUDA, cudaGetErrorString(e)); }
        ctx->had_done = ctx->had_out != nullptr;
        return exl3_check_launch(ctx, "attention");
    }
    const bool apart = append && !(one && (codes_alone || general_single));
    if (apart) {
        const int rc = attn_append(ctx, st, *append);
        if (rc != EXL3_OK) return rc;
        append = nullptr;
    }
    exl3_chain_scope chain(ctx, apart);                    // (the append itself follows what the caller has in front)
    if (codes_alone) {
        const int rc = single(ATTN_CODES, 1 << 30);
        if (rc != EXL3_ERR_WORKSPACE) return rc;
    }
    if (general_single) {
        const int rc = single(max_rows <= dec_rows ? ATTN_FEW : ATTN_MANY, max_rows <= dec_rows ? dec_rows : 1 << 30);
        if (rc == EXL3_ERR_WORKSPACE && append) {          // nothing has been launched; the keys and values are appended all the same
            const int rc2 = attn_append(ctx, st, *append);
            if (rc2 != EXL3_OK) return rc2;
            return exl3_fail(ctx, rc, "attention: context scratch too small for the split-KV partials");
        }
        return rc;
    }
    if (append) {                                          // the codes' kernel alone has been refused
        const int rc = attn_append(ctx, st, *append);
        if (rc != EXL3_OK) return rc;
    }
    // Ragged batch with both classes: the decode-class pass (bound by HBM) is issued on the context's second stream and
    // the long-class pass (bound by the tensor core and the MUFU) on the caller's; they touch disjoint sequences and
    // output rows, and each has its own scratch.  Fork and join by events, which also works while the caller's stream
    // is being captured.  What the second stream buys is the tail of one pass filling with the other's first CTAs: a
    // tcgen05 CTA takes a whole SM, so the bulk of the two passes runs one after the other (per layer of the benchmark
    // step the attention stage takes the sum of the two kernels' times).
    if (cudaEventRecord(ctx->ev_fork, st) != cudaSuccess || cudaStreamWaitEvent(ctx->aux_stream, ctx->ev_fork, 0) != cudaSuccess)
        return exl3_fail(ctx, EXL3_ERR_CUDA, "attention: stream fork failed");
    ctx->chain_break = 1;
    size_t off = 0;
    int rc = attn_pass(ctx, ctx->aux_stream, p, total_rows, dec_rows, 0, dec_rows, ATTN_FEW, quant, &off, nullptr);
    ctx->chain_break = 1;
    int rc2 = rc;
    if (rc == EXL3_OK) {
        rc2 = long_codes && !codes_alone ? attn_pass(ctx, st, p, total_rows, max_rows, dec_rows, 1 << 30, ATTN_CODES, quant, &off, nullptr) : EXL3_ERR_WORKSPACE;
        if (rc2 == EXL3_ERR_WORKSPACE) rc2 = attn_pass(ctx, st, p, total_rows, max_rows, dec_rows, 1 << 30, ATTN_MANY, quant, &off, nullptr);
    }
    ctx->chain_break = 1;
    // always join, also after an error, so that a capture in progress stays well-formed
    if (cudaEventRecord(ctx->ev_join, ctx->aux_stream) != cudaSuccess || cudaStreamWaitEvent(st, ctx->ev_join, 0) != cudaSuccess)
        return exl3_fail(ctx, EXL3_ERR_CUDA, "attention: stream join failed");
    return rc != EXL3_OK ? rc : rc2;
}

int check_common(exl3_ctx* ctx, const void* q, const void* o, const int32_t* bt, const int32_t* sl, int bsz, int q_len,
                 int kv_append, int nq, int nkv, int hd, int pages, int pps)
{
    EXL3_REQUIRE(ctx && q && o && bt && sl, "attention: null argument");
    EXL3_REQUIRE(bsz >= 0 && q_len >= 0 && kv_append >= 0 && nq > 0 && nkv > 0 && pages > 0 && pps > 0, "attention: bad shape");
    EXL3_REQUIRE(nq % nkv == 0, "attention: n_q_heads must be a multiple of n_kv_heads");
    EXL3_REQUIRE(nq / nkv <= 16, "attention: GQA ratio above 16");
    if (hd != 128) return exl3_fail(ctx, EXL3_ERR_UNSUPPORTED, "attention: head_dim must be 128");
    EXL3_REQUIRE(nkv <= 65535, "attention: too many kv heads");
    EXL3_REQUIRE(aligned16(q) && aligned16(o), "attention: pointers must be 16-byte aligned");
    return EXL3_OK;
}

}  // namespace

extern "C" int exl3_bighead_attn_paged(exl3_ctx* ctx, exl3_stream stream, const void* q, const void* k, const void* v,
                                       void* k_cache, void* v_cache, const int32_t* block_table,
                                       const int32_t* cache_seqlens, const int32_t* cu_q, void* o, int bsz, int q_len,
                                       int kv_append, int nq, int nkv, int hd, int pages, int pages_per_seq,
                                       int kv_chunk_size, int causal, float sm_scale)
{
    (void)kv_chunk_size;
    int rc = check_common(ctx, q, o, block_table, cache_seqlens, bsz, q_len, kv_append, nq, nkv, hd, pages, pages_per_seq);
    if (rc) return rc;
    EXL3_REQUIRE(k_cache && v_cache && aligned16(k_cache) && aligned16(v_cache), "attention: bad cache pointers");
    if (bsz == 0 || q_len == 0) return EXL3_OK;
    const int append = cu_q ? q_len : kv_append;
    const bool write = append > 0 && !ctx->kv_appended;
    if (write) {
        EXL3_REQUIRE(k && v, "attention: kv_append > 0 needs k and v");
        EXL3_REQUIRE(aligned16(k) && aligned16(v), "paged_kv_cache_update: pointers must be 16-byte aligned");
        EXL3_REQUIRE(bsz <= 65535 && append <= 65535, "paged_kv_cache_update: bsz and seq must be <= 65535");
    }
    exl3_chain_scope chain(ctx, append > 0 && !write);
    AttnParams p;
    memset(&p, 0, sizeof(p));
    p.q = (const half*)q; p.o = (half*)o; p.kc = (const half*)k_cache; p.vc = (const half*)v_cache;
    p.block_table = block_table; p.seqlens = cache_seqlens; p.cu_q = cu_q;
    p.bsz = bsz; p.q_len = q_len; p.kv_append = kv_append; p.nq = nq; p.nkv = nkv; p.pps = pages_per_seq; p.pages = pages;
    p.causal = causal;
    p.scale_log2 = (sm_scale == 0.0f ? rsqrtf((float)hd) : sm_scale) * 1.4426950408889634f;
    const int total_rows = cu_q ? kv_append : bsz * q_len;
    const AttnAppendArgs a = {(const half*)k, (const half*)v, (half*)k_cache, (half*)v_cache, nullptr, nullptr, nullptr, nullptr, block_table, cache_seqlens, cu_q,
                              bsz, append, cu_q ? kv_append : bsz * append, nkv, pages, pages_per_seq, 0, 0};
    return attn_impl(ctx, (cudaStream_t)stream, p, total_rows, q_len, false, write ? &a : nullptr);
}

extern "C" int exl3_bighead_attn_paged_q(exl3_ctx* ctx, exl3_stream stream, const void* q, const void* k,
                                         const void* v, void* qk, void* sk, void* qv, void* sv,
                                         const int32_t* block_table, const int32_t* cache_seqlens, const int32_t* cu_q,
                                         void* o, int bsz, int q_len, int kv_append, int nq, int nkv, int hd, int pages,
                                         int pages_per_seq, int k_bits, int v_bits, int kv_chunk_size, int causal,
                                         float sm_scale, float compand_a)
{
    (void)kv_chunk_size;
    int rc = check_common(ctx, q, o, block_table, cache_seqlens, bsz, q_len, kv_append, nq, nkv, hd, pages, pages_per_seq);
    if (rc) return rc;
    EXL3_REQUIRE(qk && sk && qv && sv, "attention: null quantised pool");
    EXL3_REQUIRE(k_bits >= 2 && k_bits <= 8 && v_bits >= 2 && v_bits <= 8, "attention: bits must be 2..8");
    if (compand_a > 0.0f) return exl3_fail(ctx, EXL3_ERR_UNSUPPORTED, "attention: compand_a > 0 is not supported");
    if (bsz == 0 || q_len == 0) return EXL3_OK;
    EXL3_REQUIRE(quant_planes_aligned(qk, sk, qv, sv), "attention: code planes must be 16-byte and scale planes 8-byte aligned");
    const int append = cu_q ? q_len : kv_append;
    const bool write = append > 0 && !ctx->kv_appended;
    if (write) {
        EXL3_REQUIRE(k && v, "attention: kv_append > 0 needs k and v");
        EXL3_REQUIRE(bsz <= 65535 && append <= 65535, "quant_cache_paged: bad shape");
    }
    exl3_chain_scope chain(ctx, append > 0 && !write);
    AttnParams p;
    memset(&p, 0, sizeof(p));
    p.q = (const half*)q; p.o = (half*)o;
    p.qk = (const uint32_t*)qk; p.sk = (const half*)sk; p.qv = (const uint32_t*)qv; p.sv = (const half*)sv;
    p.block_table = block_table; p.seqlens = cache_seqlens; p.cu_q = cu_q;
    p.bsz = bsz; p.q_len = q_len; p.kv_append = kv_append; p.nq = nq; p.nkv = nkv; p.pps = pages_per_seq; p.pages = pages;
    p.causal = causal; p.k_bits = k_bits; p.v_bits = v_bits;
    p.scale_log2 = (sm_scale == 0.0f ? rsqrtf((float)hd) : sm_scale) * 1.4426950408889634f;
    const int total_rows = cu_q ? kv_append : bsz * q_len;
    const AttnAppendArgs a = {(const half*)k, (const half*)v, nullptr, nullptr, (uint32_t*)qk, (half*)sk, (uint32_t*)qv, (half*)sv, block_table, cache_seqlens, cu_q,
                              bsz, append, cu_q ? kv_append : bsz * append, nkv, pages, pages_per_seq, k_bits, v_bits};
    return attn_impl(ctx, (cudaStream_t)stream, p, total_rows, q_len, true, write ? &a : nullptr);
}

// Attention over plain tensors: q, o [bsz, q_len, nq, hd], k, v [bsz, kv_len, nkv, hd], no cache and no block table
// (kernels/attention.cu:2292-2437).  A causal query i sees keys <= kv_len - q_len + i (:1476).  Runs the mma.sync kernels
// with the key index taken straight from the sequence's base; kv_chunk_size is accepted and ignored (the split size comes
// from the work list).
extern "C" int exl3_bighead_attn(exl3_ctx* ctx, exl3_stream stream, const void* q, const void* k, const void* v, void* o,
                                 int bsz, int q_len, int kv_len, int nq, int nkv, int hd, int kv_chunk_size, int causal,
                                 float sm_scale)
{
    EXL3_REQUIRE(ctx && q && k && v && o, "attention: null argument");
    EXL3_REQUIRE(bsz >= 0 && q_len >= 0 && kv_len >= 0 && nq > 0 && nkv > 0, "attention: bad shape");
    EXL3_REQUIRE(kv_chunk_size > 0, "attention: kv_chunk_size must be positive");
    EXL3_REQUIRE(nq % nkv == 0, "attention: n_q_heads must be a multiple of n_kv_heads");
    EXL3_REQUIRE(nq / nkv <= 16, "attention: GQA ratio above 16");
    if (hd != 128) return exl3_fail(ctx, EXL3_ERR_UNSUPPORTED, "attention: head_dim must be 128");
    EXL3_REQUIRE(nkv <= 65535, "attention: too many kv heads");
    EXL3_REQUIRE(aligned16(q) && aligned16(o) && aligned16(k) && aligned16(v), "attention: pointers must be 16-byte aligned");
    if (bsz == 0 || q_len == 0) return EXL3_OK;
    if (kv_len == 0)                                      // nothing to attend to: the reference writes zeros (l = 0)
        return cudaMemsetAsync(o, 0, (size_t)bsz * q_len * nq * hd * 2, (cudaStream_t)stream) == cudaSuccess
                   ? EXL3_OK : exl3_fail(ctx, EXL3_ERR_CUDA, "attention: cudaMemsetAsync failed");
    AttnParams p;
    memset(&p, 0, sizeof(p));
    p.q = (const half*)q; p.o = (half*)o; p.kc = (const half*)k; p.vc = (const half*)v;
    p.bsz = bsz; p.q_len = q_len; p.kv_append = kv_len; p.contig_kv = kv_len; p.nq = nq; p.nkv = nkv; p.pps = 1; p.pages = 1;
    p.causal = causal;
    p.scale_log2 = (sm_scale == 0.0f ? rsqrtf((float)hd) : sm_scale) * 1.4426950408889634f;
    // the work lists kept across the layers of a step belong to the paged batch: plan afresh
    const int keep = ctx->plan_keep;
    ctx->plan_keep = 0;
    const int rc = attn_impl(ctx, (cudaStream_t)stream, p, bsz * q_len, q_len, false, nullptr);
    ctx->plan_keep = keep;
    return rc;
}
