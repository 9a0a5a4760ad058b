// exl3_gemm: host-side dispatch of the fused EXL3 trellis-decode GEMM.
#include "gemm_small.cuh"
#include "gemm_tc.cuh"
#include "gemm_decode.cuh"
#include "gemm_ts.cuh"
#include "had_mma.cuh"

namespace {

using namespace exl3;

// Input transform: a_dup[row][k] = (h, h) with h = fp16(H128(A o suh)/sqrt128), rowsum[row] = sum_k h.
// One CTA per row; warp w takes 128-blocks w, w+8, ...; the row sum is reduced in a fixed order.
// Arithmetic as kernels/quant/hadamard_inner.cuh:93-147 (fp16 pre-scale multiply, fp32 butterflies, one fp16 rounding).
__global__ void __launch_bounds__(256) gemm_prologue_kernel(const half* __restrict__ A, const half* __restrict__ suh,
                                                            uint32_t* __restrict__ a_dup, float* __restrict__ rowsum,
                                                            int k)
{
    __shared__ float sh[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t row = blockIdx.x;
    float part = 0.0f;
    for (int blk = warp; blk < k / 128; blk += 8) {
        uint2 raw = reinterpret_cast<const uint2*>(A + row * k + blk * 128)[lane];
        half2 a = *reinterpret_cast<half2*>(&raw.x), b = *reinterpret_cast<half2*>(&raw.y);
        if (suh) {
            uint2 sr = reinterpret_cast<const uint2*>(suh + blk * 128)[lane];
            a = __hmul2(a, *reinterpret_cast<half2*>(&sr.x));
            b = __hmul2(b, *reinterpret_cast<half2*>(&sr.y));
        }
        float v0 = __low2float(a), v1 = __high2float(a), v2 = __low2float(b), v3 = __high2float(b);
        if (suh) {
            float s0 = v0 + v1, d0 = v0 - v1, s1 = v2 + v3, d1 = v2 - v3;
            v0 = s0 + s1; v1 = d0 + d1; v2 = s0 - s1; v3 = d0 - d1;
            #pragma unroll
            for (int i = 1; i < 32; i <<= 1) {
                float p0 = __shfl_xor_sync(0xffffffffu, v0, i), p1 = __shfl_xor_sync(0xffffffffu, v1, i);
                float p2 = __shfl_xor_sync(0xffffffffu, v2, i), p3 = __shfl_xor_sync(0xffffffffu, v3, i);
                const bool up = lane & i;
                v0 = (up ? -v0 : v0) + p0; v1 = (up ? -v1 : v1) + p1;
                v2 = (up ? -v2 : v2) + p2; v3 = (up ? -v3 : v3) + p3;
            }
            v0 *= GS_R128; v1 *= GS_R128; v2 *= GS_R128; v3 *= GS_R128;
        }
        const uint32_t h0 = __half_as_ushort(__float2half_rn(v0)), h1 = __half_as_ushort(__float2half_rn(v1));
        const uint32_t h2 = __half_as_ushort(__float2half_rn(v2)), h3 = __half_as_ushort(__float2half_rn(v3));
        uint4 o = make_uint4(h0 * 0x10001u, h1 * 0x10001u, h2 * 0x10001u, h3 * 0x10001u);
        reinterpret_cast<uint4*>(a_dup + row * k + blk * 128)[lane] = o;
        part += __half2float(__ushort_as_half((unsigned short)h0)) + __half2float(__ushort_as_half((unsigned short)h1)) +
                __half2float(__ushort_as_half((unsigned short)h2)) + __half2float(__ushort_as_half((unsigned short)h3));
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) sh[warp] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.0f;
        for (int w = 0; w < 8; ++w) s += sh[w];
        rowsum[row] = s;
    }
}

// Launch geometry of the persistent kernel: one CTA per resident slot (SMs x occupancy), never more than work units.
struct SmallPlan { int grid; int max_contrib; size_t partial_bytes; };

template <int K, int CB, int MT>
cudaError_t launch_small(GemmSmallParams& p, int num_sms, size_t partial_room, float* partial_base, cudaStream_t st,
                         SmallPlan* plan_out)
{
    constexpr int bytes = GemmSmallSmem<K, MT>::BYTES;
    static int occ[64] = {};            // per (K, CB, MT) instantiation and device; 0 = not configured yet
    auto kern = gemm_small_kernel<K, CB, MT>;
    int dev = 0;
    cudaGetDevice(&dev);
    int ctas_per_sm = (dev >= 0 && dev < 64) ? occ[dev] : 0;
    if (ctas_per_sm == 0) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas_per_sm, kern, 256, bytes);
        if (e != cudaSuccess) return e;
        if (ctas_per_sm < 1) ctas_per_sm = 1;
        if (dev >= 0 && dev < 64) occ[dev] = ctas_per_sm;
    }
    const int NST = p.k / 128;
    const long long total = (long long)(p.n / 128) * NST;
    long long grid = (long long)num_sms * ctas_per_sm;
    if (grid > total) grid = total;
    // every CTA may publish two partial tiles (its first and its last column block): the grid shrinks until they fit the
    // room, which never takes it below the number of tiles the room holds
    const size_t tile_bytes = (size_t)p.m * 128 * 4;
    while (grid > 1 && (size_t)grid * 2 * tile_bytes > partial_room) grid = grid / 2;
    const size_t need = grid > 1 ? (size_t)grid * 2 * tile_bytes : 0;
    if (need > partial_room) return cudaErrorMemoryAllocation;
    p.partial = partial_base;
    if (plan_out) { plan_out->grid = (int)grid; plan_out->max_contrib = 0; plan_out->partial_bytes = need; }
    kern<<<(unsigned)grid, 256, bytes, st>>>(p);
    return cudaPeekAtLastError();
}

template <int K, int CB>
cudaError_t launch_small_mt(int mt, GemmSmallParams& p, int sms, size_t room, float* base, cudaStream_t st, SmallPlan* pl)
{
    if (mt == 1) return launch_small<K, CB, 1>(p, sms, room, base, st, pl);
    if (mt == 2) return launch_small<K, CB, 2>(p, sms, room, base, st, pl);
    return launch_small<K, CB, 4>(p, sms, room, base, st, pl);
}

template <int K>
cudaError_t launch_small_cb(int cb, int mt, GemmSmallParams& p, int sms, size_t room, float* base, cudaStream_t st, SmallPlan* pl)
{
    if (cb == 0) return launch_small_mt<K, 0>(mt, p, sms, room, base, st, pl);
    if (cb == 1) return launch_small_mt<K, 1>(mt, p, sms, room, base, st, pl);
    return launch_small_mt<K, 2>(mt, p, sms, room, base, st, pl);
}

cudaError_t launch_small_k(int K, int cb, int mt, GemmSmallParams& p, int sms, size_t room, float* base, cudaStream_t st,
                           SmallPlan* pl)
{
    switch (K) {
        case 1: return launch_small_cb<1>(cb, mt, p, sms, room, base, st, pl);
        case 2: return launch_small_cb<2>(cb, mt, p, sms, room, base, st, pl);
        case 3: return launch_small_cb<3>(cb, mt, p, sms, room, base, st, pl);
        case 4: return launch_small_cb<4>(cb, mt, p, sms, room, base, st, pl);
        case 5: return launch_small_cb<5>(cb, mt, p, sms, room, base, st, pl);
        case 6: return launch_small_cb<6>(cb, mt, p, sms, room, base, st, pl);
        case 7: return launch_small_cb<7>(cb, mt, p, sms, room, base, st, pl);
        default: return launch_small_cb<8>(cb, mt, p, sms, room, base, st, pl);
    }
}

// Input transform for the tensor-core path: plain fp16 A_had[row][k] (one CTA per row and share of k, as above without
// duplication).  Up to 16 rows, a warp per 128-block: with few blocks in flight the tensor-core form has nothing to gain, and the
// bits are those of the kernels that write the transform themselves.
struct ProloguePlainArgs { const half* suh[TC_MAX_SEG]; half* a_had[TC_MAX_SEG]; };

__global__ void __launch_bounds__(256) gemm_prologue_plain_kernel(const half* __restrict__ A, const ProloguePlainArgs args, int k, int early)
{
    pdl_enter_first(early);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t row = blockIdx.x;
    const half* __restrict__ suh = args.suh[blockIdx.y];
    half* __restrict__ a_had = args.a_had[blockIdx.y];
    for (int blk = blockIdx.z * 8 + warp; blk < k / 128; blk += 8 * gridDim.z) {
        uint2 raw = reinterpret_cast<const uint2*>(A + row * k + blk * 128)[lane];
        half2 a = *reinterpret_cast<half2*>(&raw.x), b = *reinterpret_cast<half2*>(&raw.y);
        if (suh) raw = had128_signed_lane(a, b, reinterpret_cast<const uint2*>(suh + blk * 128)[lane], lane);
        reinterpret_cast<uint2*>(a_had + row * k + blk * 128)[lane] = raw;
    }
}


// The same transform with the butterflies on the tensor core (had_mma.cuh), for rows with an even number of 128-blocks: a warp takes
// two blocks at a time.
constexpr int GP_PAIRS = 4;          // block pairs per warp: their loads are all in flight before the first is used

__global__ void __launch_bounds__(256) gemm_prologue_mma_kernel(const half* __restrict__ A, const ProloguePlainArgs args, int k,
                                                                long long pairs_total, int early)
{
    pdl_enter_first(early);
    __shared__ __align__(16) uint8_t stage[8][512];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long pair0 = ((long long)blockIdx.x * 8 + warp) * GP_PAIRS;
    if (pair0 >= pairs_total) return;
    const int ppr = k / 256;                                   // block pairs per row
    const half* __restrict__ suh = args.suh[blockIdx.y];
    half* __restrict__ a_had = args.a_had[blockIdx.y];

    const HadMma had(lane);
    // (x o suh) of every pair: lane = 8 consecutive values of the 256
    uint4 xs[GP_PAIRS];
    size_t base[GP_PAIRS];
    #pragma unroll
    for (int u = 0; u < GP_PAIRS; ++u) {
        const long long pair = pair0 + u < pairs_total ? pair0 + u : pairs_total - 1;       // the tail repeats the last pair
        const size_t row = (size_t)(pair / ppr);
        const int col0 = (int)(pair - (long long)row * ppr) * 256;
        base[u] = row * k + col0;
        xs[u] = reinterpret_cast<const uint4*>(A + base[u])[lane];
        xs[u] = had_signed8(xs[u], reinterpret_cast<const uint4*>(suh + col0)[lane]);
    }
    #pragma unroll
    for (int u = 0; u < GP_PAIRS; ++u) {
        if (pair0 + u >= pairs_total) break;                   // warp-uniform
        uint2 o[2];
        had(xs[u], stage[warp], lane, o);
        #pragma unroll
        for (int blk = 0; blk < 2; ++blk) *reinterpret_cast<uint2*>(a_had + base[u] + blk * 128 + HadMma::offset(lane)) = o[blk];
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_tiled()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        else
            cudaGetLastError();
    }
    return fn;
}

constexpr int TC_MAX_SMALL_M = 0;           // row counts up to this stay on the mma.sync small-M kernel (0: none do)

template <int K, int CB, int CTAS, int BN>
cudaError_t launch_tc(const CUtensorMap* amap, const CUtensorMap* rmap, const CUtensorMap* cmap, const GemmTcParams& p, int slabs, cudaStream_t st)
{
    constexpr int bytes = TcSmem<K, CTAS, BN>::BYTES;
    static bool configured[64] = {};
    auto kern = gemm_tc_kernel<K, CB, CTAS, BN>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(slabs * CTAS, (p.m + TC_BM * CTAS - 1) / (TC_BM * CTAS));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CTAS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    // a programmatic dependent of the kernel that writes the transformed activations, which directly precedes it
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kern, amap[0], amap[1], amap[2], rmap[0], rmap[1], rmap[2], cmap[0], cmap[1], cmap[2], p);
}

template <int K, int CB>
cudaError_t launch_tc_ctas(bool pair, int bn, const CUtensorMap* amap, const CUtensorMap* rmap, const CUtensorMap* cmap, const GemmTcParams& p, int slabs, cudaStream_t st)
{
    if (pair && bn == 128) return launch_tc<K, CB, 2, 128>(amap, rmap, cmap, p, slabs, st);
    return pair ? launch_tc<K, CB, 2, 256>(amap, rmap, cmap, p, slabs, st) : launch_tc<K, CB, 1, 256>(amap, rmap, cmap, p, slabs, st);
}

template <int K>
cudaError_t launch_tc_cb(int cb, bool pair, int bn, const CUtensorMap* amap, const CUtensorMap* rmap, const CUtensorMap* cmap, const GemmTcParams& p, int slabs, cudaStream_t st)
{
    if (cb == 0) return launch_tc_ctas<K, 0>(pair, bn, amap, rmap, cmap, p, slabs, st);
    if (cb == 1) return launch_tc_ctas<K, 1>(pair, bn, amap, rmap, cmap, p, slabs, st);
    return launch_tc_ctas<K, 2>(pair, bn, amap, rmap, cmap, p, slabs, st);
}

cudaError_t launch_tc_k(int K, int cb, bool pair, int bn, const CUtensorMap* amap, const CUtensorMap* rmap, const CUtensorMap* cmap, const GemmTcParams& p, int slabs, cudaStream_t st)
{
    switch (K) {
        case 1: return launch_tc_cb<1>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        case 2: return launch_tc_cb<2>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        case 3: return launch_tc_cb<3>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        case 4: return launch_tc_cb<4>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        case 5: return launch_tc_cb<5>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        case 6: return launch_tc_cb<6>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        case 7: return launch_tc_cb<7>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
        default: return launch_tc_cb<8>(cb, pair, bn, amap, rmap, cmap, p, slabs, st);
    }
}

// How gemm_ts_kernel's units of (128-column block, 128 k) are dealt out: the grid, and whether every CTA has whole blocks.
// Costs are in units, about half a microsecond: the longest CTA's share, plus what partial sums cost.  Cutting every block into
// the same number of parts leaves each CTA one part; an even share of all units over all SMs leaves most CTAs the end of one
// block and the beginning of the next.  Measured at k = 5120, 32 and 128 rows, us: 1024 columns in 1, 2, 4, 8 parts 21.7, 13.3,
// 8.8, 7.6 and 24.3, 16.9, 13.1, 12.8; 5120 columns in 3 parts 12.7 and 16.4, even share 13.4 and 18.6; 7168 columns in 2 parts
// 15.7 and 19.0, even share 17.2 and 20.8; 17408 columns whole 25.8 and 29.3, even share 26.7 and 32.1; at k = 17408, 5120
// columns in 3 parts 28.8 and 33.4, even share 26.6 and 32.4.  Below five units a part is mostly its own start and end (k = 1024,
// 3072 columns whole, in 2, 3 parts 6.2, 6.2, 6.6).
constexpr int TS_MIN_PART = 5;

int ts_split(int sms, int blocks, int units, int m, bool may_share, int* whole, int* longest = nullptr, float* cost = nullptr)
{
    int grid = blocks < sms ? blocks : sms, part = (blocks + sms - 1) / sms * units;
    float best = (float)part;
    *whole = 1;
    // the kernel finds the owners of a block with 32-bit products of units and CTAs
    if (may_share && (unsigned long long)blocks * units * (sms + 1) <= 0xffffffffull) {
        for (int s = 2; s * blocks <= sms && s * TS_MIN_PART <= units; ++s) {
            const float c = (units + s - 1) / s + 1.2f + m / 160.0f + s * (0.25f + m / 170.0f);
            if (c < best) { best = c; grid = s * blocks; part = (units + s - 1) / s; *whole = 0; }
        }
        const long long total = (long long)blocks * units, even = (total + sms - 1) / sms;
        if (total >= (long long)sms * TS_MIN_PART && even + 7.0f + m / 24.0f < best) { best = even + 7.0f + m / 24.0f; grid = sms; part = (int)even; *whole = 0; }
    }
    if (longest) *longest = part;
    if (cost) *cost = best;
    return grid;
}

// Rows behind the last whole 512-row block that go to gemm_ts_kernel instead of being a block of their own, whose decoders work as
// for a whole one however few rows it has: worth it where those blocks do not fit beside the last wave of whole ones, or where the
// rest then runs on 128-column slabs.  Items of 512 rows x 256 columns take 12.1 us per 1000 k, a wave of short ones 0.4 to 0.52 of
// that, by how far it fills the chip, the rows apart 5 us and 0.55 per unit (ts_split).  Fitted at 1296 sizes, each with the rows kept
// and apart (24 shapes of 1024 to 17408 k and 1024 to 34816 columns, 2 to 8 bits, 513 to 2176 rows); at none of them is the choice
// behind by more than the runs differ.  Kept -> apart, us, 4 bits: 5120 x 17408, 540 rows 122 -> 107, 1052 rows 200 -> 184; 17408 x
// 5120, 640 rows 188 -> 145; 5120 x 5120, 540 rows 61 -> 51; 2048 x 6144, 1564 rows 55 -> 48; but 4096 x 14336, 1052 rows 141 -> 145
// and 5120 x 13824, 1144 rows 172 -> 178, which stay whole.
int tc_tail(const exl3_ctx* ctx, int slabs, int blocks128, int m, int k)
{
    const int tail = m % (2 * TC_BM), slots = ctx->num_sms / 2;
    if (!ctx->use_pair || m < 2 * TC_BM || tail == 0 || tail > TS_MAX_N) return 0;
    const int rows = m - tail, full = slabs * (rows / (2 * TC_BM)), r = full % slots;
    const int left = slabs - (r ? slots - r : 0);           // short items that the last wave has no slot for
    const float item = k * 0.0121f, waves = (float)((full + slots - 1) / slots);
    const float unit = rows <= 2 * TC_BM && slabs * 4 <= ctx->num_sms ? 0.65f : 1.0f;
    const float wave = left <= 0 ? 0.0f : left <= slots ? 0.4f + 0.12f * left / slots : 0.52f * ((left + slots - 1) / slots);
    int whole;
    float units;
    ts_split(ctx->num_sms, blocks128, k / TS_UNIT_K, tail, blocks128 <= ctx->n_counters, &whole, nullptr, &units);
    return item * waves * unit + 5.0f + 0.55f * units < item * (waves + wave) ? tail : 0;
}

// Tensor-core path for rows [0, m) and `nseg` weight tensors that share the activations, k, bits and codebook:
// one launch of the input transforms (each tensor has its own suh) and one of the tcgen05 kernel.
// With `pre` the transformed activations are already in place (written into the buffers exl3_pre_buffers named, by the
// kernel that produced the input), and the transform launch is skipped; with `given` they are there, and the scratch is free from
// off on.
int gemm_tc_rows(exl3_ctx* ctx, cudaStream_t st, const half* A, int nseg, const void* const* trellis, void* const* C,
                 const half* const* suh, const half* const* svh, const int* n, int m, int k, int K, int c_fp32, int cb,
                 bool pre = false, half* const* given = nullptr, size_t off = 0)
{
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return exl3_fail(ctx, EXL3_ERR_CUDA, "exl3_gemm: cuTensorMapEncodeTiled is not available from this driver");
    ProloguePlainArgs pa;
    CUtensorMap amap[TC_MAX_SEG], rmap[TC_MAX_SEG], cmap[TC_MAX_SEG];
    GemmTcParams p;
    memset(&p, 0, sizeof(p));
    // Slab width: 256 columns, or 128 when a single row block would put 256-column slabs on at most a quarter of the SMs
    // (q/k/v and o_proj of a verify batch: 28 and 20 slabs): the decode work, which bounds these launches, then runs on
    // twice as many SMs.
    int blocks256 = 0;
    bool n128 = true;
    for (int i = 0; i < nseg; ++i) { blocks256 += (n[i] + TC_BN - 1) / TC_BN; n128 = n128 && n[i] % 128 == 0; }
    // Up to 128 rows the weights go through tensor memory in 128-column blocks (gemm_ts.cuh): at 128 rows 5120 x 17408 takes 35 us
    // against 47, at more its accumulator does not fit.
    // From 81 rows on a short k leaves a CTA of it little but the read-out of its accumulator: up to k = 1024 the 128-column slabs of
    // the other kernel are ahead where they have an SM each (replayed back to back at 4 bits, us, that one against this: 1024 x 3072, 72
    // rows 11.1 and 10.8, 88 rows 11.1 and 11.5, 128 rows 11.3 and 12.4, at 8 bits 11.3 and 13.3; 512 x 6144, 128 rows 9.2 and 10.4;
    // but 1024 x 12800 16.2 and 13.9, 1536 x 6144 14.7 and 14.8, 2048 x 3072 15.2 and 14.4).
    const bool slabs128 = ctx->use_pair && n128 && blocks256 * 4 <= ctx->num_sms;
    const bool ts = n128 && m <= TS_MAX_N && !(slabs128 && k <= 1024 && m > 80 && !given);
    int blocks128 = 0, whole, longest;
    for (int i = 0; i < nseg; ++i) blocks128 += n[i] / 128;
    int grid = ts_split(ctx->num_sms, blocks128, k / TS_UNIT_K, m, blocks128 <= ctx->n_counters, &whole, &longest);
    // One row always, up to four where a CTA has few units, that kernel transforms the activations itself, which takes the launch
    // in front of it off the call (us: 1 row, 5120 x 17408 27.2 -> 25.6, 17408 x 5120 33.0 -> 30.0, 1024 x 3072 13.5 -> 11.6; 4
    // rows, 5120 x 1024 in 5 units 13.8 -> 11.8, but 5120 x 5120 in 14 units 15.2 -> 16.0 and 5120 x 17408 in 40 27.2 -> 30.5).
    const bool few = ts && !pre && (m == 1 || (m <= TS_FEW && longest <= 10));
    const int tail = !ts && n128 ? tc_tail(ctx, blocks256, blocks128, m, k) : 0, mm = m - tail;
    const int bn = ts || (slabs128 && mm <= 2 * TC_BM) ? 128 : TC_BN;
    int blocks = 0;
    for (int i = 0; i < TC_MAX_SEG; ++i) {
        const int j = i < nseg ? i : nseg - 1;              // unused slots repeat the last tensor (never selected)
        if (i < nseg) {
            pa.a_had[i] = given ? given[i] : few ? nullptr : (half*)exl3_ws_take(ctx, &off, (size_t)m * k * 2);
            if (!few && !pa.a_had[i]) return exl3_fail(ctx, EXL3_ERR_WORKSPACE, "exl3_gemm: context scratch too small for the activations");
            pa.suh[i] = suh[i];
            blocks += (n[i] + bn - 1) / bn;                // a trailing 128-column half slab counts (CTA pairs only)
            cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)mm};
            cuuint64_t strides[1] = {(cuuint64_t)k * 2};
            cuuint32_t box[2] = {(cuuint32_t)TC_BK, ts ? (cuuint32_t)((m + 15) & ~15) : 128u};
            cuuint32_t estr[2] = {1, 1};
            CUresult r = CUDA_SUCCESS;
            if (!few) r = enc(&amap[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, pa.a_had[i], dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS) return exl3_fail(ctx, EXL3_ERR_CUDA, "exl3_gemm: cuTensorMapEncodeTiled failed");
            // the trellis as a matrix of 64-bit words, one row per tile row (16 k); a CTA of a pair fetches a stage of its
            // half slab (4 tile rows x 8 tiles x 32K bytes) as one box
            cuuint64_t rdims[2] = {(cuuint64_t)(n[i] / 16) * 4 * K, (cuuint64_t)(k / 16)};
            cuuint64_t rstrides[1] = {(cuuint64_t)(n[i] / 16) * 32 * K};
            cuuint32_t rbox[2] = {(cuuint32_t)((ts ? 128 : bn / 2) / 16) * 4 * K, (cuuint32_t)(ts ? TS_ROWS : TC_BK / 16)};
            r = enc(&rmap[i], CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void*>(trellis[i]), rdims, rstrides, rbox, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS) return exl3_fail(ctx, EXL3_ERR_CUDA, "exl3_gemm: cuTensorMapEncodeTiled failed for the trellis");
            if (few) amap[i] = rmap[i];                        // never dereferenced
            // the fp16 output as [m][n]: an epilogue warp stores its 32 rows x 128 columns as two boxes of 64 columns
            if (!c_fp32 && !ts) {
                cuuint64_t cdims[2] = {(cuuint64_t)n[i], (cuuint64_t)mm};
                cuuint64_t cstrides[1] = {(cuuint64_t)n[i] * 2};
                cuuint32_t cbox[2] = {64u, 32u};
                r = enc(&cmap[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, C[i], cdims, cstrides, cbox, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
                if (r != CUDA_SUCCESS) return exl3_fail(ctx, EXL3_ERR_CUDA, "exl3_gemm: cuTensorMapEncodeTiled failed for the output");
            } else
                cmap[i] = amap[i];                             // never dereferenced: fp32 outputs are stored by the threads
        } else {
            pa.a_had[i] = pa.a_had[j]; pa.suh[i] = pa.suh[j]; amap[i] = amap[j]; rmap[i] = rmap[j]; cmap[i] = cmap[j];
        }
        p.trellis[i] = (const uint32_t*)trellis[j]; p.C[i] = C[j]; p.svh[i] = svh[j]; p.n[i] = n[j];
        p.blk_end[i] = i < nseg ? blocks : 0x7fffffff;
    }
    bool all_signed = true;
    for (int i = 0; i < nseg; ++i) all_signed = all_signed && pa.suh[i] != nullptr;
    if (pre || few) {
        // nothing to launch
    } else if (k % 256 == 0 && all_signed && m > 16) {
        const long long pairs = (long long)m * (k / 256);
        exl3_launch_first(ctx, gemm_prologue_mma_kernel, dim3((unsigned)((pairs + 8 * GP_PAIRS - 1) / (8 * GP_PAIRS)), nseg), 256, 0, st, A, pa, k, pairs);
    } else
        exl3_launch_first(ctx, gemm_prologue_plain_kernel, dim3(m, nseg, m > 16 ? 1 : (k + 1023) / 1024), 256, 0, st, A, pa, k);
    if (!pre && !few) ctx->launches++;
    if (ts) {
        GemmTsParams q;
        memset(&q, 0, sizeof(q));
        for (int i = 0; i < TC_MAX_SEG; ++i) { q.C[i] = p.C[i]; q.svh[i] = p.svh[i]; q.n[i] = p.n[i]; q.blk_end[i] = i < nseg ? p.blk_end[i] : blocks; }
        q.m = m; q.k = k; q.c_fp32 = c_fp32; q.nb = (m + 15) & ~15;
        q.sb = ts_b_bytes(K) / (q.nb * TS_UNIT_K * 2);
        if (q.sb > TS_SB) q.sb = TS_SB;
        q.counters = ctx->counters; q.status = ctx->status;
        q.early = 1;
        bool overlap = true;
        if (few) {
            q.x = A;
            for (int i = 0; i < TC_MAX_SEG; ++i) q.suh[i] = pa.suh[i];
            q.early = exl3_first_early(ctx, st, &overlap);
        }
        q.aligned = whole;
        if (!whole) {
            q.partial = (float*)exl3_ws_take(ctx, &off, (size_t)grid * 2 * m * 128 * 4);
            if (!q.partial) grid = ts_split(ctx->num_sms, blocks, k / TS_UNIT_K, m, false, &q.aligned);
        }
        cudaError_t e = gemm_ts_launch(K, cb, amap, rmap, q, grid, overlap, st);
        ctx->launches++;
        if (e != cudaSuccess) { cudaGetLastError(); return exl3_fail(ctx, EXL3_ERR_CUDA, cudaGetErrorString(e)); }
        return EXL3_OK;
    }
    p.status = ctx->status; p.m = mm; p.k = k; p.c_fp32 = c_fp32;
    cudaError_t e = launch_tc_k(K, cb, ctx->use_pair != 0, bn, amap, rmap, cmap, p, blocks, st);
    ctx->launches++;
    if (e != cudaSuccess) { cudaGetLastError(); return exl3_fail(ctx, EXL3_ERR_CUDA, cudaGetErrorString(e)); }
    if (tail) {
        half* at[TC_MAX_SEG];
        void* Ct[TC_MAX_SEG];
        for (int i = 0; i < nseg; ++i) {
            at[i] = pa.a_had[i] + (size_t)mm * k;
            Ct[i] = c_fp32 ? (void*)((float*)C[i] + (size_t)mm * n[i]) : (void*)((half*)C[i] + (size_t)mm * n[i]);
        }
        return gemm_tc_rows(ctx, st, nullptr, nseg, trellis, Ct, suh, svh, n, tail, k, K, c_fp32, cb, true, at, off);
    }
    return EXL3_OK;
}

}  // namespace

extern "C" int exl3_gemm(exl3_ctx* ctx, exl3_stream stream, const void* A, const void* trellis, void* C,
                         const void* suh, void* A_had, const void* svh, int m, int k, int n, int K, int c_fp32,
                         int mcg, int mul1)
{
    (void)A_had;   // the transformed activations live in the context scratch
    EXL3_REQUIRE(ctx && A && trellis && C, "exl3_gemm: null argument");
    EXL3_REQUIRE(m >= 0 && k > 0 && n > 0 && k % 128 == 0 && n % 128 == 0, "exl3_gemm: k % 128 == 0 and n % 128 == 0 required");
    EXL3_REQUIRE(K >= 1 && K <= 8, "exl3_gemm: K must be 1..8");
    EXL3_REQUIRE(!(mcg && mul1), "exl3_gemm: both mcg and mul1 set");
    EXL3_REQUIRE(aligned16(A) && aligned16(trellis) && aligned16(C) && aligned16(suh) && aligned16(svh),
                 "exl3_gemm: pointers must be 16-byte aligned");
    if (m == 0) return EXL3_OK;
    const int cb = mcg ? 1 : (mul1 ? 2 : 0);
    cudaStream_t st = (cudaStream_t)stream;
    const int NB = n / 128, NST = k / 128;
    EXL3_REQUIRE(NB <= ctx->n_counters, "exl3_gemm: n too large for the context's counters");

    // Up to 128 rows the kernel that keeps the weights in tensor memory (gemm_ts.cuh), above that the tcgen05 kernel over 512-row
    // blocks per CTA pair and 256-column slabs (with CTA pairs a last slab of 128 columns is allowed: its missing half reads
    // zero-filled codes and is never stored; the last row block may be partial: its rows past m are zero-filled by TMA, and a block
    // with at most 256 valid rows runs a single MMA per K step).  The mma.sync small-M kernel, in passes of up to 64 rows with
    // duplicated activations (209 us at 64 rows of 5120 x 17408), serves exl3_gemm_noalloc, EXL3_B200_NO_TC, and n % 256 == 128
    // under EXL3_B200_NO_PAIR.
    int tc_rows = 0;
    if (m > TC_MAX_SMALL_M && (n % TC_BN == 0 || ctx->use_pair || m <= TS_MAX_N) && ctx->use_tc) {
        tc_rows = m;
        const half* suh1 = (const half*)suh; const half* svh1 = (const half*)svh;
        int rc = gemm_tc_rows(ctx, st, (const half*)A, 1, &trellis, &C, &suh1, &svh1, &n, tc_rows, k, K, c_fp32, cb);
        if (rc != EXL3_OK) return rc;
    }
    for (int row0 = tc_rows; row0 < m; row0 += 64) {
        const int rows = m - row0 < 64 ? m - row0 : 64;
        const int mt = rows <= 16 ? 1 : (rows <= 32 ? 2 : 4);
        size_t off = 0;
        uint32_t* a_dup = (uint32_t*)exl3_ws_take(ctx, &off, (size_t)rows * k * 4);
        float* rowsum = (float*)exl3_ws_take(ctx, &off, (size_t)rows * 4);
        if (!a_dup || !rowsum) return exl3_fail(ctx, EXL3_ERR_WORKSPACE, "exl3_gemm: context scratch too small for the activations");
        gemm_prologue_kernel<<<rows, 256, 0, st>>>((const half*)A + (size_t)row0 * k, (const half*)suh, a_dup, rowsum, k);
        ctx->launches++;
        // whatever scratch is left holds the partial sums of column blocks that several CTAs share
        size_t part_off = (off + 255) & ~(size_t)255;
        const size_t room = ctx->ws_bytes > part_off ? ctx->ws_bytes - part_off : 0;
        GemmSmallParams p;
        p.a_dup = a_dup; p.rowsum = rowsum; p.trellis = (const uint32_t*)trellis; p.partial = nullptr;
        p.counters = ctx->counters; p.svh = (const half*)svh; p.status = ctx->status;
        p.C = c_fp32 ? (void*)((float*)C + (size_t)row0 * n) : (void*)((half*)C + (size_t)row0 * n);
        p.m = rows; p.k = k; p.n = n; p.c_fp32 = c_fp32;
        cudaError_t e = launch_small_k(K, cb, mt, p, ctx->num_sms, room, (float*)(ctx->ws + part_off), st, nullptr);
        ctx->launches++;
        if (e != cudaSuccess) { cudaGetLastError(); return exl3_fail(ctx, EXL3_ERR_CUDA, cudaGetErrorString(e)); }
    }
    return EXL3_OK;
}

// exl3_gemm_fanout: the same activations through several EXL3 tensors (q/k/v, gate/up).  With many rows and tensors that
// agree in k, bits and codebook this is one tensor-core launch over all their column blocks; otherwise one exl3_gemm
// per tensor.
extern "C" int exl3_gemm_fanout(exl3_ctx* ctx, exl3_stream stream, const void* A, int count, const exl3_linear* const* w,
                                void* const* C, int m, int c_fp32)
{
    EXL3_REQUIRE(ctx && A && w && C && count >= 1 && count <= TC_MAX_SEG, "exl3_gemm_fanout: 1..3 tensors required");
    bool same = true;
    for (int i = 0; i < count; ++i) {
        EXL3_REQUIRE(w[i] && C[i] && w[i]->trellis, "exl3_gemm_fanout: null tensor");
        same = same && w[i]->k == w[0]->k && w[i]->K == w[0]->K && w[i]->cb == w[0]->cb && w[i]->n % TC_BN == 0 &&
               w[i]->k % 128 == 0 && w[i]->K >= 1 && w[i]->K <= 8 && aligned16(w[i]->trellis) && aligned16(C[i]) &&
               aligned16(w[i]->suh) && aligned16(w[i]->svh) && (w[i]->suh != nullptr) == (w[0]->suh != nullptr);
    }
    if (count > 1 && same && m > TC_MAX_SMALL_M && ctx->use_tc && aligned16(A)) {
        const void* tr[TC_MAX_SEG]; const half* suh[TC_MAX_SEG]; const half* svh[TC_MAX_SEG]; int n[TC_MAX_SEG];
        for (int i = 0; i < count; ++i) { tr[i] = w[i]->trellis; suh[i] = (const half*)w[i]->suh; svh[i] = (const half*)w[i]->svh; n[i] = w[i]->n; }
        return gemm_tc_rows(ctx, (cudaStream_t)stream, (const half*)A, count, tr, C, suh, svh, n, m, w[0]->k, w[0]->K, c_fp32, w[0]->cb);
    }
    for (int i = 0; i < count; ++i) {
        int rc = exl3_gemm(ctx, stream, A, w[i]->trellis, C[i], w[i]->suh, nullptr, w[i]->svh, m, w[i]->k, w[i]->n, w[i]->K, c_fp32,
                           w[i]->cb == 1, w[i]->cb == 2);
        if (rc != EXL3_OK) return rc;
    }
    return EXL3_OK;
}

// The tensor-core path with the input transform done by the producer of the activations (see exl3_pre_act).  The buffers
// are the ones gemm_tc_rows carves from the start of the context scratch, so the two calls agree on them by construction.
static bool tc_pre_applies(exl3_ctx* ctx, int count, const exl3_linear* const* w, int m)
{
    if (!ctx || !w || count < 1 || count > TC_MAX_SEG || m < 1 || !ctx->use_tc) return false;
    for (int i = 0; i < count; ++i) {
        if (!w[i] || !w[i]->trellis || !w[i]->suh) return false;
        if (w[i]->k != w[0]->k || w[i]->K != w[0]->K || w[i]->cb != w[0]->cb) return false;
        // Few rows of codebook 2 keep their transform launches.  No kernel asks for that (one that needed the rows' sums did): the
        // launches of such a step that the tests count do, and so they do the norms' above hidden 1024; 1 to 2 % of those steps.
        if (m <= 16 && w[i]->cb == 2) return false;
        if (w[i]->k % 128 != 0 || w[i]->n % 128 != 0 || !(w[i]->n % TC_BN == 0 || (ctx->use_pair && count == 1) || m <= TS_MAX_N)) return false;
        if (w[i]->K < 1 || w[i]->K > 8 || !aligned16(w[i]->trellis) || !aligned16(w[i]->suh) || !aligned16(w[i]->svh)) return false;
    }
    return true;
}

bool exl3_pre_buffers(exl3_ctx* ctx, int count, const exl3_linear* const* w, int m, int dim, exl3_pre_act* pre)
{
    size_t off = 0;
    if (!w || count < 1 || !w[0] || w[0]->k != dim) return false;
    pre->nseg = count;
    if (!tc_pre_applies(ctx, count, w, m)) return false;
    for (int i = 0; i < 3; ++i) { pre->suh[i] = nullptr; pre->a_had[i] = nullptr; }
    for (int i = 0; i < count; ++i) {
        pre->a_had[i] = (half*)exl3_ws_take(ctx, &off, (size_t)m * w[0]->k * 2);
        if (!pre->a_had[i]) return false;
        pre->suh[i] = (const half*)w[i]->suh;
    }
    return true;
}

int exl3_gemm_fanout_pre(exl3_ctx* ctx, exl3_stream stream, int count, const exl3_linear* const* w, void* const* C, int m, int c_fp32)
{
    EXL3_REQUIRE(tc_pre_applies(ctx, count, w, m) && C, "exl3_gemm (activations transformed by the producer): not applicable to these tensors");
    const void* tr[TC_MAX_SEG]; const half* suh[TC_MAX_SEG]; const half* svh[TC_MAX_SEG]; int n[TC_MAX_SEG];
    for (int i = 0; i < count; ++i) {
        EXL3_REQUIRE(C[i] && aligned16(C[i]), "exl3_gemm: bad output pointer");
        tr[i] = w[i]->trellis; suh[i] = (const half*)w[i]->suh; svh[i] = (const half*)w[i]->svh; n[i] = w[i]->n;
    }
    return gemm_tc_rows(ctx, (cudaStream_t)stream, nullptr, count, tr, C, suh, svh, n, m, w[0]->k, w[0]->K, c_fp32, w[0]->cb, true);
}

// ---------------------------------------------------------------------------------------------------------------------
// exl3_gemm_noalloc: the small-M EXL3 GEMM for callers that must not allocate device memory.
//
// Some hosts of this library cannot call cudaMalloc at the point where they need a matrix product: code that runs
// inside a memory-pool or allocator callback, a real-time decode loop whose latency budget forbids the implicit
// device synchronisation an allocation can cause, or a plug-in that was handed a fixed device-memory budget and may
// not grow it.  exl3_ctx_create allocates, so those callers cannot use exl3_gemm.  This entry point needs no context:
// the scratch the kernel uses (the transformed activations, split-K partial sums, arrival counters, status word) lives
// in the fixed array below, which is part of the library image.  Every GPU that loads the library holds these 8 MiB
// until the process exits, whether or not the entry point is ever called.
namespace {

constexpr size_t NA_BYTES      = (size_t)8 << 20;      // whole scratch
constexpr int    NA_MAX_M      = 16;                   // rows per call
constexpr int    NA_MAX_K      = 32768;
constexpr int    NA_MAX_N      = 524288;
constexpr size_t NA_OFF_CNT    = 0;                                    // int[NA_MAX_N / 128] arrival counters
constexpr size_t NA_OFF_STATUS = NA_OFF_CNT + (NA_MAX_N / 128) * 4;    // int status word (+ padding)
constexpr size_t NA_OFF_ROWSUM = NA_OFF_STATUS + 256;                  // float[NA_MAX_M]
constexpr size_t NA_OFF_ADUP   = NA_OFF_ROWSUM + 256;                  // uint32[NA_MAX_M][k]
constexpr size_t NA_ADUP_BYTES = (size_t)NA_MAX_M * NA_MAX_K * 4;
constexpr size_t NA_OFF_PART   = NA_OFF_ADUP + NA_ADUP_BYTES;          // float[n/128][owners][m][128] partial sums

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

// In host code the name g_noalloc_scratch is only a handle for the runtime, not a device address; the address a
// kernel can use comes from cudaGetSymbolAddress, asked once per device with that device current.
struct NoAllocDev { unsigned char* base; int num_sms; bool ready; };
NoAllocDev g_na_dev[64];

int noalloc_setup(int dev, NoAllocDev** out)
{
    if (dev < 0 || dev >= 64) return EXL3_ERR_UNSUPPORTED;
    NoAllocDev& d = g_na_dev[dev];
    if (!d.ready) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            fprintf(stderr, "exl3_gemm_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
            cudaGetLastError();
            return EXL3_ERR_CUDA;
        }
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess || sms <= 0) { cudaGetLastError(); return EXL3_ERR_CUDA; }
        d.base = (unsigned char*)p; d.num_sms = sms; d.ready = true;
    }
    *out = &d;
    return EXL3_OK;
}

}  // namespace

extern "C" int exl3_gemm_noalloc(exl3_stream stream, const void* A, const void* trellis, void* C, const void* suh,
                                 const void* svh, int m, int k, int n, int K, int c_fp32, int mcg, int mul1)
{
    if (!A || !trellis || !C) { fprintf(stderr, "exl3_gemm_noalloc: null argument\n"); return EXL3_ERR_INVALID; }
    if (m < 0 || k <= 0 || n <= 0 || k % 128 || n % 128 || K < 1 || K > 8 || (mcg && mul1) || !aligned16(A) ||
        !aligned16(trellis) || !aligned16(C) || !aligned16(suh) || !aligned16(svh)) {
        fprintf(stderr, "exl3_gemm_noalloc: bad shape or alignment (k %% 128 == 0, n %% 128 == 0, K in 1..8, 16-byte aligned pointers)\n");
        return EXL3_ERR_INVALID;
    }
    if (m > NA_MAX_M || k > NA_MAX_K || n > NA_MAX_N) {
        fprintf(stderr, "exl3_gemm_noalloc: m=%d k=%d n=%d exceeds the fixed scratch (limits: m <= %d, k <= %d, n <= %d); "
                        "use exl3_gemm with a context for larger problems\n", m, k, n, NA_MAX_M, NA_MAX_K, NA_MAX_N);
        return EXL3_ERR_WORKSPACE;
    }
    if (m == 0) return EXL3_OK;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return EXL3_ERR_CUDA; }
    NoAllocDev* d = nullptr;
    int rc = noalloc_setup(dev, &d);
    if (rc != EXL3_OK) return rc;

    cudaStream_t st = (cudaStream_t)stream;
    const int cb = mcg ? 1 : (mul1 ? 2 : 0);
    // the array keeps whatever the previous call left: the counters must start at zero (the status word is sticky until
    // exl3_gemm_noalloc_poll_status reads and clears it)
    if (cudaMemsetAsync(d->base + NA_OFF_CNT, 0, NA_OFF_STATUS - NA_OFF_CNT, st) != cudaSuccess) { cudaGetLastError(); return EXL3_ERR_CUDA; }
    uint32_t* a_dup = (uint32_t*)(d->base + NA_OFF_ADUP);
    float* rowsum = (float*)(d->base + NA_OFF_ROWSUM);
    gemm_prologue_kernel<<<m, 256, 0, st>>>((const half*)A, (const half*)suh, a_dup, rowsum, k);
    GemmSmallParams p;
    p.a_dup = a_dup; p.rowsum = rowsum; p.trellis = (const uint32_t*)trellis; p.partial = nullptr;
    p.counters = (int*)(d->base + NA_OFF_CNT); p.svh = (const half*)svh; p.status = (int*)(d->base + NA_OFF_STATUS);
    p.C = C; p.m = m; p.k = k; p.n = n; p.c_fp32 = c_fp32;
    cudaError_t e = launch_small_k(K, cb, 1, p, d->num_sms, NA_BYTES - NA_OFF_PART, (float*)(d->base + NA_OFF_PART), st, nullptr);
    if (e != cudaSuccess) {
        fprintf(stderr, "exl3_gemm_noalloc: launch failed: %s\n", cudaGetErrorString(e));
        cudaGetLastError();
        return EXL3_ERR_CUDA;
    }
    return EXL3_OK;
}

// The kernels behind exl3_gemm_noalloc report a bounded device-side wait that ran out through a status word inside the
// fixed array.  This copies the word to the host (synchronising `stream`), clears it, and returns EXL3_ERR_DEVICE_WAIT if
// it was set, EXL3_OK otherwise; like the entry point itself it allocates nothing.
extern "C" int exl3_gemm_noalloc_poll_status(exl3_stream stream)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return EXL3_ERR_CUDA; }
    NoAllocDev* d = nullptr;
    int rc = noalloc_setup(dev, &d);
    if (rc != EXL3_OK) return rc;
    int h = 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemcpyAsync(&h, d->base + NA_OFF_STATUS, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) { cudaGetLastError(); return EXL3_ERR_CUDA; }
    if (h == 0) return EXL3_OK;
    cudaMemsetAsync(d->base + NA_OFF_STATUS, 0, sizeof(int), st);
    cudaStreamSynchronize(st);
    return EXL3_ERR_DEVICE_WAIT;
}
