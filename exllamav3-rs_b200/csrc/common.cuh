// Shared declarations for the kernels of libexl3b200.so (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <utility>
#include "../../include/exl3_abi.h"

#define EXL3_PAGE 256

struct exl3_graph;

// Per-device state the ops share.  The reference keeps the equivalent in process-wide singletons
// (kernels/quant/exl3_devctx.cu:26-70); here it is explicit and owned by the caller.
struct exl3_ctx {
    int device;
    int num_sms;
    size_t ws_bytes;        // general scratch: split-K partials, attention split-KV partials, A_had
    uint8_t* ws;
    int* counters;          // arrival counters, all zero between calls
    int n_counters;
    int* status;            // device status word (0 = ok)
    cudaStream_t side_stream;
    cudaStream_t aux_stream;    // second lane inside one call: the decode-class attention pass runs beside the long-class one
    cudaEvent_t ev_fork, ev_join;
    uint64_t launches;
    int mma_attn;
    int use_tc;             // 1: tcgen05 GEMM for large M (default), 0: small-M kernel in passes (for A/B runs)
    int use_pair;           // 1: the tcgen05 GEMM runs on CTA pairs (cta_group::2, default), 0: one CTA per tile
    // per-stage device times of exl3_step_forward (off by default): events recorded at the stage boundaries of a step that
    // is not being captured, read back at its end
    int stage_prof;
    cudaEvent_t* prof_ev; int* prof_stage; int prof_ev_n;
    double stage_ms[EXL3_STAGES]; int stage_steps;
    int fuse_transform;     // 1: in the step runner the norm / activation kernels write the next GEMM's transformed activations (default), 0: separate launches
    // Work lists of the attention kernels kept across the layers of one exl3_step_forward call (they depend on the batch's
    // lengths only, not on the layer): slot 0 = decode class, slot 1 = long class.  plan_keep is set for the duration of a
    // step; outside of it every attention call builds its list anew.  plan_shape says how a kept list cuts the batch (0: none is
    // kept), because not every layer's pools need suit the same kernel.
    uint8_t* plan_slots;
    size_t plan_slot_bytes;
    int plan_keep;
    unsigned long long plan_shape[2];
    // Set for one attention call of a step: where the input transform of o_proj's activations goes and its signs.  The combine
    // kernel, which has a head's 128 values in a warp, writes it (had_done says that it does); had_bytes of the scratch in front
    // of the attention's own are taken by it.
    const half* had_suh; half* had_out; size_t had_bytes; int had_done;
    int kv_appended;        // set for one attention call of a step whose new keys and values are in the pools already
    // Programmatic dependent launches (exl3_launch): set while the work in front of a launch on its stream is known to be a
    // kernel of this library - inside a step, and after the first launch of a call of several - and broken for one launch
    // where a stream forks or joins.
    int chain, chain_break;
    char err[256];
};

// Programmatic dependent launches.  Every kernel that exl3_launch starts waits (griddepcontrol.wait) until the kernels before it are
// complete and their writes visible, and lets the next kernel of the chain be set up on the SMs that fall free
// (griddepcontrol.launch_dependents).  Ahead of its wait a kernel may
//  * read weights, sign vectors, norm weights and frequencies, which no kernel of a chain writes;
//  * read what was complete before its chain began, which the chain's first kernel sees to: a step's lengths, block table, positions and
//    slots (build_desc_kernel and the embedding are launched in full order), a call's lengths and block table (pdl_enter_first lets go
//    only behind its own wait).  The pools are not among it: the chain's append writes them;
//  * prefetch into L2 whatever it will read behind the wait;
//  * read what a kernel further in front wrote, if the kernel directly in front lets go behind its own wait (pdl_enter_late): the
//    merge of few rows reads the attention's work list;
//  * take tensor memory, if no kernel in front that has yet to take its own can be on the same SM (EXL3_TMEM_SMEM).
// At least one thread of every kernel waits, or the kernel would be complete before those in front of it.
// This is the plain form: lets go at once and touches nothing ahead of the wait.
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Two kernels on one SM that both take tensor memory ahead of their waits, the one behind first, would wait for each other: the GEMMs let
// their dependents go before they allocate, and the attention over codes allocates ahead of its wait (behind it, a verify step of 64
// layers took 10064 us instead of 10013).  Shared memory keeps them apart: a GEMM that takes tensor memory has at least this much of an
// SM's 228 KB, the attention over codes at least the rest.
constexpr int EXL3_TMEM_SMEM = 120 * 1024, EXL3_SM_SMEM = 228 * 1024;

// The same where the kernel behind reads, before its own wait, what the kernels in front of this one wrote.
__device__ __forceinline__ void pdl_enter_late()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The same for the first kernel of a call: the kernel behind it may read weights at once, so unless the work in front is known to
// be this library's (early), it is let go only when that is complete.
__device__ __forceinline__ void pdl_enter_first(int early)
{
    if (early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// 128-point Hadamard transform of a block whose elements 4 * lane + j are a, b of lane `lane`: fp32 butterflies, one fp16 rounding.
__device__ __forceinline__ uint2 had128_lane(half2 a, half2 b, int lane)
{
    float v0 = __low2float(a), v1 = __high2float(a), v2 = __low2float(b), v3 = __high2float(b);
    const float s0 = v0 + v1, d0 = v0 - v1, s1 = v2 + v3, d1 = v2 - v3;
    v0 = s0 + s1; v1 = d0 + d1; v2 = s0 - s1; v3 = d0 - d1;
    #pragma unroll
    for (int i = 1; i < 32; i <<= 1) {
        const float p0 = __shfl_xor_sync(0xffffffffu, v0, i), p1 = __shfl_xor_sync(0xffffffffu, v1, i);
        const float p2 = __shfl_xor_sync(0xffffffffu, v2, i), p3 = __shfl_xor_sync(0xffffffffu, v3, i);
        const bool up = lane & i;
        v0 = (up ? -v0 : v0) + p0; v1 = (up ? -v1 : v1) + p1;
        v2 = (up ? -v2 : v2) + p2; v3 = (up ? -v3 : v3) + p3;
    }
    constexpr float R128 = 0.088388347648f;
    a = __floats2half2_rn(v0 * R128, v1 * R128);
    b = __floats2half2_rn(v2 * R128, v3 * R128);
    uint2 o; o.x = *reinterpret_cast<uint32_t*>(&a); o.y = *reinterpret_cast<uint32_t*>(&b);
    return o;
}
// The same of (x o signs), `signs` holding the lane's four.  Same arithmetic as the GEMM's input transform of few rows: fp16 product first.
__device__ __forceinline__ uint2 had128_signed_lane(half2 a, half2 b, uint2 signs, int lane)
{
    return had128_lane(__hmul2(a, *reinterpret_cast<const half2*>(&signs.x)), __hmul2(b, *reinterpret_cast<const half2*>(&signs.y)), lane);
}

// Launch as a programmatic dependent of the previous kernel where the context says that there is one: the launch then
// overlaps the tail of its predecessor.  A decode step of a small model is some fifteen kernels of 3 to 10 us per layer
// (28 layers, hidden 1024, 8 rows: 2.79 -> 2.23 ms; verify step of 64 layers at 32 rows: 20.55 -> 20.11 ms).
static inline bool exl3_chained(exl3_ctx* ctx)
{
    const bool on = ctx->chain && !ctx->chain_break;
    ctx->chain_break = 0;
    return on;
}
template <typename... P, typename... A>
static inline cudaError_t exl3_launch(exl3_ctx* ctx, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = exl3_chained(ctx) ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
// The first kernel of a call, which begins with pdl_enter_first and takes its argument last: a programmatic dependent whatever is
// in front of it, because it touches nothing and lets nothing go before that is complete.  Back to back, the set-up of its blocks
// and the launch of the kernel behind it then overlap the tail of the call before (EXL3 GEMM at 4 bits, us: 5120 x 5120, 1 row
// 17.1 -> 15.1, 5120 x 17408, 52 rows 33.1 -> 29.2).  A call that is waited for before the next has none of this.  Under stream
// capture the node in front has to be a kernel for it, and the only one (replayed, against a plain launch there, us: 1024 x 3072 at 8
// bits, 1 and 8 rows 9.1 -> 8.1 and 10.1 -> 9.5; 5120 x 17408 at 4 bits, 1 and 52 rows 26.7 -> 25.7 and 31.1 -> 29.0).
static inline int exl3_first_early(exl3_ctx* ctx, cudaStream_t st, bool* overlap)
{
    if (exl3_chained(ctx)) { *overlap = true; return 1; }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    *overlap = cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone;
    if (cs == cudaStreamCaptureStatusActive) {
        const cudaGraphNode_t* deps = nullptr;
        size_t n = 0;
        cudaGraphNodeType type = cudaGraphNodeTypeEmpty;
        *overlap = cudaStreamGetCaptureInfo_v2(st, &cs, nullptr, nullptr, &deps, &n) == cudaSuccess && n == 1 &&
                   cudaGraphNodeGetType(deps[0], &type) == cudaSuccess && type == cudaGraphNodeTypeKernel;
    }
    if (!*overlap) cudaGetLastError();
    return 0;
}
template <typename... P, typename... A>
static inline cudaError_t exl3_launch_first(exl3_ctx* ctx, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
    bool overlap;
    const int early = exl3_first_early(ctx, st, &overlap);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)..., early);
}
// Marks the launches of a scope as a chain.
struct exl3_chain_scope {
    exl3_ctx* c; int old;
    explicit exl3_chain_scope(exl3_ctx* ctx, bool on = true) : c(ctx), old(ctx->chain) { if (on) c->chain = 1; }
    ~exl3_chain_scope() { c->chain = old; }
};

static inline int exl3_fail(exl3_ctx* ctx, int code, const char* msg)
{
    if (ctx) { strncpy(ctx->err, msg, sizeof(ctx->err) - 1); ctx->err[sizeof(ctx->err) - 1] = 0; }
    return code;
}

#define EXL3_REQUIRE(cond, msg) do { if (!(cond)) return exl3_fail(ctx, EXL3_ERR_INVALID, msg); } while (0)

static inline int exl3_check_launch(exl3_ctx* ctx, const char* what)
{
    cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        char buf[256];
        snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
        cudaGetLastError();
        return exl3_fail(ctx, EXL3_ERR_CUDA, buf);
    }
    return EXL3_OK;
}

static inline bool aligned16(const void* p) { return (((uintptr_t)p) & 15) == 0; }
// what the attention's copies of a head's codes and scales need
static inline bool quant_planes_aligned(const void* qk, const void* sk, const void* qv, const void* sv)
{
    return aligned16(qk) && aligned16(qv) && ((((uintptr_t)sk) | ((uintptr_t)sv)) & 7) == 0;
}

// Transformed activations of up to three EXL3 tensors that share an input, written by the kernel that produces the input
// (norm, activation) instead of by the GEMM's own transform launch: where each tensor's copy goes and its sign vector.
struct exl3_pre_act { const half* suh[3]; half* a_had[3]; int nseg; };
// gemm.cu: fills `pre` and returns true when exl3_gemm_fanout_pre can run these tensors on m rows of `dim` values (a tensor
// whose k is not the producer's width keeps the separate launches: the buffers are sized by k, the producer fills rows of dim)
bool exl3_pre_buffers(exl3_ctx* ctx, int count, const exl3_linear* const* w, int m, int dim, exl3_pre_act* pre);
int exl3_gemm_fanout_pre(exl3_ctx* ctx, exl3_stream stream, int count, const exl3_linear* const* w, void* const* C, int m, int c_fp32);
// elementwise.cu
// Where a step's new keys and values go: pools of one layer (kc and vc in fp16, or codes and scales) and every row's token slot
// (page * 256 + offset, -1: none).
struct exl3_kv_dst { const half* v; half* kc; half* vc; uint32_t* qk; half* sk; uint32_t* qv; half* sv; const int32_t* slot; int bits; };
// exl3_rope for head_dim 128 whose keys go to the pool instead of back to k, together with v
int exl3_rope_append(exl3_ctx* ctx, exl3_stream stream, void* q, const void* k, const float* inv_freq, int n_freq, const int32_t* row_pos,
                     const void* q_norm, const void* k_norm, float norm_eps, int rope_mode, float attn_factor, int rows, int nq, int nk,
                     const exl3_kv_dst* dst);
int exl3_rms_norm_pre(exl3_ctx* ctx, exl3_stream stream, const void* x, int x_fp32, const void* w, float* r, float eps,
                      float cbias, float cscale, int rows, int dim, const exl3_pre_act* pre);
int exl3_silu_mul_pre(exl3_ctx* ctx, exl3_stream stream, const void* x, const void* y, int rows, int dim, const exl3_pre_act* pre);

// Carve `bytes` out of the context scratch starting at *off (256-byte aligned); NULL when it does not fit.
static inline void* exl3_ws_take(exl3_ctx* ctx, size_t* off, size_t bytes)
{
    size_t o = (*off + 255) & ~(size_t)255;
    if (o + bytes > ctx->ws_bytes) return nullptr;
    *off = o + bytes;
    return ctx->ws + o;
}
