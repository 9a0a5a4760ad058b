// The instantiations of gemm_ts_kernel and their launch.
#include "gemm_ts.cuh"

namespace {

using namespace exl3;

template <int K, int CB>
cudaError_t launch_ts(const CUtensorMap* amap, const CUtensorMap* rmap, const GemmTsParams& p, int grid, bool overlap, cudaStream_t st)
{
    constexpr int bytes = TsSmem<K>::BYTES;
    static bool configured[64] = {};
    auto kern = gemm_ts_kernel<K, CB>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    // a programmatic dependent of the kernel that writes the transformed activations, which directly precedes it
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(TS_THREADS); cfg.dynamicSmemBytes = bytes; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, amap[0], amap[1], amap[2], rmap[0], rmap[1], rmap[2], p);
}

template <int K>
cudaError_t launch_ts_cb(int cb, const CUtensorMap* amap, const CUtensorMap* rmap, const GemmTsParams& p, int grid, bool overlap, cudaStream_t st)
{
    if (cb == 0) return launch_ts<K, 0>(amap, rmap, p, grid, overlap, st);
    if (cb == 1) return launch_ts<K, 1>(amap, rmap, p, grid, overlap, st);
    return launch_ts<K, 2>(amap, rmap, p, grid, overlap, st);
}

}  // namespace

cudaError_t exl3::gemm_ts_launch(int K, int cb, const CUtensorMap* amap, const CUtensorMap* rmap, const GemmTsParams& p, int grid, bool overlap, cudaStream_t st)
{
    switch (K) {
        case 1: return launch_ts_cb<1>(cb, amap, rmap, p, grid, overlap, st);
        case 2: return launch_ts_cb<2>(cb, amap, rmap, p, grid, overlap, st);
        case 3: return launch_ts_cb<3>(cb, amap, rmap, p, grid, overlap, st);
        case 4: return launch_ts_cb<4>(cb, amap, rmap, p, grid, overlap, st);
        case 5: return launch_ts_cb<5>(cb, amap, rmap, p, grid, overlap, st);
        case 6: return launch_ts_cb<6>(cb, amap, rmap, p, grid, overlap, st);
        case 7: return launch_ts_cb<7>(cb, amap, rmap, p, grid, overlap, st);
        default: return launch_ts_cb<8>(cb, amap, rmap, p, grid, overlap, st);
    }
}
