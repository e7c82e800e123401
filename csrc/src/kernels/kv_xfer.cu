// Fused paged-KV-cache transfer kernel (see include/kernels/nixl_kernels.h for the contract).
// The data movement itself is in kv_xfer_body.cuh, shared with the allocation-free entry point.
#include "kernels/kv_xfer_body.cuh"
#include "kernels/programmatic_launch.cuh"

namespace {

template<bool kCast, int kVec> __global__ void __launch_bounds__(nixl_kv::kKvThreads, 4) kvXferKernel(const __grid_constant__ nixl_kv::KvPlan k) {
    nixl_pdl::allowNextKernel();
    nixl_pdl::waitForPreviousKernel();
    nixl_kv::moveBlocks<kCast, kVec>(k, k.p.src_blocks, k.p.dst_blocks);
    nixl_kv::signalWhenAllDone(k.p, k.p.done_counter);
}

} // namespace

extern "C" int nixl_kv_xfer_launch(const NixlKvXferParams *params, void *stream) {
    if (!params || !params->src_view || !params->dst_view || !params->src_blocks || !params->dst_blocks || !params->done_counter)
        return cudaErrorInvalidValue;
    const NixlKvXferParams &p = *params;
    if (const cudaError_t e = nixl_kv::checkShape(p); e != cudaSuccess) return e;
    int dev = 0;
    cudaGetDevice(&dev);
    const nixl_kv::KvPlan k = nixl_kv::planFor(p);
    const int grid = nixl_kv::gridFor(k, dev);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const auto kernel = p.cast_fp8 ? (k.vec_bytes == 32 ? kvXferKernel<true, 32> : kvXferKernel<true, 16>)
                                   : (k.vec_bytes == 32 ? kvXferKernel<false, 32> : kvXferKernel<false, 16>);
    static std::atomic<bool> l1_done[4][64];
    if (const cudaError_t e = nixl_pdl::preferL1(reinterpret_cast<const void *>(kernel), dev, l1_done[(p.cast_fp8 != 0) * 2 + (k.vec_bytes == 32)]); e != cudaSuccess) return e;
    // Requests posted one behind another: the next one's CTAs move in as this one's leave.
    return static_cast<int>(nixl_pdl::launch(kernel, grid, nixl_kv::kKvThreads, 0, s, k));
}
