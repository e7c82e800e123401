// Launches whose beginning overlaps the end of the kernel in front of them in the stream (programmatic dependent launch).
//
// The later kernel's CTAs become resident once every CTA of the earlier one has called allowNextKernel() or has left, and set
// themselves up; whatever an earlier kernel of the stream may have written is touched only behind waitForPreviousKernel(), which
// returns when that kernel is complete and its stores are visible.  Every kernel launched this way calls it, in every CTA, so
// that a kernel that is complete implies that all before it in the stream are.
//
// A kernel that waits for something outside its stream (another GPU's flags, a dispatch on another stream) does not call
// allowNextKernel(): the next kernel's CTAs would hold their SMs' shared memory and registers, idle, for as long as that takes,
// and keep out the very work of other streams that the wait may depend on.  Its successor then starts when it is complete.
#ifndef NIXL_B200_PROGRAMMATIC_LAUNCH_CUH
#define NIXL_B200_PROGRAMMATIC_LAUNCH_CUH

#include <atomic>

#include <cuda_runtime.h>

namespace nixl_pdl {

__device__ __forceinline__ void waitForPreviousKernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allowNextKernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline cudaLaunchAttribute overlapAttribute() {
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    return a;
}

// Launches a kernel that calls waitForPreviousKernel().
template<class... Params, class... Args>
cudaError_t launch(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream, const Args &...args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = overlapAttribute();
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// For an overlapped kernel that has loads in flight rather than shared memory: asks for the whole of an SM's L1, once per device
// (`dev` is the current one, `done` belongs to the kernel).  Without it the kernel's CTAs take an SM over as the kernel in front has split it, and behind a
// GEMM, whose ring leaves some 28 KB to L1, that bounds the bytes in flight: combine of 4096 tokens x 4096 behind its expert GEMM,
// whole step 562 -> 550 us (2048 channels 218 -> 212, 1024 channels 116 -> 112); with all of it asked for as shared memory and no
// overlap 562 as well.  Asking for 8, 14, 17 or 25 percent of shared memory instead gives the same times.
inline cudaError_t preferL1(const void *kernel, int dev, std::atomic<bool> (&done)[64]) {
    if (dev < 0 || dev >= 64 || done[dev].load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1);
    if (e == cudaSuccess) done[dev].store(true, std::memory_order_relaxed);
    return e;
}

} // namespace nixl_pdl

#endif
