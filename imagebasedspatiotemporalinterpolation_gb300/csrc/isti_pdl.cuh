// Programmatic dependent launches (PTX griddepcontrol), used by every chain of kernels.
//
// The kernels of a call depend on each other one after the other, and on what was in the stream
// before.  Each lets the next one's blocks take SMs as soon as its own blocks have all started
// (or ended), and waits for the kernel before it to complete, writes visible, before it touches
// anything that kernel writes or reads (the wait returns at once in an ordinary launch, or after
// work that is not a kernel).  That hides the launch latency between them: about 3 of 4.8 us per
// kernel, most of a small frame (640x360: 24.6 -> 19.0 us a call from within the call, 17.2 with
// the first kernel too; a lone call on an idle device 36.0 -> 32.5 us from call to result).
//
// So a kernel may be resident while others still write what it will read, and not only the one
// before it.  The read-only path (__ldg, const __restrict__ parameters) is for data that nobody
// writes meanwhile: what earlier kernels or the caller's may have written -- every image, table and
// intermediate -- is read by ordinary loads.
#pragma once

#include <cuda_runtime.h>

namespace isti
{
__device__ __forceinline__ void dependents_may_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_prerequisites() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a kernel after what was enqueued before it; `early`: as a programmatic dependent launch
// (the kernel waits by itself), otherwise in full order (around timing events, behind weights).
template <class... P, class... A>
cudaError_t launch_after(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const A &...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
} // namespace isti
