// Launches of kernels that follow one another on a stream.
//
// A kernel of a chain (pack, sweep, reduction, step stage) is often a few
// microseconds long, so the gap between two is a part of the time.  Launched
// as a programmatic dependent, a kernel's blocks are set up while the last
// blocks of the one before it end, and wait in chain_begin() until that one
// has completed and its writes are visible.  chain_begin() comes first in
// such a kernel, in every thread: also a block that has nothing to do waits,
// so that a kernel never completes before the one it follows.
//
// Back to back on a stream: 1000 x 1000 SPLIT Phi (three kernels) 14.7 ->
// 8.4 us, 200 x 65536 Acc 33.9 -> 28.6, EXACT Phi at 256 (one) 14.7 -> 12.2,
// a centred Acc sweep of 46400 (20) 1374 -> 1331.
// A kernel gives no earlier signal than its end: with one at its start the
// next kernel's blocks went to the SMs that the last blocks of this one left
// free, and a sweep of one wave then stood on half the chip (200 x 65536
// AccJerk 44.8 us without, 67 with; EXACT AccJerk at 3001 526 and 712).
#pragma once

#include <cuda_runtime.h>

namespace tg {

__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Set while this thread captures a graph of plain kernel nodes of its own.
extern thread_local bool g_chain_capture;

// Launches `kernel`, which begins with chain_begin().  In any other capture
// the launch stays an ordinary one: a captured sweep may land in any graph,
// the body of a conditional node included.
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block,
                           size_t smem, cudaStream_t st, const A &...args)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = g_chain_capture ||
                           (cudaStreamIsCapturing(st, &cap) == cudaSuccess &&
                            cap == cudaStreamCaptureStatusNone) ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel,
                                             static_cast<P>(args)...);
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

}  // namespace tg
