// pdl.cuh -- programmatic dependent launch: a kernel that starts while the one
// before it in the stream finishes.
//
// A kernel launched with launch_overlapped may be placed on the SMs as soon
// as every block of its predecessor has passed pdl_start (or, behind a kernel
// without it, has ended). It computes its indices, then pdl_start waits until
// the predecessor has completed and its writes are visible, and only then
// lets its own successor come up. So at most two kernels of a stream overlap,
// and none touches memory before its predecessor is done: what is saved is
// the launch gap (2.5 us between dependent kernels) and the index arithmetic:
// FP64 CG at 8^3x16 0.95 -> 0.71 ms, F64 xpay hop at 24^3x48 93 -> 90 us, the
// 4x6x8x10 hop 5.5 -> 4.5 us (a call's host time).
//
// Rules for such a kernel: every thread calls pdl_start before its first
// memory access; what it reads may have been written by the predecessor, so
// it is read with ordinary loads (raw_loads.cuh), never through the
// non-coherent path, whose loads the compiler may move ahead of the wait.
#pragma once

#include <cuda_runtime.h>

#include "internal.h"

namespace plqcd {
namespace dev {

__device__ __forceinline__ void pdl_start() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace dev

// Without the attribute where the stream is being captured: the graphs here
// (conditional bodies, forked copies) take plain kernel nodes.
template <class... P, class... A>
int launch_overlapped(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t s, A... args) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
    if (capturing) cudaGetLastError();
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = capturing ? 0 : 1;
    PLQCD_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    return PLQCD_OK;
}

}  // namespace plqcd
