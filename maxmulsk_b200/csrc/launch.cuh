// Kernel launches that overlap the end of the kernel before them.
//
// The kernels launched through launch_overlapped start with grid_wait() and have
// the programmatic-serialization attribute: their blocks may become resident while
// the kernel before it in the stream drains -- from the moment that all blocks
// of that one have called grid_release(), or left -- and wait there until it
// has completed and its writes are visible. Launch latency, block start-up,
// barrier and tensor-memory set-up then run beside the predecessor's tail
// instead of after it. Nothing reads or writes global memory before
// grid_wait(), and every block calls it, so that a kernel's completion implies
// its predecessors'. A waiting block never holds up a running one: successors
// start only when no block of the predecessor is left to be scheduled.
//
// The tensor-core kernels, one block an SM, release at the end of their last
// products. The others release by leaving: where a block still running shares
// its SM with room for more, the successor's early blocks crowd the SMs that
// have most of it (FP32 calls back to back at 1024^3: 64 x 64 tiles 57 -> 84 us
// with a release at the start, 128 x 64 tiles 54 -> 73 with one before the
// stores). Measured (us a call from Python, this attribute off -> on, in turn on one
// B200): FP32 256^3 13.4 -> 12.7 (in a graph 4.42 -> 4.00), 777 x 1531 x 901 75.8 ->
// 71.0, BF16x6 64 x 8192 x 512 16.4 -> 13.5, 128 x 32768 x 512 37.5 -> 35.1, BF16x9 1500 x
// 2049 x 1999 124.9 -> 120.3, a picker training step 38.9 -> 29.7.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace mmsk {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s,
                              unsigned cluster, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster > 1) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = cluster;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) cudaGetLastError();      // reported by the status alone, not by the next check too
    return e;
}

}  // namespace mmsk
