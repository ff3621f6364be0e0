// A launch that fails reports its error once, through the returned status: the
// runtime's last-error slot is left clean for the next check. The runtime's
// launch and its error slot are stood in for here, so no GPU is needed. Prints
// the status and what the slot holds after a failed and after a good launch.
#include <cstdio>
#include <cuda_runtime.h>

static cudaError_t g_result, g_slot = cudaSuccess;
template <typename... A>
static cudaError_t fake_launch(A...) {
    if (g_result != cudaSuccess) g_slot = g_result;
    return g_result;
}
static cudaError_t fake_last_error() {
    const cudaError_t e = g_slot;
    g_slot = cudaSuccess;
    return e;
}
#define cudaLaunchKernelEx fake_launch
#define cudaGetLastError fake_last_error
#include "launch.cuh"

__global__ void noop() {}

int main() {
    for (const cudaError_t r : {cudaErrorInvalidConfiguration, cudaSuccess}) {
        g_result = r;
        const cudaError_t st = mmsk::launch_overlapped(noop, dim3(1), 32, 0, nullptr, 1);
        std::printf("%d %d\n", (int)st, (int)g_slot);
    }
    return 0;
}
