// CUDA runtime calls that fail on request, for a copy of the library that is linked with
// --wrap for each of them.  Nothing fails on the GPU: a launch that "loses a row" runs as
// ever, and its error word is set behind it.
#include <cuda_runtime.h>

namespace {
int g_lose = 0;        // the launch with a cluster, counted from the next, that loses a row
int g_most = 1 << 30;  // clusters of more blocks do not fit
bool g_error = false;  // and say so with an error
}

extern "C" {
void failing_lose_row(int launch) { g_lose = launch; }

cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* func, void** args);

cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* func, void** args) {
    const cudaError_t e = __real_cudaLaunchKernelExC(config, func, args);
    bool cluster = false;
    for (unsigned i = 0; i < config->numAttrs; ++i) cluster |= config->attrs[i].id == cudaLaunchAttributeClusterDimension;
    if (e != cudaSuccess || !cluster || g_lose == 0 || --g_lose > 0) return e;
    return cudaMemsetAsync(*static_cast<int**>(args[5]), 1, sizeof(int), config->stream);   // the kernel's `error`
}

void failing_most_blocks(int blocks, int error) {
    g_most = blocks;
    g_error = error != 0;
}

cudaError_t __real_cudaOccupancyMaxActiveClusters(int* clusters, const void* func, const cudaLaunchConfig_t* config);

cudaError_t __wrap_cudaOccupancyMaxActiveClusters(int* clusters, const void* func, const cudaLaunchConfig_t* config) {
    unsigned blocks = 1;
    for (unsigned i = 0; i < config->numAttrs; ++i)
        if (config->attrs[i].id == cudaLaunchAttributeClusterDimension) blocks = config->attrs[i].val.clusterDim.x;
    if (blocks <= (unsigned)g_most) return __real_cudaOccupancyMaxActiveClusters(clusters, func, config);
    *clusters = 0;
    if (!g_error) return cudaSuccess;
    cudaSetDevice(-1);   // refused: an error stays behind, as the query's own would
    return cudaErrorInvalidClusterSize;
}
}
