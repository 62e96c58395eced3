// Launches whose start overlaps the end of the kernel in front of them on the stream (programmatic dependent launch).
//
// A kernel launched this way may be resident while its predecessor still runs: before it touches global memory that the
// predecessor (or anything before it) reads or writes it must call launch_wait(), which returns once all of that is
// complete and visible.  launch_next(), called by every block, lets the successor start; called early it hides the
// successor's launch and prologue.  In a chain of small kernels those were most of the time (a 14 x 14 layer's forward:
// three kernels, 23 us).
#pragma once

#include <string.h>

#include "common.cuh"

__device__ __forceinline__ void launch_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Once per kernel and device (and whenever more is asked for): its dynamic shared memory, and the largest shared-memory
// partition of the SM, so that kernels that follow each other do not make the SM re-partition its memory, which it only
// does when it is idle.
int32_t katsu_prepare_kernel(katsu_cuda_ctx *ctx, const void *kernel, size_t smem);

template <typename... Params, typename... Args>
int32_t katsu_launch_chained(katsu_cuda_ctx *ctx, void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem,
                             unsigned cluster, Args &&...args) {
    cudaLaunchConfig_t config;
    memset(&config, 0, sizeof(config));
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(block, 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = ctx->stream;
    cudaLaunchAttribute attributes[2];
    memset(attributes, 0, sizeof(attributes));
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = 1;
    if (cluster > 1) {
        attributes[1].id = cudaLaunchAttributeClusterDimension;
        attributes[1].val.clusterDim.x = cluster;
        attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
        config.numAttrs = 2;
    }
    const cudaError_t err = cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
    ctx->launches += 1;
    if (err != cudaSuccess) {
        cudaGetLastError();
        return katsu_set_error(KATSU_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(err));
    }
    return KATSU_OK;
}
