// Kernel launches that may begin before the kernel in front of them on the stream has ended.
#pragma once

#include "cuda_common.h"

#include <cuda_runtime.h>

#include <cstddef>
#include <utility>

namespace dscuda {

// Programmatic dependent launch: the blocks of a grid may start when every block of the preceding grid has exited, so its
// launch latency, barrier set-up and tensor-memory allocation overlap the end of that grid (the flush of its writes).
// Every kernel launched this way calls sm100::grid_dependency_wait() before it touches memory that another kernel writes; that
// returns when the preceding grid has ended and its writes are visible.  The one thing read earlier is the kernel family's own
// status word.  Loads are plain, not ld.global.nc: that form wants memory that nothing writes while the kernel lives, and its
// life begins before the grid in front has ended.  No kernel lets its dependents go early
// (griddepcontrol.launch_dependents): blocks of the next grid that sit beside a running decode slowed it (8 ragged sequences,
// 128 heads: 35.3 us without, 41-44 us with), and nothing else gained.
template <class... Parameters, class... Arguments>
void launch_chained(void (*kernel)(Parameters...), dim3 grid, dim3 block, std::size_t shared_bytes, cudaStream_t stream, Arguments&&... arguments) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = shared_bytes;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    const cudaError_t result = cudaLaunchKernelEx(&config, kernel, std::forward<Arguments>(arguments)...);
    if (result != cudaSuccess) {
        (void)cudaGetLastError();       // reported here: the caller's next check must not find it again
    }
    CUDA_CHECK(result);
}

}  // namespace dscuda
