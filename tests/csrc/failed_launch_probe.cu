// Test-only: a launch that the runtime refuses (more threads to a block than there are), through launch_chained.
#include "launch.h"

#include <exception>

namespace {
__global__ void nothing_kernel(int) {}
}  // namespace

// 0: the launch threw and left no error behind, 1: it did not throw, 2: the error is still the runtime's last one
extern "C" int dscuda_test_failed_launch() {
    (void)cudaGetLastError();
    try {
        dscuda::launch_chained(nothing_kernel, dim3(1), dim3(4096), 0, nullptr, 0);
        return 1;
    } catch (const std::exception&) {
        return cudaPeekAtLastError() == cudaSuccess ? 0 : 2;
    }
}
