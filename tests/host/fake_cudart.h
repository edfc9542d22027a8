// A CUDA runtime without a GPU, for tests of the library's host paths: "device"
// memory is host memory (new allocations read 0xA5 in every byte), copies are
// done at once, and kernels do nothing unless a test's hook does something.
#pragma once
#include <cuda_runtime_api.h>

#include <functional>

namespace fake {
// Each hook is called in place of the runtime's answer; unset: success.
extern std::function<cudaError_t()> launch;  // every kernel launch
extern std::function<cudaError_t()> copy;    // every asynchronous copy
extern std::function<cudaError_t()> query;   // cudaStreamQuery
extern std::function<cudaError_t()> sync;    // cudaStreamSynchronize
extern long long clock_skew_s;               // added to the monotonic clock
}  // namespace fake
