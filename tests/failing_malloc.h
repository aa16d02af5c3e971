// Included before a translation unit of the library (tests/test_gpu_no_memory.py):
// its cudaMalloc calls fail while lb_test_no_memory is set, as on a full GPU.
#pragma once

#include <cuda_runtime.h>

inline int &lb_test_no_memory_flag() {
    static int flag = 0;
    return flag;
}
extern "C" __attribute__((used, visibility("default"))) inline void lb_test_no_memory(int on) {
    lb_test_no_memory_flag() = on;
}
template <typename T> cudaError_t lb_test_malloc(T **p, size_t bytes) {
    return lb_test_no_memory_flag() ? cudaErrorMemoryAllocation : cudaMalloc(p, bytes);
}
#define cudaMalloc lb_test_malloc
