// Where a kernel whose bounded wait ran out leaves word of it: one int per translation unit in page-locked host memory,
// so that the host's sync reads plain memory instead of copying every kernel family's flag from the device (seven copies
// with a synchronisation each: 97 us of an rt_device_sync with nothing left to wait for, 5 us now).
#pragma once
#include <cuda_runtime.h>

namespace rt {
namespace {

__device__ int *g_wait_error = nullptr; // this translation unit's word on the current device; null: nobody listens

// Any of the sites that gave up may end up in the word: the caller only learns that one did.
__device__ __forceinline__ void report_wait_error(int site) {
    int *const word = g_wait_error;
    if (word) {
        *reinterpret_cast<volatile int *>(word) = site;
        __threadfence_system();
    }
}

inline cudaError_t bind_wait_error(int *word) { return cudaMemcpyToSymbol(g_wait_error, &word, sizeof(word)); }

} // namespace
} // namespace rt
