// Where a kernel whose bounded wait ran out leaves word of it: one int per translation unit in page-locked host memory, which
// rt_device_sync reads once the stream has drained (no copy from the device, no second synchronisation).  The wait itself
// only notes its site in device memory; a CTA that gave up hands it on to the host on its way out.  With the host's word
// written in the waits themselves (an address to load, a store, a fence in every wait loop) the decode chain's 64 GEMVs took
// 423.8 us instead of 418.7, the Whisper encoder's eight GEMMs 83.7 instead of 82.9.
#pragma once
#include <cuda_runtime.h>

namespace rt {
namespace {

__device__ int *g_wait_error = nullptr; // this translation unit's word on the current device; null: nobody listens
__device__ int g_wait_site = 0;         // the site that gave up, until a CTA on its way out reports it

// In the wait that gave up: the first site is kept.
__device__ __forceinline__ void note_wait_error(int site) { atomicCAS(&g_wait_site, 0, site); }

// On the way out of a CTA that gave up.
__device__ __forceinline__ void report_wait_error() {
    const int site = atomicExch(&g_wait_site, 0);
    int *const word = g_wait_error;
    if (word && site) {
        *reinterpret_cast<volatile int *>(word) = site;
        __threadfence_system();
    }
}

inline cudaError_t bind_wait_error(int *word) { return cudaMemcpyToSymbol(g_wait_error, &word, sizeof(word)); }

} // namespace
} // namespace rt
