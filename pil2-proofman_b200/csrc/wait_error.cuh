// Error word of the kernels' bounded waits (a TMA tile copy, a tensor core product).
//
// A wait that runs out cannot end its kernel with an error that CUDA reports, and the kernel's results are wrong, so
// it raises a word that the host looks at wherever it has waited for the device and hands results on.  The word is
// pinned host memory that the device writes through its mapping: looking costs no copy, and a commit whose waits
// hold pays nothing.  It stays raised until it is cleared, so a failure in a call that does not wait
// for the device is reported by the next one that does.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

__device__ int *g_wait_error;  // this device's word

namespace wait_error {

constexpr int MAX_DEVICES = 64;

__device__ __forceinline__ void raise()
{
    if (volatile int *w = g_wait_error) *w = 1;
    __threadfence_system();
}

inline std::atomic<int> *&word(int dev)
{
    static std::atomic<int> *words[MAX_DEVICES];
    return words[dev];
}

// the current device's word (dev its index, below MAX_DEVICES), before its first kernel
inline cudaError_t init(int dev)
{
    if (word(dev)) return cudaSuccess;
    void *h = nullptr, *d = nullptr;
    cudaError_t e = cudaHostAlloc(&h, sizeof(std::atomic<int>), cudaHostAllocMapped | cudaHostAllocPortable);
    if (e != cudaSuccess) return e;
    auto *w = new (h) std::atomic<int>(0);
    static_assert(sizeof(*w) == sizeof(int) && std::atomic<int>::is_always_lock_free, "the device writes an int");
    if ((e = cudaHostGetDevicePointer(&d, h, 0)) == cudaSuccess) e = cudaMemcpyToSymbol(g_wait_error, &d, sizeof(d));
    if (e != cudaSuccess) {
        cudaFreeHost(h);
        return e;
    }
    word(dev) = w;
    return cudaSuccess;
}

inline bool raised(int dev) { return dev >= 0 && dev < MAX_DEVICES && word(dev) && word(dev)->load() != 0; }
inline bool clear(int dev) { return dev >= 0 && dev < MAX_DEVICES && word(dev) && word(dev)->exchange(0) != 0; }

}  // namespace wait_error
