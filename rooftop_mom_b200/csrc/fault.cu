// The fault words: kernels whose waits are bounded (the pipelined x-mix of grid_fast.cu) record
// RTM_ERR_TIMEOUT in their device's word when a wait runs out, instead of hanging; the host reads it after a
// synchronisation. The words lie in pinned host memory that the devices map, so a check is a synchronisation and a
// load: copying a word of device memory back had cost every call about 9 us (13.5 us with its synchronisation, a
// 32 x 32 plate's product call 31 us in all). One page a process, held until it ends; it is no device memory.
#include <mutex>

#include "internal.h"

namespace rtm {

constexpr int kFaultStride = 32;  // a device's word on a cache line of its own
static std::mutex g_fault_mu;
static int* g_fault_words = nullptr;  // [64][kFaultStride]

int device_fault_word(int** out) {
    int dev = 0;
    RTM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_fault_mu);
    if (!g_fault_words) {
        void* p = nullptr;
        RTM_CUDA(cudaHostAlloc(&p, 64 * kFaultStride * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
        g_fault_words = static_cast<int*>(p);
        for (int i = 0; i < 64 * kFaultStride; ++i) g_fault_words[i] = 0;
    }
    *out = g_fault_words + (dev & 63) * kFaultStride;  // one address on host and devices (unified addressing)
    return RTM_OK;
}

int device_fault_check(cudaStream_t s) {
    int* w = nullptr;
    RTM_TRY(device_fault_word(&w));
    RTM_CUDA(cudaStreamSynchronize(s));
    if (__atomic_load_n(w, __ATOMIC_RELAXED) == 0 || __atomic_exchange_n(w, 0, __ATOMIC_RELAXED) == 0) return RTM_OK;
    return fail(RTM_ERR_TIMEOUT, "a bounded wait of a product kernel ran out on the device; the result is invalid");
}

}  // namespace rtm
