// The fault words: kernels whose waits are bounded (the pipelined x-mix of grid_fast.cu) record RTM_ERR_TIMEOUT in the
// word of the operator they run for when a wait runs out, instead of hanging; the host reads it after a synchronisation.
// An operator has its own, so that a call on another operator, stream or thread cannot take the sign of a fault away.
// The words lie in pinned host memory that the devices map, so a check is a synchronisation and a load (copying a word of
// device memory back costs a call about 9 us). A page holds 1024 of them and is kept until the process ends; words
// of destroyed operators are used again.
#include <mutex>
#include <vector>

#include "ops.h"

namespace rtm {

constexpr int kPageWords = 1024;
static std::mutex g_words_mu;
static std::vector<int*> g_idle_words;

int FaultWord::acquire() {
    if (ptr) return RTM_OK;
    std::lock_guard<std::mutex> lk(g_words_mu);
    if (g_idle_words.empty()) {
        void* p = nullptr;
        RTM_CUDA(cudaHostAlloc(&p, kPageWords * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
        for (int i = kPageWords; i-- > 0;) g_idle_words.push_back(static_cast<int*>(p) + i);
    }
    ptr = g_idle_words.back();  // one address on host and devices (unified addressing)
    g_idle_words.pop_back();
    __atomic_store_n(ptr, 0, __ATOMIC_RELAXED);
    return RTM_OK;
}

FaultWord::~FaultWord() {
    if (!ptr) return;
    std::lock_guard<std::mutex> lk(g_words_mu);
    g_idle_words.push_back(ptr);
}

bool FaultWord::take() {
    return ptr && __atomic_load_n(ptr, __ATOMIC_RELAXED) != 0 && __atomic_exchange_n(ptr, 0, __ATOMIC_RELAXED) != 0;
}

int fault_check(cudaStream_t s, std::initializer_list<LinearOp*> ops) {
    RTM_CUDA(cudaStreamSynchronize(s));
    bool fault = false;
    for (LinearOp* op : ops) fault |= op && op->take_fault();
    if (!fault) return RTM_OK;
    return fail(RTM_ERR_TIMEOUT, "a bounded wait of a product kernel ran out on the device; the result is invalid");
}

}  // namespace rtm
