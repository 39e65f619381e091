// The host side of the library (runtime.cpp, fault.cu) on a stand-in for the CUDA runtime that only counts and copies, so
// that it runs without a GPU. Prints "<name> <values>" a line; the first argument names the scenario.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "../../rooftop_mom_b200/csrc/ops.h"

static size_t g_free_bytes = size_t(100) << 30;
static int g_mallocs = 0, g_copies = 0, g_host_allocs = 0;

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "error"; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = g_free_bytes, *t = size_t(180) << 30, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > g_free_bytes) return cudaErrorMemoryAllocation;
    ++g_mallocs;
    return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    ++g_host_allocs;
    return *p = std::malloc(n), cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    ++g_copies;
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)std::malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free((void*)s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}

using namespace rtm;

struct Op : LinearOp {
    FaultWord word;
    int apply(const void*, void*, int, cudaStream_t, SkipFlags) override { return RTM_OK; }
    bool take_fault() override { return word.take(); }
};

// Two operators, a wait of the first one's kernels run out: only the first one's check reports it, once.
static void faults() {
    Op a, b;
    a.word.acquire();
    b.word.acquire();
    *a.word.ptr = RTM_ERR_TIMEOUT;
    std::printf("other %d\n", fault_check(nullptr, {&b, nullptr}));
    std::printf("own %d\n", fault_check(nullptr, {&b, &a}));
    std::printf("again %d\n", fault_check(nullptr, {&b, &a}));
    // words of destroyed operators are used again, cleared
    for (int i = 0; i < 5000; ++i) {
        Op c;
        c.word.acquire();
        *c.word.ptr = RTM_ERR_TIMEOUT;
    }
    Op d;
    d.word.acquire();
    std::printf("reused %d pages %d\n", fault_check(nullptr, {&d}), g_host_allocs);
}

// Memory that another user of the device takes between two checks.
static void budget() {
    const double gib = double(1 << 30);
    std::printf("first %d\n", budget_require(gib, "The request", true));
    g_free_bytes = size_t(1) << 29;
    std::printf("taken %d\n", budget_require(gib, "The request", true));
    DeviceBuffer b;
    const int checked = budget_require(gib, "The product");
    std::printf("allocated %d\n", checked != RTM_OK ? checked : b.alloc(size_t(1) << 30));
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "faults") faults();
    if (what == "budget") budget();
    return 0;
}
