// The host side of the library (runtime.cpp, fault.cu) on a stand-in for the CUDA runtime that only counts and copies, so
// that it runs without a GPU. Prints "<name> <values>" a line; the first argument names the scenario.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

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

// The tables of a length against their definitions in long double: the largest error of each precision, relative to the
// largest entry of its table, and the allocations and copies that they took.
static double g_err64 = 0, g_err32 = 0;
template <typename F> static void compare(const double2* a, const float2* b, int count, F&& want) {
    long double most = 0, e64 = 0, e32 = 0;
    for (int i = 0; i < count; ++i) {
        long double re, im;
        want(i, re, im);
        most = std::max(most, hypotl(re, im));
        e64 = std::max(e64, hypotl(a[i].x - re, a[i].y - im));
        e32 = std::max(e32, hypotl(b[i].x - re, b[i].y - im));
    }
    g_err64 = std::max(g_err64, (double)(e64 / most));
    g_err32 = std::max(g_err32, (double)(e32 / most));
}

static const long double kPi = 3.141592653589793238462643383279502884L;

// exp(-i pi num / den)
static void root(long double num, long double den, long double& re, long double& im) {
    re = cosl(kPi * num / den);
    im = -sinl(kPi * num / den);
}

static void bluestein(int n, int m, const double2* chirp64, const float2* chirp32, const double2* kern64,
                      const float2* kern32, const double2* tw64, const float2* tw32) {
    compare(chirp64, chirp32, n, [&](int j, long double& re, long double& im) { root((long long)j * j % (2 * n), n, re, im); });
    compare(tw64, tw32, m, [&](int k, long double& re, long double& im) { root(2 * k, m, re, im); });
    std::vector<long double> c(2 * n), w(2 * m);
    for (int j = 0; j < n; ++j) root((long long)j * j % (2 * n), n, c[2 * j], c[2 * j + 1]);
    for (int k = 0; k < m; ++k) root(2 * k, m, w[2 * k], w[2 * k + 1]);
    compare(kern64, kern32, m, [&](int k, long double& re, long double& im) {
        re = im = 0;
        for (int j = -(n - 1); j < n; ++j) {
            const int d = std::abs(j), e = (int)(((long long)(j + m) * k) % m);  // conj(c_|j|) w^(j k)
            re += c[2 * d] * w[2 * e] + c[2 * d + 1] * w[2 * e + 1];
            im += c[2 * d] * w[2 * e + 1] - c[2 * d + 1] * w[2 * e];
        }
        re /= m;
        im /= m;
    });
}

static void tables(int n) {
    const FftTables* t = nullptr;
    g_mallocs = g_copies = 0;
    const int st = fft_tables(n, &t);
    std::printf("cost %d %d %d\n", st, g_mallocs, g_copies);
    if (st != RTM_OK) return;
    compare(t->tw64, t->tw32, n, [&](int k, long double& re, long double& im) { root(2 * k, n, re, im); });
    compare(t->mod64, t->mod32, n, [&](int k, long double& re, long double& im) { root(k, n, re, im); });
    const FftPlan& p = t->plan;
    const RegPlan& r = t->reg;
    if (p.m != n) bluestein(n, p.m, p.chirp64, p.chirp32, p.kern64, p.kern32, p.twm64, p.twm32);
    if (r.n1 && r.m != n) bluestein(n, r.m, r.chirp64, r.chirp32, r.kern64, r.kern32, r.tw64, r.tw32);
    if (r.n1 && r.m == n) compare(r.tw64, r.tw32, n, [&](int k, long double& re, long double& im) { root(2 * k, n, re, im); });
    if (t->ta64) {
        compare(t->ta64, t->ta32, n, [&](int i, long double& re, long double& im) { root(2 * (i / r.n2) * (i % r.n2), n, re, im); });
        compare(t->tb64, t->tb32, n, [&](int i, long double& re, long double& im) { root(2 * (i / r.n1) * (i % r.n1), n, re, im); });
    }
    if (t->t364) {
        compare(t->t364, t->t332, n, [&](int i, long double& re, long double& im) { root(2 * (i / 64) * (i % 64), n, re, im); });
        compare(t->t364 + n, t->t332 + n, 64, [&](int i, long double& re, long double& im) { root(2 * (i / 8) * (i % 8), 64, re, im); });
    }
    std::printf("kind %d %d %d\n", p.m != n, r.n1 ? r.m != n : -1, (t->ta64 != nullptr) + (t->t364 != nullptr));
    std::printf("errors %.3e %.3e\n", g_err64, g_err32);
}

// The split of every length that has one: "<n> <n1> <n2> <m>", m == n without a Bluestein convolution.
static void splits() {
    for (int n = 2; n <= kRegMax; ++n) {
        const FftTables* t = nullptr;
        if (fft_tables(n, &t) == RTM_OK && t->reg.n1) std::printf("%d %d %d %d\n", n, t->reg.n1, t->reg.n2, t->reg.m);
    }
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "faults") faults();
    if (what == "budget") budget();
    if (what == "splits") splits();
    if (what == "tables") tables(std::atoi(argv[2]));
    return 0;
}
