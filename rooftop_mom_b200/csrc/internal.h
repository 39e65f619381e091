// Internal declarations shared by the CUDA and C++ sources of librtm.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <vector>

#include "../../include/rtm.h"

namespace rtm {

// ---------------------------------------------------------------------------------------------
// Errors: every entry point returns a status and records a thread-local message.
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);
inline int check_cuda(cudaError_t e, const char* what) { return e == cudaSuccess ? RTM_OK : cuda_fail(e, what); }

#define RTM_CUDA(call)                                        \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess) return ::rtm::cuda_fail(e_, #call); \
    } while (0)

#define RTM_TRY(call)                   \
    do {                                \
        int s_ = (call);                \
        if (s_ != RTM_OK) return s_;    \
    } while (0)

// Streaming multiprocessors of a B200: what launch shapes are sized by. Kernels whose CTAs wait for one another ask the
// device instead.
constexpr int kDeviceSms = 148;

extern int64_t g_launches;  // launches of this library's kernels (incremented by the launchers)
inline void count_launch(int n = 1) { __atomic_fetch_add(&g_launches, (int64_t)n, __ATOMIC_RELAXED); }

// One-time set-up per device, such as kernel attributes, which belong to the device's context. Host
// threads that reach the same device's set-up together may both run it, so the set-up must be
// idempotent; the flags are atomic, so that race is well defined. The flag is set only when the
// set-up succeeds. Ordinals above 63 run the set-up on every call.
struct DeviceOnce {
    std::atomic<bool> done[64] = {};
    template <typename F> int operator()(F&& setup) {
        int dev = 0;
        RTM_CUDA(cudaGetDevice(&dev));
        const bool tracked = dev >= 0 && dev < 64;
        if (tracked && done[dev].load(std::memory_order_acquire)) return RTM_OK;
        RTM_TRY(setup());
        if (tracked) done[dev].store(true, std::memory_order_release);
        return RTM_OK;
    }
};

// ---------------------------------------------------------------------------------------------
// Budget ledger of device bytes (Budget.m). Thread-safe.
// fresh: no allocation of the bytes follows, so the device's free memory is read anew however small they are.
int budget_require(double bytes, const char* what, bool fresh = false);
// A byte count as the reference's messages write it (formatBytes.m): "512 B", "1.5 kB", "3.0 GB".
std::string format_bytes(double bytes);
void budget_hold(double bytes);
void budget_release(double bytes);
// Returns the cached idle blocks of the current device to the driver.
void release_cached_blocks();

// Device buffer owned by a handle; its bytes are held in the budget while it lives.
// Blocks come from a per-device cache of freed blocks (no cudaFree, whose implicit device-wide
// synchronisation would stall concurrent solves); the cache is emptied when cudaMalloc fails.
struct DeviceBuffer {
    void* ptr = nullptr;
    size_t bytes = 0;     // requested (held in the budget)
    size_t capacity = 0;  // size of the cached block
    int device = 0;
    DeviceBuffer() = default;
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    ~DeviceBuffer() { reset(); }
    int alloc(size_t n);
    void reset();
    template <typename T> T* as() const { return reinterpret_cast<T*>(ptr); }
    // Moves another buffer's block into this one.
    void take(DeviceBuffer& o) {
        reset();
        ptr = o.ptr; bytes = o.bytes; capacity = o.capacity; device = o.device;
        o.ptr = nullptr; o.bytes = 0; o.capacity = 0;
    }
};

// Synchronises a stream when it leaves scope. Declared after a function's device buffers, it runs
// before their blocks return to the cache, on every path out of the function.
struct StreamSyncGuard {
    cudaStream_t s;
    explicit StreamSyncGuard(cudaStream_t st) : s(st) {}
    ~StreamSyncGuard() { cudaStreamSynchronize(s); }
};

// Non-blocking streams from a pool of idle ones, since making and destroying one costs about 114 us on the host
// and every handle has its own. stream_release synchronises the stream, then keeps it for the next handle on its
// device (at most kIdleStreams a device) or destroys it. Safe from several threads; a stream has one owner at a
// time.
constexpr int kIdleStreams = 32;
int stream_acquire(cudaStream_t* s);
void stream_release(cudaStream_t s);

// ---------------------------------------------------------------------------------------------
// FFT plans: a length n factorised into radices; twiddle tables exp(-2 pi i m / n), m < n, in
// FP64 and FP32, computed on the host in long double and kept on the device for the life of the
// process (one table per length and device).
constexpr int kMaxStages = 20;
constexpr int kMaxGenericRadix = 64;  // largest prime factor this build transforms

// A length whose factorisation needs a prime above kMaxGenericRadix runs as a Bluestein (chirp-z)
// convolution: m is then the power of two >= 2n - 1 that a line buffer must hold, the radices are those
// of m, and the plan points to the chirp, the convolution kernel's spectrum and the roots of length m.
// Otherwise m == n and the pointers are null.
struct FftPlan {
    int n;
    int nstages;
    int radix[kMaxStages];
    int m;
    const double2* chirp64;  // exp(-i pi (j^2 mod 2n) / n), j < n
    const float2* chirp32;
    const double2* kern64;   // DFT_m of exp(+i pi d^2 / n) wrapped to length m, divided by m
    const float2* kern32;
    const double2* twm64;    // exp(-2 pi i k / m), k < m
    const float2* twm32;
};

// A length's split for the register-resident transforms (regfft.cuh): m = n1 n2 with n1 >= n2, both codelet
// lengths; m == n, or m >= 2 n - 1 for a Bluestein convolution (chirp and kernel spectrum then set). n1 == 0: the
// length has none.
constexpr int kRegMax = 1024;
struct RegPlan {
    int n, m, n1, n2;
    const double2* tw64;  // exp(-2 pi i k / m), k < m
    const float2* tw32;
    const double2* chirp64;  // exp(-i pi (j^2 mod 2n) / n), j < n
    const float2* chirp32;
    const double2* kern64;  // DFT_m of exp(+i pi d^2 / n) wrapped to length m, divided by m
    const float2* kern32;
};

struct FftTables {
    FftPlan plan;
    RegPlan reg;
    // Powers of two from 32 to kRegMax, for grid_fast.cu: the twiddles w^(t k1) of the split n = n1 n2 (t < n2, k1 < n1)
    // as its two steps read them, consecutive threads on consecutive entries: at k1 n2 + t, and at t n1 + k1. (Gathered
    // from the roots at t k1, a load touches up to 16 lines: FP32 256 x 256 product 15.3 us, 12.1 with these; FP64 64 x 64
    // 8.7, 8.0. The lines of grid_reg.cu, whose y passes share a t between 8 threads, gained nothing and lost cache.)
    const double2* ta64;
    const double2* tb64;
    const float2* ta32;
    const float2* tb32;
    // Lengths n >= 256, for the three-step lines of grid_fast.cu: w_n^(t k1) at 64 k1 + t, then w_64^(t0 k2) at 8 k2 + t0.
    const double2* t364;
    const float2* t332;
    const double2* tw64;   // n entries
    const float2* tw32;
    const double2* mod64;  // exp(-i pi d / n), d < n (the odd-subband modulation)
    const float2* mod32;
};

// Returns the cached tables of length n on the current device (a Bluestein plan when n has a prime
// factor above kMaxGenericRadix).
int fft_tables(int n, const FftTables** out);

// Shift-phase factors of generateShiftPhases.m: u(m) = 1 - exp(i pi (2m + parity) / n).
int shift_factors(int n, int parity, const double2** out64, const float2** out32);

template <typename T> struct Cx;
template <> struct Cx<double> { using T2 = double2; };
template <> struct Cx<float> { using T2 = float2; };

// Host FP64 helpers used by the assembler set-up.
void gauss_legendre(int order, double a, double b, std::vector<double>& points, std::vector<double>& weights);
void extracted_moments(double size_x, double size_y, double k, double out[7][4]);

int fast_fft_size(int count);

// An operator's fault word, which its kernels with bounded waits set to RTM_ERR_TIMEOUT when a wait runs out: pinned
// host memory mapped by the devices. acquire() may allocate, so it is called when the operator is built, outside any
// stream capture; take() reads and clears the word, after a synchronisation.
struct FaultWord {
    int* ptr = nullptr;
    FaultWord() = default;
    FaultWord(const FaultWord&) = delete;
    FaultWord& operator=(const FaultWord&) = delete;
    ~FaultWord();
    int acquire();
    bool take();
};

}  // namespace rtm
