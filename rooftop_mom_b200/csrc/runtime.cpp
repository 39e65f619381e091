// Host runtime of librtm.so: error reporting, the HBM budget ledger, device buffers, the FFT plan
// and twiddle caches, and the FP64 host tables of the assembler (Gauss-Legendre rules and the
// closed-form touching moments).
#include <cmath>
#include <cstdio>
#include <algorithm>
#include <chrono>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "internal.h"

namespace rtm {

int64_t g_launches = 0;

static thread_local std::string t_error;

void set_error(const std::string& msg) { t_error = msg; }

int fail(int status, const std::string& msg) {
    set_error(msg);
    return status;
}

int cuda_fail(cudaError_t e, const char* what) {
    set_error(std::string("CUDA error ") + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ") in " + what);
    return RTM_ERR_CUDA;
}

// ---------------------------------------------------------------------------------------------
// Budget (src/+rooftopMoM/+resources/Budget.m:43-106): a ceiling on the bytes the live handles
// hold together, and the device's free memory.
static std::mutex g_budget_mu;
static double g_ceiling = 0.0;  // <= 0: none
static double g_held = 0.0;

// A byte count as the reference's messages write it (src/+rooftopMoM/+resources/+utils/formatBytes.m):
// whole bytes below 1 kB, else one decimal in kB, MB, GB or TB (powers of 1024); an infinite count (no
// ceiling) reads "unlimited", an unknown one "unknown".
std::string format_bytes(double b) {
    if (std::isinf(b)) return "unlimited";
    if (std::isnan(b)) return "unknown";
    const char* units[] = {"B", "kB", "MB", "GB", "TB"};
    const int e = std::min(std::max((int)std::floor(std::log2(std::max(b, 1.0)) / 10), 0), 4);
    char buf[64];
    if (e == 0) snprintf(buf, sizeof buf, "%.0f B", std::round(b));
    else snprintf(buf, sizeof buf, "%.1f %s", b / std::pow(1024.0, e), units[e]);
    return buf;
}

// The device's free memory as far as a request of `bytes` depends on it, for a request whose memory is allocated right
// after the check: the allocation itself then refuses what other users of the device have taken since the reading, with
// the same status. cudaMemGetInfo takes 0.2 to 1 ms in a process that uses torch and every set-up and solve asks, so a
// reading decides such requests of up to a sixteenth of it for kReadingAge; larger requests and older readings read
// again, and so does a check that nothing follows (fresh). The library's own allocations are taken off the reading. Called
// with g_budget_mu held.
constexpr double kReadingAge = 0.1;  // seconds
struct FreeReading {
    double bytes = -1;
    std::chrono::steady_clock::time_point at;
};
static FreeReading g_free[64];

static bool free_memory(double bytes, bool fresh, double* out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    FreeReading& r = g_free[dev & 63];
    const auto now = std::chrono::steady_clock::now();
    if (!fresh && dev < 64 && r.bytes >= 16 * bytes && std::chrono::duration<double>(now - r.at).count() < kReadingAge) {
        *out = r.bytes;
        return true;
    }
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
    r.bytes = (double)free_b;
    r.at = now;
    *out = r.bytes;
    return true;
}

int budget_require(double bytes, const char* what, bool fresh) {
    std::lock_guard<std::mutex> lk(g_budget_mu);
    if (g_ceiling > 0 && g_held + bytes > g_ceiling) {
        return fail(RTM_ERR_OOM_BUDGET, std::string(what) + " needs " + format_bytes(bytes) + ", but only " +
                                            format_bytes(std::max(0.0, g_ceiling - g_held)) +
                                            " of the memory ceiling of " + format_bytes(g_ceiling) + " are left.");
    }
    double free_b = 0;
    if (free_memory(bytes, fresh, &free_b) && bytes > free_b) {
        return fail(RTM_ERR_OOM_BUDGET, std::string(what) + " needs " + format_bytes(bytes) + ", but only " +
                                            format_bytes(free_b) + " are free on this device.");
    }
    return RTM_OK;
}

void budget_hold(double bytes) {
    std::lock_guard<std::mutex> lk(g_budget_mu);
    g_held += bytes;
}

void budget_release(double bytes) {
    std::lock_guard<std::mutex> lk(g_budget_mu);
    g_held -= bytes;
}

// Per-device cache of idle device blocks, by capacity.
static std::mutex g_pool_mu;
static std::multimap<size_t, void*> g_pool[64];

static size_t block_capacity(size_t n) {
    if (n <= (1u << 20)) {
        size_t c = 512;
        while (c < n) c <<= 1;
        return c;
    }
    const size_t mb = 1u << 20;
    return (n + mb - 1) / mb * mb;
}

void release_cached_blocks() {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_pool_mu);
    for (auto& kv : g_pool[dev & 63]) cudaFree(kv.second);
    g_pool[dev & 63].clear();
}

int DeviceBuffer::alloc(size_t n) {
    reset();
    if (n == 0) return RTM_OK;
    cudaGetDevice(&device);
    const size_t cap = block_capacity(n);
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        auto& pool = g_pool[device & 63];
        auto it = pool.lower_bound(cap);
        if (it != pool.end() && it->first <= cap + cap / 2) {
            ptr = it->second;
            capacity = it->first;
            pool.erase(it);
        }
    }
    if (!ptr) {
        cudaError_t e = cudaMalloc(&ptr, cap);
        if (e != cudaSuccess) {
            cudaGetLastError();
            release_cached_blocks();
            e = cudaMalloc(&ptr, cap);
        }
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();
            return fail(RTM_ERR_OOM_BUDGET, "device allocation of " + format_bytes((double)n) + " failed: " +
                                                cudaGetErrorString(e));
        }
        capacity = cap;
        std::lock_guard<std::mutex> lk(g_budget_mu);
        g_free[device & 63].bytes -= (double)cap;
    }
    bytes = n;
    budget_hold((double)n);
    return RTM_OK;
}

void DeviceBuffer::reset() {
    if (ptr) {
        {
            std::lock_guard<std::mutex> lk(g_pool_mu);
            g_pool[device & 63].emplace(capacity, ptr);
        }
        budget_release((double)bytes);
    }
    ptr = nullptr;
    bytes = 0;
    capacity = 0;
}

// ---------------------------------------------------------------------------------------------
// Idle streams by device, and the device of every stream handed out.
static std::mutex g_streams_mu;
static std::vector<cudaStream_t> g_idle_streams[64];
static std::map<cudaStream_t, int> g_stream_device;

int stream_acquire(cudaStream_t* s) {
    *s = nullptr;
    int dev = 0;
    RTM_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(g_streams_mu);
        auto& idle = g_idle_streams[dev & 63];
        if (dev < 64 && !idle.empty()) {
            *s = idle.back();
            idle.pop_back();
            return RTM_OK;
        }
    }
    RTM_CUDA(cudaStreamCreateWithFlags(s, cudaStreamNonBlocking));
    std::lock_guard<std::mutex> lk(g_streams_mu);
    g_stream_device[*s] = dev;
    return RTM_OK;
}

void stream_release(cudaStream_t s) {
    const bool sound = cudaStreamSynchronize(s) == cudaSuccess;
    {
        std::lock_guard<std::mutex> lk(g_streams_mu);
        auto it = g_stream_device.find(s);
        const int dev = it == g_stream_device.end() ? 64 : it->second;
        if (sound && dev < 64 && (int)g_idle_streams[dev].size() < kIdleStreams) {
            g_idle_streams[dev].push_back(s);
            return;
        }
        if (it != g_stream_device.end()) g_stream_device.erase(it);
    }
    cudaStreamDestroy(s);
}

// ---------------------------------------------------------------------------------------------
// FFT plans and tables.
int fast_fft_size(int count) {
    // generateFastFFTSize.m:11-15: the smallest size >= count with prime factors <= 7.
    for (int n = count;; ++n) {
        int m = n;
        for (int p : {2, 3, 5, 7})
            while (m % p == 0) m /= p;
        if (m == 1) return n;
    }
}

static bool make_plan(int n, FftPlan& p) {
    p = FftPlan{};
    p.n = n;
    p.m = n;
    p.nstages = 0;
    int m = n;
    auto push = [&](int r) {
        if (p.nstages >= kMaxStages) return false;
        p.radix[p.nstages++] = r;
        m /= r;
        return true;
    };
    for (int r : {16, 8, 4, 2, 3, 5, 7}) {
        while (m % r == 0)
            if (!push(r)) return false;
    }
    for (int r = 11; m > 1; r += 2) {
        if (r > kMaxGenericRadix) return false;
        while (m % r == 0)
            if (!push(r)) return false;
    }
    return true;
}

// The codelet lengths of the register-resident transforms by class (regfft.cuh): n1 of class 0 and 1, n2 <= n1.
static const std::vector<int> kRegN1[2] = {{4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16},
                                           {18, 20, 21, 24, 25, 27, 28, 30, 32, 35, 36}};
static const std::vector<int> kRegN2[2] = {{3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16},
                                           {5, 7, 9, 10, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32}};

// The split of m with the smallest n1 (the fewest values a thread holds); false when m has none.
static bool reg_split(int m, int* n1, int* n2) {
    for (int c = 0; c < 2; ++c)
        for (int a : kRegN1[c]) {
            if (m % a) continue;
            const int b = m / a;
            if (b <= a && std::find(kRegN2[c].begin(), kRegN2[c].end(), b) != kRegN2[c].end()) {
                *n1 = a;
                *n2 = b;
                return true;
            }
        }
    return false;
}

// The host side of the tables, in long double, rounded once to double.
struct Cl {
    long double re, im;
};
constexpr long double kPiL = 3.141592653589793238462643383279502884L;

// exp(-i pi k / n) for k < n.
static std::vector<Cl> half_roots(int n) {
    std::vector<Cl> w(n);
    for (int k = 0; k < n; ++k) {
        const long double a = kPiL * (long double)k / (long double)n;
        w[k] = {cosl(a), -sinl(a)};
    }
    return w;
}

// exp(-i pi k / n) for any k >= 0, from those of k < n.
static Cl half_root(const std::vector<Cl>& half, int64_t k) {
    const int64_t n = (int64_t)half.size(), q = k % (2 * n);
    return q < n ? half[q] : Cl{-half[q - n].re, -half[q - n].im};
}

// exp(-2 pi i k / m) for k < m; sines and cosines of the first quarter or half alone where m allows it.
static std::vector<Cl> roots(int m) {
    std::vector<Cl> w(m);
    const int part = m % 4 == 0 ? m / 4 : m % 2 == 0 ? m / 2 : m;
    for (int k = 0; k < m; ++k) {
        if (k < part) {
            const long double a = 2 * kPiL * (long double)k / (long double)m;
            w[k] = {cosl(a), -sinl(a)};
        } else {
            const Cl v = w[k - part];  // times -i or -1
            w[k] = m % 4 == 0 ? Cl{v.im, -v.re} : Cl{-v.re, -v.im};
        }
    }
    return w;
}

static Cl mul(const Cl& a, const Cl& b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }

// out = DFT of the n values in[stride j], n a product of primes up to 7, recursively over its smallest one; w: the roots
// of length wn (a multiple of n). n log n: a sum over two factors of 1024 points takes 1.6 ms, this 0.2.
static void host_dft(const Cl* in, int stride, Cl* out, int n, const Cl* w, int wn) {
    if (n == 1) {
        out[0] = in[0];
        return;
    }
    int p = 2;
    while (n % p) ++p;
    const int q = n / p;
    for (int r = 0; r < p; ++r) host_dft(in + (size_t)r * stride, stride * p, out + (size_t)r * q, q, w, wn);
    Cl t[7];
    for (int k = 0; k < q; ++k) {
        for (int r = 0; r < p; ++r) t[r] = r && k ? mul(out[r * q + k], w[(size_t)r * k * (wn / n)]) : out[r * q + k];
        if (p == 2) {
            out[k] = {t[0].re + t[1].re, t[0].im + t[1].im};
            out[q + k] = {t[0].re - t[1].re, t[0].im - t[1].im};
            continue;
        }
        for (int b = 0; b < p; ++b) {
            Cl sum = t[0];
            for (int r = 1; r < p; ++r) {
                const Cl v = mul(t[r], w[(size_t)(b * r % p) * (wn / p)]);
                sum = {sum.re + v.re, sum.im + v.im};
            }
            out[b * q + k] = sum;
        }
    }
}

// Bluestein: X_k = c_k sum_j (x_j c_j) b_(k-j) with c_j = exp(-i pi j^2 / n) and b_d = conj(c_d), the linear
// convolution evaluated as a circular one of length m >= 2n - 1. Returns the spectrum of b, divided by m. chirp: the c_j;
// wm: the roots of length m.
static std::vector<Cl> chirp_spectrum(const std::vector<Cl>& chirp, const std::vector<Cl>& wm) {
    const int n = (int)chirp.size(), m = (int)wm.size();
    std::vector<Cl> b(m, Cl{0, 0}), out(m);
    for (int j = 0; j < n; ++j) {
        b[j] = {chirp[j].re, -chirp[j].im};
        if (j) b[m - j] = b[j];
    }
    host_dft(b.data(), 1, out.data(), m, wm.data(), m);
    for (Cl& v : out) v = {v.re / m, v.im / m};
    return out;
}

// The plan of length n for the register-resident transforms, without its tables.
static void make_reg_plan(int n, RegPlan& p) {
    p = RegPlan{};
    p.n = p.m = n;
    if (n > kRegMax || reg_split(n, &p.n1, &p.n2)) return;
    int m = 2 * n - 1;
    while (m <= kRegMax && !reg_split(m, &p.n1, &p.n2)) ++m;
    // lengths whose factors are all codelets run in the Stockham engine when they have no split
    if (m > kRegMax || fast_fft_size(n) == n || n < 16) {
        p.n1 = p.n2 = 0;
        return;
    }
    p.m = m;
}

struct TableKey {
    int device;
    int n;
    bool operator<(const TableKey& o) const { return device != o.device ? device < o.device : n < o.n; }
};

// A length's tables and their one device allocation, kept for the life of the process.
struct TableEntry {
    FftTables t{};
    void* mem = nullptr;
};

static std::mutex g_tables_mu;
static std::map<TableKey, TableEntry> g_tables;

int fft_tables(int n, const FftTables** out) {
    if (n < 1) return fail(RTM_ERR_ARG, "FFT length must be positive");
    int dev = 0;
    RTM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_tables_mu);
    auto it = g_tables.find({dev, n});
    if (it != g_tables.end()) {
        *out = &it->second.t;
        return RTM_OK;
    }
    TableEntry e;
    FftPlan& plan = e.t.plan;
    RegPlan& reg = e.t.reg;
    if (!make_plan(n, plan)) {
        int m = 1;
        while (m < 2 * n - 1) m <<= 1;
        if (!make_plan(m, plan))
            return fail(RTM_ERR_UNSUPPORTED, "FFT length " + std::to_string(n) + " has no plan in this build");
        plan.n = n;
        plan.m = m;
    }
    make_reg_plan(n, reg);
    // All tables one after the other, in FP64 and again in FP32, so that a length costs one allocation and one copy.
    std::vector<double2> all;
    auto put = [&all](const std::vector<Cl>& v) {
        const size_t at = all.size();
        all.resize(at + v.size());
        for (size_t i = 0; i < v.size(); ++i) all[at + i] = make_double2((double)v[i].re, (double)v[i].im);
        return at;
    };
    const std::vector<Cl> half = half_roots(n);
    std::vector<Cl> line(n);
    for (int k = 0; k < n; ++k) line[k] = half_root(half, 2 * (int64_t)k);
    const size_t at_tw = put(line), at_mod = put(half);
    size_t at_chirp = 0, at_kern = 0, at_twm = 0, at_rtw = 0, at_rkern = 0;
    const bool blue = plan.m != n, reg_blue = reg.n1 && reg.m != n;
    if (blue || reg_blue) {
        for (int j = 0; j < n; ++j) line[j] = half_root(half, (int64_t)j * j);
        at_chirp = put(line);
        if (blue) {
            const std::vector<Cl> wm = roots(plan.m);
            at_kern = put(chirp_spectrum(line, wm));
            at_twm = put(wm);
        }
        if (reg_blue) {
            const std::vector<Cl> wm = roots(reg.m);
            at_rkern = put(chirp_spectrum(line, wm));
            at_rtw = put(wm);
        }
    }
    // the orders that the power-of-two kernels read their twiddles in (FftTables)
    const bool pow2 = reg.n1 && n >= 32 && (n & (n - 1)) == 0, three = pow2 && n >= 256;
    const size_t at_ta = all.size(), at_tb = at_ta + n, at_t3 = at_tb + n;
    if (pow2) {
        const int r1 = n / 64;
        all.resize(at_t3 + (three ? n + 64 : 0));
        const double2* tw = all.data() + at_tw;
        for (int k1 = 0; k1 < reg.n1; ++k1)
            for (int t = 0; t < reg.n2; ++t) all[at_ta + k1 * reg.n2 + t] = all[at_tb + t * reg.n1 + k1] = tw[t * k1];
        if (three) {
            for (int k1 = 0; k1 < r1; ++k1)
                for (int t = 0; t < 64; ++t) all[at_t3 + 64 * k1 + t] = tw[t * k1];
            for (int k2 = 0; k2 < 8; ++k2)
                for (int t0 = 0; t0 < 8; ++t0) all[at_t3 + n + 8 * k2 + t0] = tw[r1 * t0 * k2];
        }
    }
    const size_t count = all.size(), wide = count * sizeof(double2), bytes = wide + count * sizeof(float2);
    std::vector<char> host(bytes);
    memcpy(host.data(), all.data(), wide);
    float2* host32 = reinterpret_cast<float2*>(host.data() + wide);
    for (size_t i = 0; i < count; ++i) host32[i] = make_float2((float)all[i].x, (float)all[i].y);
    cudaError_t err = cudaMalloc(&e.mem, bytes);
    if (err != cudaSuccess) {
        cudaGetLastError();
        release_cached_blocks();
        err = cudaMalloc(&e.mem, bytes);
    }
    if (err != cudaSuccess) {
        cudaGetLastError();
        return fail(RTM_ERR_OOM_BUDGET, "device allocation of " + format_bytes((double)bytes) + " failed: " +
                                            cudaGetErrorString(err));
    }
    err = cudaMemcpy(e.mem, host.data(), bytes, cudaMemcpyHostToDevice);
    if (err != cudaSuccess) {
        cudaFree(e.mem);
        return cuda_fail(err, "cudaMemcpy of the tables of an FFT length");
    }
    const double2* d64 = static_cast<const double2*>(e.mem);
    const float2* d32 = reinterpret_cast<const float2*>(d64 + count);
    e.t.tw64 = d64 + at_tw;
    e.t.tw32 = d32 + at_tw;
    e.t.mod64 = d64 + at_mod;
    e.t.mod32 = d32 + at_mod;
    if (blue) {
        plan.chirp64 = d64 + at_chirp;
        plan.chirp32 = d32 + at_chirp;
        plan.kern64 = d64 + at_kern;
        plan.kern32 = d32 + at_kern;
        plan.twm64 = d64 + at_twm;
        plan.twm32 = d32 + at_twm;
    }
    if (reg.n1) {
        reg.tw64 = d64 + (reg_blue ? at_rtw : at_tw);
        reg.tw32 = d32 + (reg_blue ? at_rtw : at_tw);
    }
    if (reg_blue) {
        reg.chirp64 = d64 + at_chirp;
        reg.chirp32 = d32 + at_chirp;
        reg.kern64 = d64 + at_rkern;
        reg.kern32 = d32 + at_rkern;
    }
    if (pow2) {
        e.t.ta64 = d64 + at_ta;
        e.t.ta32 = d32 + at_ta;
        e.t.tb64 = d64 + at_tb;
        e.t.tb32 = d32 + at_tb;
    }
    if (three) {
        e.t.t364 = d64 + at_t3;
        e.t.t332 = d32 + at_t3;
    }
    auto res = g_tables.emplace(TableKey{dev, n}, e);
    *out = &res.first->second.t;
    return RTM_OK;
}

struct ShiftEntry {
    double2* d64 = nullptr;
    float2* d32 = nullptr;
};
static std::map<std::pair<TableKey, int>, ShiftEntry> g_shifts;

int shift_factors(int n, int parity, const double2** out64, const float2** out32) {
    // generateShiftPhases.m:16-17: s(m) = exp(i pi (2m + parity) / n); returns u(m) = 1 - s(m).
    int dev = 0;
    RTM_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_tables_mu);
    auto key = std::make_pair(TableKey{dev, n}, parity);
    auto it = g_shifts.find(key);
    if (it == g_shifts.end()) {
        const long double pi = 3.141592653589793238462643383279502884L;
        std::vector<double2> u(n);
        std::vector<float2> u32(n);
        for (int m = 0; m < n; ++m) {
            long double a = pi * (long double)(2 * m + parity) / (long double)n;
            u[m] = make_double2((double)(1.0L - cosl(a)), (double)(-sinl(a)));
            u32[m] = make_float2((float)u[m].x, (float)u[m].y);
        }
        ShiftEntry e;
        RTM_CUDA(cudaMalloc(&e.d64, n * sizeof(double2)));
        RTM_CUDA(cudaMalloc(&e.d32, n * sizeof(float2)));
        RTM_CUDA(cudaMemcpy(e.d64, u.data(), n * sizeof(double2), cudaMemcpyHostToDevice));
        RTM_CUDA(cudaMemcpy(e.d32, u32.data(), n * sizeof(float2), cudaMemcpyHostToDevice));
        it = g_shifts.emplace(key, e).first;
    }
    *out64 = it->second.d64;
    *out32 = it->second.d32;
    return RTM_OK;
}

// ---------------------------------------------------------------------------------------------
// Gauss-Legendre points and weights on [a, b] by Newton's method on P_n (same rule as the
// Golub-Welsch eigenvalue method of generateGaussLegendre1D.m:16-25, to rounding).
static void gauss_legendre_unit(int order, std::vector<double>& points, std::vector<double>& weights) {
    points.assign(order, 0.0);
    weights.assign(order, 0.0);
    const long double pi = 3.141592653589793238462643383279502884L;
    // P_order and its derivative at x by the three-term recurrence.
    auto legendre = [order](long double x, long double& p, long double& dp) {
        long double p0 = 1, p1 = x;
        for (int k = 2; k <= order; ++k) {
            long double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
            p0 = p1;
            p1 = p2;
        }
        p = order == 0 ? 1 : p1;
        dp = order * (x * p1 - p0) / (x * x - 1);
    };
    if (order == 1) {
        points[0] = 0.0;
        weights[0] = 2.0;
    } else {
        for (int i = 0; i < order / 2; ++i) {
            long double x = cosl(pi * (i + 0.75L) / (order + 0.5L));
            long double p = 0, dp = 1;
            for (int iter = 0; iter < 100; ++iter) {
                legendre(x, p, dp);
                const long double dx = p / dp;
                x -= dx;
                if (fabsl(dx) < 1e-19L) break;
            }
            legendre(x, p, dp);
            const long double w = 2 / ((1 - x * x) * dp * dp);
            points[i] = (double)(-x);
            points[order - 1 - i] = (double)x;
            weights[i] = weights[order - 1 - i] = (double)w;
        }
        if (order % 2 == 1) {
            long double p = 0, dp = 1;
            legendre(0.0L, p, dp);
            points[order / 2] = 0.0;
            weights[order / 2] = (double)(2 / (dp * dp));
        }
    }
}

// The rules of an order on [a, b]. The unit rules of orders up to kCachedOrder are computed once a process (an
// assembly asks for seven, about 1 ms of long-double Newton steps otherwise).
void gauss_legendre(int order, double a, double b, std::vector<double>& points, std::vector<double>& weights) {
    constexpr int kCachedOrder = 64;
    static std::mutex mu;
    static std::map<int, std::pair<std::vector<double>, std::vector<double>>> unit;
    if (order > kCachedOrder) {
        gauss_legendre_unit(order, points, weights);
    } else {
        std::lock_guard<std::mutex> lk(mu);
        auto it = unit.find(order);
        if (it == unit.end()) {
            gauss_legendre_unit(order, points, weights);
            it = unit.emplace(order, std::make_pair(points, weights)).first;
        }
        points = it->second.first;
        weights = it->second.second;
    }
    for (int i = 0; i < order; ++i) {
        points[i] = (a + b) / 2 + (b - a) / 2 * points[i];
        weights[i] = (b - a) / 2 * weights[i];
    }
}

// ---------------------------------------------------------------------------------------------
// Closed-form moments of R^power over the touching offsets (generatePowerMoments.m:17-155,
// integrateMonomial.m:18-81). The mixed antiderivatives are the integrals themselves.
static double monomial(int power, int m, int n, double a, double b) {
    if (a == 0 || b == 0) return 0.0;
    const double R = std::sqrt(a * a + b * b);
    const double lb = std::asinh(b / a), la = std::asinh(a / b);
    const double a2 = a * a, b2 = b * b, a4 = a2 * a2, b4 = b2 * b2;
    auto P = [](double x, int k) { double r = 1; for (int i = 0; i < k; ++i) r *= x; return r; };
    if (power == -1) {
        if (m == 0 && n == 0) return a * lb + b * la;
        if (m == 0 && n == 1) return (-a2 + a * R + b2 * la) / 2;
        if (m == 1 && n == 0) return (-b2 + b * R + a2 * lb) / 2;
        if (m == 1 && n == 1) return (-P(a, 3) - P(b, 3) + (a2 + b2) * R) / 3;
        if (m == 2 && n == 0) return (a * b * R + 2 * P(a, 3) * lb - P(b, 3) * la) / 6;
        if (m == 2 && n == 1) return (-2 * a4 + a * (2 * a2 + b2) * R - b4 * la) / 8;
        if (m == 3 && n == 0) return (2 * b4 + b * (a2 - 2 * b2) * R + 3 * a4 * lb) / 12;
        if (m == 3 && n == 1) return (-3 * P(a, 5) + 2 * P(b, 5) + (3 * a4 + a2 * b2 - 2 * b4) * R) / 15;
    } else if (power == 1) {
        if (m == 0 && n == 0) return (2 * a * b * R + P(a, 3) * lb + P(b, 3) * la) / 6;
        if (m == 0 && n == 1) return (-2 * a4 + a * (2 * a2 + 5 * b2) * R + 3 * b4 * la) / 24;
        if (m == 1 && n == 0) return (-2 * b4 + b * (5 * a2 + 2 * b2) * R + 3 * a4 * lb) / 24;
        if (m == 1 && n == 1) return (-P(a, 5) - P(b, 5) + (a4 + 2 * a2 * b2 + b4) * R) / 15;
        if (m == 2 && n == 0) return (a * b * (6 * a2 + b2) * R + 4 * P(a, 5) * lb - P(b, 5) * la) / 40;
        if (m == 2 && n == 1) return (-8 * P(a, 6) + a * (8 * a4 + 14 * a2 * b2 + 3 * b4) * R - 3 * P(b, 6) * la) / 144;
        if (m == 3 && n == 0) return (4 * P(b, 6) + b * (21 * a4 + 2 * a2 * b2 - 4 * b4) * R + 15 * P(a, 6) * lb) / 180;
        if (m == 3 && n == 1)
            return (-5 * P(a, 7) + 2 * P(b, 7) + (5 * P(a, 6) + 8 * a4 * b2 + a2 * b4 - 2 * P(b, 6)) * R) / 105;
    } else if (power == 3) {
        if (m == 0 && n == 0) return (7 * a * b * (a2 + b2) * R + 3 * P(a, 5) * lb + 3 * P(b, 5) * la) / 40;
        if (m == 0 && n == 1) return (-8 * P(a, 6) + a * (8 * a4 + 26 * a2 * b2 + 33 * b4) * R + 15 * P(b, 6) * la) / 240;
        if (m == 1 && n == 0) return (-8 * P(b, 6) + b * (33 * a4 + 26 * a2 * b2 + 8 * b4) * R + 15 * P(a, 6) * lb) / 240;
        if (m == 1 && n == 1)
            return (-P(a, 7) - P(b, 7) + (P(a, 6) + 3 * a4 * b2 + 3 * a2 * b4 + P(b, 6)) * R) / 35;
        if (m == 2 && n == 0)
            return (a * b * (38 * a4 + 26 * a2 * b2 + 3 * b4) * R + 18 * P(a, 7) * lb - 3 * P(b, 7) * la) / 336;
        if (m == 2 && n == 1)
            return (-48 * P(a, 8) + a * (48 * P(a, 6) + 136 * a4 * b2 + 118 * a2 * b4 + 15 * P(b, 6)) * R -
                    15 * P(b, 8) * la) / 1920;
        if (m == 3 && n == 0)
            return (16 * P(b, 8) + b * (215 * P(a, 6) + 134 * a4 * b2 + 8 * a2 * b4 - 16 * P(b, 6)) * R +
                    105 * P(a, 8) * lb) / 2240;
        if (m == 3 && n == 1)
            return (-7 * P(a, 9) + 2 * P(b, 9) +
                    (7 * P(a, 8) + 19 * P(a, 6) * b2 + 15 * a4 * b4 + a2 * P(b, 6) - 2 * P(b, 8)) * R) / 315;
    }
    return NAN;
}

// rect[q][m][n][iu][iv]: integral of u^m v^n R^power over [iu, iu+1] x ratio [iv, iv+1], power = kPowers[q]. The
// rectangles away from the corner take a 20 x 20-point rule, all powers and monomials at once from one square root
// a point (a pow per factor had cost 1.2 ms an assembly).
static const int kPowers[3] = {-1, 1, 3};
static void rectangles(double ratio, double rect[3][4][2][2][2]) {
    for (int q = 0; q < 3; ++q)
        for (int m = 0; m < 4; ++m)
            for (int n = 0; n < 2; ++n) {
                double c[3][3];
                for (int k = 0; k < 3; ++k)
                    for (int l = 0; l < 3; ++l) c[k][l] = monomial(kPowers[q], m, n, (double)k, ratio * l);
                for (int k = 0; k < 2; ++k)
                    for (int l = 0; l < 2; ++l)
                        rect[q][m][n][k][l] = (c[k + 1][l + 1] - c[k][l + 1]) - (c[k + 1][l] - c[k][l]);
            }
    std::vector<double> pts, w;
    gauss_legendre(20, 0.0, 1.0, pts, w);
    for (int k = 0; k < 2; ++k)
        for (int l = 0; l < 2; ++l) {
            if (std::hypot((double)k, ratio * l) < std::max(1.0, ratio)) continue;
            double s[3][4][2] = {};
            for (int i = 0; i < 20; ++i) {
                double inner[3][2] = {};
                const double u = k + pts[i];
                for (int j = 0; j < 20; ++j) {
                    const double v = ratio * (l + pts[j]);
                    const double r2 = u * u + v * v, r = std::sqrt(r2);
                    const double f[3] = {1.0 / r, r, r * r2};
                    for (int q = 0; q < 3; ++q) {
                        inner[q][0] += w[j] * f[q];
                        inner[q][1] += w[j] * v * f[q];
                    }
                }
                double um = 1;
                for (int m = 0; m < 4; ++m, um *= u)
                    for (int q = 0; q < 3; ++q)
                        for (int n = 0; n < 2; ++n) s[q][m][n] += w[i] * (um * inner[q][n]);
            }
            for (int q = 0; q < 3; ++q)
                for (int m = 0; m < 4; ++m)
                    for (int n = 0; n < 2; ++n) rect[q][m][n][k][l] = ratio * s[q][m][n];
        }
}

static const double kWeights[4][2][4] = {
    {{1.0, 1.0, 0, 0}, {1.0, -1.0, 0, 0}},
    {{0.5, 1.0, 0.5, 0}, {0.5, 0.0, -0.5, 0}},
    {{0.5, 0.0, -0.5, 0}, {0.5, -1.0, 0.5, 0}},
    {{1.0 / 3, 0.5, 0.0, -1.0 / 6}, {1.0 / 3, -0.5, 0.0, 1.0 / 6}},
};
static const int kWeightLen[4] = {2, 3, 3, 4};
static const int kTouching[4][2] = {{0, 0}, {1, 0}, {0, 1}, {1, 1}};

// The weight on part [-1,0] or [0,1] as a polynomial in u = sigma * cell * (nu - offset).
static void compose_part(const double* weight, int len, int part, int offset, double cell, int count, double* coeffs,
                         int* interval) {
    const double e0 = part == 0 ? -1.0 : 0.0, e1 = part == 0 ? 0.0 : 1.0;
    const double s0 = e0 - offset, s1 = e1 - offset;
    const double sigma = s1 <= 0 ? -1.0 : 1.0;
    *interval = (int)std::min(sigma * s0, sigma * s1);
    for (int i = 0; i < count; ++i) coeffs[i] = 0;
    double term[8] = {1, 0, 0, 0, 0, 0, 0, 0};
    int tl = 1;
    for (int k = 0; k < len; ++k) {
        for (int i = 0; i < tl && i < count; ++i) coeffs[i] += weight[k] * term[i];
        double nt[8] = {0};
        for (int i = 0; i < tl; ++i) {
            nt[i] += term[i] * offset;
            nt[i + 1] += term[i] * (sigma / cell);
        }
        ++tl;
        for (int i = 0; i < tl; ++i) term[i] = nt[i];
    }
}

static void along_x(double a, double b, int power, const double rect[4][2][2][2], double out[4][4]) {
    const double ratio = b / a;
    for (int k = 0; k < 4; ++k)
        for (int l = 0; l < 4; ++l) {
            double acc = 0;
            for (int s = 0; s < 2; ++s) {
                double ca[4];
                int ia;
                compose_part(kWeights[k][s], kWeightLen[k], s, kTouching[l][0], 1.0, 4, ca, &ia);
                for (int t = 0; t < 2; ++t) {
                    double cb[2];
                    int ib;
                    compose_part(kWeights[0][t], kWeightLen[0], t, kTouching[l][1], ratio, 2, cb, &ib);
                    for (int m = 0; m < 4; ++m)
                        for (int n = 0; n < 2; ++n) acc += ca[m] * rect[m][n][ia][ib] * cb[n];
                }
            }
            out[k][l] = std::pow(a, power) * acc / ratio;
        }
}

// rx, ry: the rectangles of kPowers' entry `power` for the ratios size_y / size_x and size_x / size_y.
static void power_moments(double size_x, double size_y, int power, const double rx[4][2][2][2],
                          const double ry[4][2][2][2], double out[7][4]) {
    double ax[4][4], ay[4][4];
    along_x(size_x, size_y, power, rx, ax);
    along_x(size_y, size_x, power, ry, ay);
    static const int perm[4] = {0, 2, 1, 3};
    for (int l = 0; l < 4; ++l) {
        for (int k = 0; k < 4; ++k) out[k][l] = ax[k][l];
        for (int k = 1; k < 4; ++k) out[3 + k][l] = ay[k][perm[l]];
    }
}

void extracted_moments(double size_x, double size_y, double k, double out[7][4]) {
    double m[3][7][4], rx[3][4][2][2][2], ry[3][4][2][2][2];
    rectangles(size_y / size_x, rx);
    rectangles(size_x / size_y, ry);
    for (int q = 0; q < 3; ++q) power_moments(size_x, size_y, kPowers[q], rx[q], ry[q], m[q]);
    const auto &m1 = m[0], &p1 = m[1], &p3 = m[2];
    for (int r = 0; r < 7; ++r)
        for (int c = 0; c < 4; ++c) out[r][c] = m1[r][c] - k * k / 2 * p1[r][c] + k * k * k * k / 24 * p3[r][c];
}

}  // namespace rtm

// ---------------------------------------------------------------------------------------------
extern "C" int rtm_last_error(char* buf, size_t len) {
    if (!buf || len == 0) return RTM_ERR_ARG;
    const std::string& e = rtm::t_error;
    const size_t n = std::min(len - 1, e.size());
    std::memcpy(buf, e.data(), n);
    buf[n] = '\0';
    return RTM_OK;
}

extern "C" int rtm_budget_configure(double ceiling_bytes) {
    std::lock_guard<std::mutex> lk(rtm::g_budget_mu);
    rtm::g_ceiling = ceiling_bytes > 0 ? ceiling_bytes : 0.0;
    return RTM_OK;
}

extern "C" int rtm_budget_query(double* ceiling_bytes, double* held_bytes) {
    std::lock_guard<std::mutex> lk(rtm::g_budget_mu);
    if (ceiling_bytes) *ceiling_bytes = rtm::g_ceiling;
    if (held_bytes) *held_bytes = rtm::g_held;
    return RTM_OK;
}

