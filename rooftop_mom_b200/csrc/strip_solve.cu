// COCG on strips in one kernel. The vectors, lines and roots of a plate one face wide fit one CTA's shared memory (up to
// about 1600 unknowns in FP64), so a CTA per right-hand side runs whole iterations (the recurrences of krylov.cu's cocg,
// ConjugateGradient.m:12-62) from there. The general form launches six kernels an iteration for a few microseconds of
// work each, 16 iterations at a time: 845 us for a strip of 400 faces that converges in 6; this
// takes 132 us on the device, 241 with the call around it.
//
// Bound: latency, a chain of four line transforms, two products with spectra and three sums over the CTA an iteration.
// The transforms are the Stockham stages of fft.cuh, small functions a whole CTA shares; the register-resident ones of
// regfft.cuh would bring 86 codelets into this one kernel and spill.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft.cuh"
#include "grid.h"
#include "krylov.h"

namespace rtm {
namespace {

constexpr int kStripThreads = 256;
constexpr int kStripLaunch = 512;  // iterations a launch runs at most, where no cancel can arrive
constexpr size_t kStripSmem = 200 * 1024;

// One strip product: ns subbands of a line of plan.n points (k_strip in grid.cu).
template <typename T> struct StripOp {
    using T2 = typename Cx<T>::T2;
    FftPlan plan;
    int ns, ls;       // subbands; elements of a line's buffer
    const T2* tw;     // roots
    const T2* mod;    // odd subband's modulation
    const T2* spec;   // [ns][plan.n]
    T scale;
};

struct StripState {
    double2 rho;
    double bnorm, residual;  // ||b||, and ||b - A x|| once done
    int iteration, done, converged, zero_rhs;
};

template <typename T> struct StripArgs {
    using T2 = typename Cx<T>::T2;
    StripOp<T> op[2];      // the product, the preconditioner
    int has_m;
    int n, first;          // unknowns; 1: the launch that starts the solve
    int has_x0;
    double tol;
    const double* tols;    // one per right-hand side, or null
    int max_iterations, limit;
    int lines;             // elements of the lines' buffer
    const T2* b;
    T2* x;                 // the initial guess on entry where has_x0
    T2* r;
    T2* d;
    StripState* st;
    double* hist;
    int hist_stride;
};

// out = Op in, both n entries in shared memory (tws: the operator's roots there); starts and ends with the CTA in step.
template <typename T, typename T2>
__device__ __forceinline__ void strip_apply(const StripOp<T>& o, int n, T2* A, const T2* tws, const T2* in, T2* out) {
    const int L = o.plan.n, ls = o.ls, ns = o.ns;
    for (int i = threadIdx.x; i < L; i += kStripThreads) {
        const T2 v = i < n ? in[i] : czero<T2>();
        A[sk(i)] = v;
        if (ns == 2) A[ls + sk(i)] = cmul(v, __ldg(&o.mod[i]));
    }
    __syncthreads();
    fft_inplace<false, false>(A, ns, ls, 1, o.plan, tws);
    for (int it = threadIdx.x; it < ns * L; it += kStripThreads) {
        const int s = it / L, i = it - s * L;
        A[s * ls + sk(i)] = cmul(A[s * ls + sk(i)], __ldg(&o.spec[it]));
    }
    __syncthreads();
    fft_inplace<true, false>(A, ns, ls, 1, o.plan, tws);
    for (int i = threadIdx.x; i < n; i += kStripThreads) {
        T2 v = A[sk(i)];
        if (ns == 2) v = cadd(v, cmulc(A[ls + sk(i)], __ldg(&o.mod[i])));
        out[i] = cscale(v, o.scale);
    }
    __syncthreads();
}

__device__ __forceinline__ double2 wide(double2 v) { return v; }
__device__ __forceinline__ double2 wide(float2 v) { return make_double2(v.x, v.y); }

// The CTA's sum of v, for every thread.
__device__ __forceinline__ double2 strip_sum(double2 v) {
    __shared__ double2 part[kStripThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
    __syncthreads();  // the sum before is read
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    double2 s = make_double2(0, 0);
#pragma unroll
    for (int w = 0; w < kStripThreads / 32; ++w) s = cadd(s, part[w]);
    return s;
}

__device__ __forceinline__ double2 strip_div(double2 a, double2 b) {
    const double d = b.x * b.x + b.y * b.y;
    return make_double2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}

// The solve as a chain of operator applies, so that their codelets (most of the kernel's code) stand here once.
enum StripPhase { kInit, kPrecondition, kMultiply, kFinal };

template <typename T> __global__ void __launch_bounds__(kStripThreads, 1) k_strip_cocg(const __grid_constant__ StripArgs<T> a) {
    using T2 = typename Cx<T>::T2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = a.n, rhs = blockIdx.x, tid = threadIdx.x;
    T2* lines = reinterpret_cast<T2*>(smem_raw);
    T2* roots = lines + a.lines;  // of the product, then of the preconditioner
    T2* x = roots + a.op[0].plan.n + (a.has_m ? a.op[1].plan.n : 0);
    T2* r = x + n;
    T2* d = r + n;
    T2* q = d + n;
    T2* z = a.has_m ? q + n : r;
    const T2* b = a.b + (int64_t)rhs * n;
    T2* xg = a.x + (int64_t)rhs * n;
    T2* rg = a.r + (int64_t)rhs * n;
    T2* dg = a.d + (int64_t)rhs * n;
    double* hist = a.hist + (int64_t)rhs * a.hist_stride;
    StripState S = a.st[rhs];
    if (!a.first && S.done) return;
    const double tol = a.tols ? a.tols[rhs] : a.tol;
    int phase, it = 0;
    // vectors in T, products and sums over the CTA in FP64
    auto norm2 = [&](const T2* v) {
        double2 s = make_double2(0, 0);
        for (int i = tid; i < n; i += kStripThreads) {
            const double2 w = wide(v[i]);
            s.x += w.x * w.x + w.y * w.y;
        }
        return strip_sum(s).x;
    };
    auto dot = [&](const T2* u, const T2* v) {
        double2 s = make_double2(0, 0);
        for (int i = tid; i < n; i += kStripThreads) s = cadd(s, cmul(wide(u[i]), wide(v[i])));
        return strip_sum(s);
    };
    for (int k = 0; k <= a.has_m; ++k)
        for (int i = tid; i < a.op[k].plan.n; i += kStripThreads) roots[(k ? a.op[0].plan.n : 0) + i] = a.op[k].tw[i];
    // what follows a residual in r: the next iteration's preconditioner or direction, or the end
    auto direction = [&]() {
        const double2 s = dot(r, z);
        const bool start = S.iteration == 0;
        const double2 beta = start ? make_double2(0, 0) : strip_div(s, S.rho);
        S.rho = s;
        for (int i = tid; i < n; i += kStripThreads) {
            const double2 w = cadd(wide(z[i]), cmul(beta, wide(d[i])));
            d[i] = start ? z[i] : cmake<T2>(w.x, w.y);
        }
    };
    auto next = [&]() {
        if (S.done || it >= a.limit) return (int)kFinal;
        if (a.has_m) return (int)kPrecondition;
        direction();
        return (int)kMultiply;
    };
    auto begin = [&]() {
        const double h0 = S.zero_rhs ? 0.0 : sqrt(norm2(r)) / S.bnorm;
        S.converged = S.zero_rhs || h0 < tol;
        S.done = S.converged || a.max_iterations <= 0;
        if (tid == 0) hist[0] = h0;
        return next();
    };
    if (a.first) {
        for (int i = tid; i < n; i += kStripThreads) {
            r[i] = b[i];
            x[i] = a.has_x0 ? xg[i] : czero<T2>();
            d[i] = czero<T2>();
        }
        for (int i = 1 + tid; i < a.hist_stride; i += kStripThreads) hist[i] = NAN;
        S.rho = make_double2(0, 0);
        S.bnorm = sqrt(norm2(r));
        S.iteration = 0;
        S.residual = 0;
        S.zero_rhs = S.bnorm == 0.0;
        phase = a.has_x0 ? (int)kInit : begin();
    } else {
        for (int i = tid; i < n; i += kStripThreads) {
            x[i] = xg[i];
            r[i] = rg[i];
            d[i] = dg[i];
        }
        phase = next();
    }
    while (true) {
        const bool pre = phase == kPrecondition;
        __syncthreads();  // the input is written
        strip_apply(a.op[pre], n, lines, roots + (pre ? a.op[0].plan.n : 0), pre ? r : phase == kMultiply ? d : x,
                    pre ? z : q);
        if (phase == kFinal) break;
        if (phase == kInit) {
            for (int i = tid; i < n; i += kStripThreads) r[i] = csub(r[i], q[i]);
            phase = begin();
        } else if (phase == kPrecondition) {
            direction();
            phase = kMultiply;
        } else {
            const double2 alpha = strip_div(S.rho, dot(d, q));
            for (int i = tid; i < n; i += kStripThreads) {
                const double2 u = cadd(wide(x[i]), cmul(alpha, wide(d[i])));
                const double2 v = csub(wide(r[i]), cmul(alpha, wide(q[i])));
                x[i] = cmake<T2>(u.x, u.y);
                r[i] = cmake<T2>(v.x, v.y);
            }
            const double h = sqrt(norm2(r)) / S.bnorm;
            S.iteration += 1;
            ++it;
            S.converged = h < tol;
            // a breakdown (d^T A d = 0) leaves Inf or NaN (ConjugateGradient.m:55-58)
            S.done = S.converged || !isfinite(h) || S.iteration >= a.max_iterations;
            if (tid == 0) hist[S.iteration] = h;
            phase = next();
        }
    }
    // q = A x: the true residual of the current iterate (IterativeMethod.m:52), whether the solve is done or stops here
    double2 s = make_double2(0, 0);
    for (int i = tid; i < n; i += kStripThreads) {
        const double2 v = csub(wide(b[i]), wide(q[i]));
        s.x += v.x * v.x + v.y * v.y;
    }
    S.residual = sqrt(strip_sum(s).x);
    for (int i = tid; i < n; i += kStripThreads) {
        xg[i] = S.zero_rhs ? czero<T2>() : x[i];
        rg[i] = r[i];
        dg[i] = d[i];
    }
    if (tid == 0) a.st[rhs] = S;
}

template <typename T> bool strip_op(const LinearOp* op, StripOp<T>* out) {
    using T2 = typename Cx<T>::T2;
    const auto* g = dynamic_cast<const GridApplicator*>(op);
    if (!g || g->mode != kStrip || (g->precision == RTM_FP64) != (sizeof(T) == 8)) return false;
    out->plan = g->tP->plan;
    out->ns = g->nsx;
    out->ls = fft_span(out->plan) + 2;  // the second line starts on other banks
    if constexpr (sizeof(T) == 8) {
        out->tw = g->tP->tw64;
        out->mod = g->tP->mod64;
    } else {
        out->tw = g->tP->tw32;
        out->mod = g->tP->mod32;
    }
    out->spec = g->spec.as<T2>();
    out->scale = (T)(1.0 / g->P);
    return fft_threads(out->ns, out->plan) <= kStripThreads;
}

}  // namespace

template <typename T>
int strip_cocg(LinearOp* A, LinearOp* M, const SolveConfig& cfg, const void* b, const void* x0, void* x, int64_t n,
               int nrhs, SolveResult& res, cudaStream_t s, bool* taken) {
    using T2 = typename Cx<T>::T2;
    *taken = false;
    StripArgs<T> a{};
    if (!strip_op(A, &a.op[0]) || (M && !strip_op(M, &a.op[1]))) return RTM_OK;
    a.has_m = M != nullptr;
    a.lines = a.op[0].ns * a.op[0].ls;
    if (M) a.lines = std::max(a.lines, a.op[1].ns * a.op[1].ls);
    const size_t smem = ((size_t)a.lines + a.op[0].plan.n + (M ? a.op[1].plan.n : 0) + (M ? 5 : 4) * (size_t)n) * sizeof(T2);
    if (smem > kStripSmem) return RTM_OK;
    *taken = true;
    a.n = (int)n;
    a.has_x0 = x0 != nullptr;
    a.tol = cfg.tolerance;
    a.max_iterations = cfg.max_iterations;
    static DeviceOnce once;
    RTM_TRY(once([]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_strip_cocg<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStripSmem));
        return RTM_OK;
    }));
    const size_t vec = (size_t)n * nrhs * sizeof(T2);
    const int hs = cfg.max_iterations + 1;
    // history and states in one block, so that one copy brings both back
    const size_t hist_bytes = (sizeof(double) * (size_t)hs * nrhs + 15) / 16 * 16;
    const size_t back_bytes = hist_bytes + sizeof(StripState) * nrhs;
    DeviceBuffer rd, back, tols;
    StreamSyncGuard guard(s);
    RTM_TRY(rd.alloc(2 * vec));
    RTM_TRY(back.alloc(back_bytes));
    if (cfg.tolerances) {
        RTM_TRY(tols.alloc(sizeof(double) * nrhs));
        RTM_CUDA(cudaMemcpyAsync(tols.ptr, cfg.tolerances, tols.bytes, cudaMemcpyHostToDevice, s));
        a.tols = tols.as<double>();
    }
    if (x0) RTM_CUDA(cudaMemcpyAsync(x, x0, vec, cudaMemcpyDeviceToDevice, s));
    a.b = static_cast<const T2*>(b);
    a.x = static_cast<T2*>(x);
    a.r = rd.as<T2>();
    a.d = a.r + (int64_t)n * nrhs;
    a.hist = back.as<double>();
    a.hist_stride = hs;
    a.st = reinterpret_cast<StripState*>(back.as<char>() + hist_bytes);
    std::vector<char> host(back_bytes);
    const auto* st = reinterpret_cast<const StripState*>(host.data() + hist_bytes);
    // a cancel is looked for before the first iteration and after every check_every (krylov.cu's cocg does the same)
    const int limit = !cfg.cancel ? kStripLaunch : cfg.check_every > 0 ? cfg.check_every : 16;
    const bool small = hist_bytes <= 16 * 1024;  // the history comes back with every look at the states, or once
    for (a.first = 1;; a.first = 0) {
        a.limit = cfg.cancel && *cfg.cancel ? 0 : limit;
        k_strip_cocg<T><<<nrhs, kStripThreads, smem, s>>>(a);
        count_launch();
        RTM_CUDA(cudaGetLastError());
        const size_t from = small ? 0 : hist_bytes;
        RTM_CUDA(cudaMemcpyAsync(host.data() + from, back.as<char>() + from, back_bytes - from, cudaMemcpyDeviceToHost, s));
        RTM_CUDA(cudaStreamSynchronize(s));
        bool all = true;
        for (int k = 0; k < nrhs; ++k) all = all && st[k].done;
        if (all || (cfg.cancel && *cfg.cancel)) break;
    }
    if (!small) {
        RTM_CUDA(cudaMemcpyAsync(host.data(), back.ptr, hist_bytes, cudaMemcpyDeviceToHost, s));
        RTM_CUDA(cudaStreamSynchronize(s));
    }
    const auto* hist = reinterpret_cast<const double*>(host.data());
    res.history.assign(hist, hist + (size_t)hs * nrhs);
    res.hist_stride = hs;
    res.matvecs = x0 ? 1 : 0;
    res.stats.resize(nrhs);
    for (int k = 0; k < nrhs; ++k) {
        rtm_solve_stats& o = res.stats[k];
        o.converged = st[k].converged;
        o.iteration_count = st[k].zero_rhs ? 0 : st[k].iteration;
        o.residual_norm = st[k].zero_rhs ? 0.0 : st[k].residual / st[k].bnorm;
        o.refinements = 0;
        o.matvecs = res.matvecs + st[k].iteration + 1;
    }
    return RTM_OK;
}

template int strip_cocg<float>(LinearOp*, LinearOp*, const SolveConfig&, const void*, const void*, void*, int64_t, int,
                               SolveResult&, cudaStream_t, bool*);
template int strip_cocg<double>(LinearOp*, LinearOp*, const SolveConfig&, const void*, const void*, void*, int64_t, int,
                                SolveResult&, cudaStream_t, bool*);

}  // namespace rtm
