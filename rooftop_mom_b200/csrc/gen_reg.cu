// The spectra builders' transforms on register-resident lines (regfft.cuh), in FP64: sources along y, then rows along x.
//
// The generators' embeddings and circulant folds are even in both directions. Along x the unmodulated source at P - i is
// the one at i, negated for the odd subband, so the y pass transforms P / 2 + 1 columns; along y the transforms are even
// in the frequency, so Q / 2 + 1 rows are kept, transformed along x and written twice. Twelve spectra of 256 x 256 points:
// 88 + 42 us on the Stockham kernels of grid.cu (255 registers, 11 % of the warps active), which write and read every row; 33 + 8
// here.
#include <algorithm>

#include "gen.cuh"
#include "regfft.cuh"

namespace rtm {
namespace {

__device__ __forceinline__ bool even_source(const GenArgs& a) { return a.kind == kSrcEmbed || a.kind == kSrcCirculant; }

// y pass: TI columns of one item, line-fastest (thread line + TI t); dst[k][i] = FFT_y(source(i, j)).
template <int CLS, bool BLUE>
__global__ void __launch_bounds__(RegShape<double, CLS>::threads, (RegShape<double, CLS>::blocks))
    k_reg_gen_y(const GenArgs a, const RegPlan q) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const GenItem& item = a.items[blockIdx.y];
    const int TI = a.ti, t = threadIdx.x / TI, line = threadIdx.x - t * TI;
    const int i = blockIdx.x * TI + line;
    const bool even = even_source(a), on = i < (even ? a.P / 2 + 1 : a.P);
    const int keep = even ? a.Q / 2 : a.Q - 1;  // the highest row kept
    const RegLine<double2> buf{reinterpret_cast<double2*>(smem_raw) + line, q.n2 * TI, TI};
    double2* dst = item.dst + i;
    // through the line's buffer (only thread t touches column t of it): the sources' code stands here once
    if (on && t < q.n2) {
#pragma unroll 4
        for (int m1 = 0; m1 < q.n1; ++m1) {
            const int j = q.n2 * m1 + t;
            buf.at(m1, t) = j < q.n ? gen_value(a, item, i, j, !even) : make_double2(0, 0);
        }
    }
    with_n1<CLS>(q.n1, [&](auto len) {
        constexpr int R = decltype(len)::value;
        if (!on || t >= q.n2) return;
        double2 v[R];
#pragma unroll
        for (int m1 = 0; m1 < R; ++m1) v[m1] = buf.at(m1, t);
        if constexpr (BLUE) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) v[m1] = cmul(v[m1], __ldg(&q.chirp64[min(q.n2 * m1 + t, q.n - 1)]));
        }
        reg_a_fwd<R>(v, t, q.tw64, buf);
    });
    if constexpr (BLUE) {
        reg_convolve<CLS, false>(q, t, on, buf);
        with_n1<CLS>(q.n1, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= q.n2) return;
            double2 v[R];
            reg_a_inv<R>(v, t, buf);
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int j = q.n2 * m1 + t;
                const double2 w = cmul(v[m1], __ldg(&q.chirp64[min(j, q.n - 1)]));
                if (j <= keep) dst[(int64_t)j * a.P] = w;
            }
        });
    } else {
        __syncthreads();
        with_n2<CLS>(q.n2, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= q.n1) return;
            double2 v[R];
            reg_b_fwd<R>(v, t, buf);
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) {
                const int k = t + q.n1 * k2;
                if (k <= keep) dst[(int64_t)k * a.P] = v[k2];
            }
        });
    }
}

// x pass: rows of one item in place, a line a row (thread t + n1 line).
template <int CLS, bool BLUE>
__global__ void __launch_bounds__(RegShape<double, CLS>::threads, (RegShape<double, CLS>::blocks))
    k_reg_gen_x(const GenArgs a, const RegPlan p, int lines) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const GenItem& item = a.items[blockIdx.y];
    const int line = threadIdx.x / p.n1, t = threadIdx.x - line * p.n1, ls = p.n1 * (p.n2 | 1);
    const int j = blockIdx.x * lines + line;
    const bool even = even_source(a);
    const int mirror = a.Q - j - item.py;  // the row with the same spectrum
    const bool on = line < lines && (even ? j <= mirror : j < a.Q);
    const bool twice = even && mirror != j && mirror < a.Q;
    const RegLine<double2> buf{reinterpret_cast<double2*>(smem_raw) + (on ? line : 0) * ls, p.n2 | 1, 1};
    double2* row = item.dst + (int64_t)(on ? j : 0) * a.P;
    double2* copy = item.dst + (int64_t)(on && twice ? mirror : 0) * a.P;
    auto put = [&](int k, double2 v) {
        if (a.realify) v.y = 0.0;
        row[k] = v;
        if (twice) copy[k] = v;
    };
    with_n1<CLS>(p.n1, [&](auto len) {
        constexpr int R = decltype(len)::value;
        if (!on || t >= p.n2) return;
        double2 v[R];
#pragma unroll
        for (int m1 = 0; m1 < R; ++m1) {
            const int i = p.n2 * m1 + t;
            const bool far = even && 2 * i > a.P;
            double2 w = i < p.n ? row[far ? a.P - i : i] : make_double2(0, 0);
            if (far && item.px) w = make_double2(-w.x, -w.y);
            v[m1] = w;
        }
        if (even && item.px) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) v[m1] = cmul(v[m1], __ldg(&a.modP[min(p.n2 * m1 + t, p.n - 1)]));
        }
        if constexpr (BLUE) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) v[m1] = cmul(v[m1], __ldg(&p.chirp64[min(p.n2 * m1 + t, p.n - 1)]));
        }
        reg_a_fwd<R>(v, t, p.tw64, buf);
    });
    if constexpr (BLUE) {
        reg_convolve<CLS, false>(p, t, on, buf);
        with_n1<CLS>(p.n1, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= p.n2) return;
            double2 v[R];
            reg_a_inv<R>(v, t, buf);
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int k = p.n2 * m1 + t;
                if (k < p.n) put(k, cmul(v[m1], __ldg(&p.chirp64[min(k, p.n - 1)])));
            }
        });
    } else {
        __syncthreads();
        with_n2<CLS>(p.n2, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= p.n1) return;
            double2 v[R];
            reg_b_fwd<R>(v, t, buf);
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) put(t + p.n1 * k2, v[k2]);
        });
    }
}

}  // namespace

template <int CLS, bool BLUE> int launch_reg_gen(bool x, const GenArgs& args, const RegPlan& r, cudaStream_t s) {
    GenArgs a = args;
    constexpr int kThreads = RegShape<double, CLS>::threads;
    const bool even = a.kind == kSrcEmbed || a.kind == kSrcCirculant;
    constexpr int kSmem = 200 * 1024;
    static DeviceOnce once;
    RTM_TRY(once([]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_reg_gen_y<CLS, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        RTM_CUDA(cudaFuncSetAttribute(k_reg_gen_x<CLS, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
        return RTM_OK;
    }));
    if (x) {
        const int lines = std::max(1, kThreads / r.n1), rows = even ? a.Q / 2 + 1 : a.Q;
        const int threads = (lines * r.n1 + 31) / 32 * 32;
        const size_t smem = (size_t)lines * r.n1 * (r.n2 | 1) * sizeof(double2);
        k_reg_gen_x<CLS, BLUE><<<dim3((rows + lines - 1) / lines, a.nitems), threads, smem, s>>>(a, r, lines);
    } else {
        a.ti = 4;  // columns of 64 bytes
        const int columns = even ? a.P / 2 + 1 : a.P, threads = (a.ti * r.n1 + 31) / 32 * 32;
        const size_t smem = (size_t)a.ti * r.m * sizeof(double2);
        k_reg_gen_y<CLS, BLUE><<<dim3((columns + a.ti - 1) / a.ti, a.nitems), threads, smem, s>>>(a, r);
    }
    count_launch();
    return RTM_OK;
}

// One form a translation unit (build.py), so that they compile side by side.
#if RTM_GEN_FORM == 0
template int launch_reg_gen<0, false>(bool, const GenArgs&, const RegPlan&, cudaStream_t);
#elif RTM_GEN_FORM == 1
template int launch_reg_gen<1, false>(bool, const GenArgs&, const RegPlan&, cudaStream_t);
#elif RTM_GEN_FORM == 2
template int launch_reg_gen<0, true>(bool, const GenArgs&, const RegPlan&, cudaStream_t);
#elif RTM_GEN_FORM == 3
template int launch_reg_gen<1, true>(bool, const GenArgs&, const RegPlan&, cudaStream_t);
#endif

}  // namespace rtm
