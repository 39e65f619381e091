// Products on transform grids of any length with a register-resident split (regfft.cuh): the embedding, lean and
// split products of grids that are no powers of two, and the circulant preconditioners.
//
// The same three passes as k_grid_y_fwd / k_grid_x_mix / k_grid_y_inv in grid.cu (the reference's
// @SplitFFTApplicator/applyBothDirections_.m:14-85, FFTApplicator.m:52-87), whose Stockham stages keep 255
// registers a thread and one CTA an SM (8 % of the warps active) and pass every radix through shared memory. An FP64 product
// of 301 x 187 faces: 175 us a call there, 45 here; both wait for loads and exchanges with few warps in flight, not for
// bandwidth or arithmetic. Passes along lengths of 256, 512 and 1024 run in three steps (grid_fast.cu).
#include <algorithm>

#include "grid.h"
#include "grid_args.cuh"
#include "pdl.cuh"
#include "regfft.cuh"

namespace rtm {
namespace {

// The lower of a frequency m of subband parity p on n frequencies and its mirror image (the generators' spectra
// are even, see grid_fast.cu).
__device__ __forceinline__ int lower_freq(int m, int p, int n) { return min(m, n - m - p); }

// A value of the stored precision in the precision of the transform, and back.
template <typename C2, typename T2> __device__ __forceinline__ C2 cast(T2 v) {
    using C = decltype(C2{}.x);
    C2 r;
    r.x = (C)v.x;
    r.y = (C)v.y;
    return r;
}

// The kernels below hold no condition on an element but those of its load and its store: tables are read at clamped
// positions and padding is multiplied along, since a branch an element breaks the straight run of instructions
// (100 x 72 faces, FP64, with such branches: 6.6 warps an issue waiting for instructions against 0.3).
//
// T: the vectors', W's and spectra's precision; C: the transforms'. They differ for FP32 lines that run as a
// Bluestein convolution, which transforms in FP64: in FP32 its three transforms would lose twice the digits of the
// direct form.

// y-forward: TI x columns of one component and npy subbands, L = npy TI lines, line-fastest (consecutive threads on
// consecutive columns): thread line + L t, line = pyi TI + l.
template <typename T, typename C, int CLS, bool BLUE>
__global__ void __launch_bounds__(RegShape<C, CLS>::threads, (RegShape<C, CLS>::blocks))
    k_reg_y_fwd(const GridArgs<T> a, const RegPlan q, const typename Cx<T>::T2* __restrict__ x) {
    using T2 = typename Cx<T>::T2;
    using C2 = typename Cx<C>::T2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    griddep_launch_dependents();
    const int c = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const int rows = a.rows[c], cols = a.cols[c];
    const int TI = a.ti, L = a.npy * TI;
    if ((int)blockIdx.x * TI >= rows) return;
    const int t = threadIdx.x / L, line = threadIdx.x - t * L;
    const int pyi = line / TI, i = blockIdx.x * TI + line - pyi * TI;
    const bool odd = (a.py0 + pyi) != 0, on = i < rows;
    const RegLine<C2> buf{reinterpret_cast<C2*>(smem_raw) + line, q.n2 * L, L};
    const C2* tw = RegTables<C2>::roots(q);
    const C2* chirp = RegTables<C2>::chirp(q);
    const T2* xr = x + (int64_t)rhs * a.n + a.off[c] + i;
    T2* dst = a.work + (int64_t)rhs * a.work_rhs + (int64_t)(pyi * a.ncomp + c) * a.Q * a.P + i;
    with_n1<CLS>(q.n1, [&](auto len) {
        constexpr int R = decltype(len)::value;
        if (!on || t >= q.n2) return;
        C2 v[R];
#pragma unroll
        for (int m1 = 0; m1 < R; ++m1) {
            const int j = q.n2 * m1 + t;
            v[m1] = cast<C2>(j < cols ? xr[(int64_t)j * rows] : czero<T2>());
        }
        if (odd) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int j = q.n2 * m1 + t;
                v[m1] = cmul(v[m1], cast<C2>(__ldg(&a.modQ[BLUE ? min(j, q.n - 1) : j])));
            }
        }
        if constexpr (BLUE) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) v[m1] = cmul(v[m1], __ldg(&chirp[min(q.n2 * m1 + t, q.n - 1)]));
        }
        reg_a_fwd<R>(v, t, tw, buf);
    });
    if constexpr (BLUE) {
        reg_convolve<CLS, false>(q, t, on, buf);
        with_n1<CLS>(q.n1, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= q.n2) return;
            C2 v[R];
            reg_a_inv<R>(v, t, buf);
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int j = q.n2 * m1 + t;
                const C2 w = cmul(v[m1], __ldg(&chirp[min(j, q.n - 1)]));
                if (j < q.n) dst[(int64_t)j * a.P] = cast<T2>(w);
            }
        });
    } else {
        __syncthreads();
        with_n2<CLS>(q.n2, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= q.n1) return;
            C2 v[R];
            reg_b_fwd<R>(v, t, buf);
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) dst[(int64_t)(t + q.n1 * k2) * a.P] = cast<T2>(v[k2]);
        });
    }
}

// The 2 x 2 mix of one line's transformed values: v[r] at frequency f0 + fs r of (x subband px, y frequency j of
// subband py); the partner component's values are exchanged at (at + step r) of the two lines' buffers. Starts
// with a write to the own buffer; ends with a barrier. BLUE: frequencies from P on are padding (clamped).
template <int R, bool BLUE, typename T, typename C2>
__device__ __forceinline__ void reg_mix(C2 (&v)[R], const GridArgs<T>& a, C2* own, const C2* partner, int at, int step,
                                        int f0, int fs, int c, int px, int py, int j, bool on) {
    using C = decltype(C2{}.x);
    using T2 = typename Cx<T>::T2;
    if (on) {
#pragma unroll
        for (int r = 0; r < R; ++r) own[at + step * r] = v[r];
    }
    __syncthreads();
    if (on) {
        const int64_t QP = (int64_t)a.Q * a.P;
        if (a.mode == kGen3) {
            const T2* spec = a.spec + (int64_t)((px + a.nsx * py) * 3) * QP + (int64_t)lower_freq(j, py, a.Q) * a.P;
            const T2* ux = px ? a.ux1 : a.ux0;
            const C2 vv = cast<C2>(__ldg(&(py ? a.vy1 : a.vy0)[j]));
            const C cv = (vv.x * vv.x + vv.y * vv.y) * (C)a.inv_b2;
            const C ia = (C)a.inv_a2, iab = (C)a.inv_ab;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int k = BLUE ? min(f0 + fs * r, a.P - 1) : f0 + fs * r;
                const int ke = lower_freq(k, px, a.P);
                const C2 E = cast<C2>(__ldg(&spec[ke]));
                const C2 M = cast<C2>(__ldg(&spec[(1 + c) * QP + ke]));
                const C2 uu = cast<C2>(__ldg(&ux[k]));
                const C cu = (uu.x * uu.x + uu.y * uu.y) * ia;
                // qc = -u conj(v) / (ab): XY = qc E, YX = conj(qc) E
                C2 qc = cmulc(uu, vv);
                qc.x = -qc.x * iab;
                qc.y = -qc.y * iab;
                if (c) qc.y = -qc.y;
                const C cself = c ? cv : cu;
                const C2 me = v[r], other = partner[at + step * r];
                // M me - cself E me + coupling E other = M me + E (coupling other - cself me)
                C2 d = cmul(qc, other);
                d.x -= cself * me.x;
                d.y -= cself * me.y;
                v[r] = cadd(cmul(M, me), cmul(E, d));
            }
        } else {
            // blocks XX, XY, YX, YY: row c of the 2 x 2 block
            const T2* same = a.spec + (int64_t)(c ? 3 : 0) * QP + (int64_t)j * a.P;
            const T2* cross = a.spec + (int64_t)(c ? 2 : 1) * QP + (int64_t)j * a.P;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int k = BLUE ? min(f0 + fs * r, a.P - 1) : f0 + fs * r;
                v[r] = cadd(cmul(cast<C2>(__ldg(&same[k])), v[r]),
                            cmul(cast<C2>(__ldg(&cross[k])), partner[at + step * r]));
            }
        }
    }
    __syncthreads();
}

// x-mix: CB y frequencies, nsx subbands and both components, line (jj nsx + px) 2 + c, thread t + n1 line.
template <typename T, typename C, int CLS, bool BLUE>
__global__ void __launch_bounds__(RegShape<C, CLS>::threads, (RegShape<C, CLS>::blocks))
    k_reg_x_mix(const GridArgs<T> a, const RegPlan p) {
    using T2 = typename Cx<T>::T2;
    using C2 = typename Cx<C>::T2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    griddep_launch_dependents();
    const int pyi = blockIdx.y, rhs = blockIdx.z, py = a.py0 + pyi;
    if (skipped(a, rhs)) return;
    const int line = threadIdx.x / p.n1, t = threadIdx.x - line * p.n1;
    const int c = line & 1, px = a.nsx == 2 ? (line >> 1) & 1 : 0, jj = line / (2 * a.nsx);
    const int j = blockIdx.x * a.cb + jj;
    const bool on = jj < a.cb && j < a.Q;
    const int rows = a.rows[c];
    C2* own = reinterpret_cast<C2*>(smem_raw) + (jj < a.cb ? line : 0) * a.ls;
    const RegLine<C2> buf{own, p.n2 | 1, 1};
    const C2* partner = c ? own - a.ls : own + a.ls;
    const C2* tw = RegTables<C2>::roots(p);
    const C2* chirp = RegTables<C2>::chirp(p);
    T2* row = a.work + (int64_t)rhs * a.work_rhs + ((int64_t)(pyi * a.ncomp + c) * a.Q + (on ? j : 0)) * a.P;
    with_n1<CLS>(p.n1, [&](auto len) {
        constexpr int R = decltype(len)::value;
        if (!on || t >= p.n2) return;
        C2 v[R];
#pragma unroll
        for (int m1 = 0; m1 < R; ++m1) {
            const int i = p.n2 * m1 + t;
            v[m1] = cast<C2>(i < rows ? row[i] : czero<T2>());
        }
        if (px) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int i = p.n2 * m1 + t;
                v[m1] = cmul(v[m1], cast<C2>(__ldg(&a.modP[BLUE ? min(i, p.n - 1) : i])));
            }
        }
        if constexpr (BLUE) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) v[m1] = cmul(v[m1], __ldg(&chirp[min(p.n2 * m1 + t, p.n - 1)]));
        }
        reg_a_fwd<R>(v, t, tw, buf);
    });
    if constexpr (BLUE) {
        reg_convolve<CLS, false>(p, t, on, buf);
        with_n1<CLS>(p.n1, [&](auto len) {
            constexpr int R = decltype(len)::value;
            const bool mine = on && t < p.n2;
            C2 v[R];
            if (mine) {
                reg_a_inv<R>(v, t, buf);
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) v[m1] = cmul(v[m1], __ldg(&chirp[min(p.n2 * m1 + t, p.n - 1)]));
            }
            reg_mix<R, true>(v, a, own, partner, t, p.n2 | 1, t, p.n2, c, px, py, j, mine);
            if (mine) {
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) {
                    const int k = p.n2 * m1 + t;
                    const C2 w = cmulc(v[m1], __ldg(&chirp[min(k, p.n - 1)]));
                    v[m1] = k < p.n ? w : czero<C2>();
                }
                reg_a_fwd<R>(v, t, tw, buf);
            }
        });
        reg_convolve<CLS, true>(p, t, on, buf);
    } else {
        __syncthreads();
        with_n2<CLS>(p.n2, [&](auto len) {
            constexpr int R = decltype(len)::value;
            const bool mine = on && t < p.n1;
            C2 v[R];
            if (mine) reg_b_fwd<R>(v, t, buf);
            reg_mix<R, false>(v, a, own, partner, t * (p.n2 | 1), 1, t, p.n1, c, px, py, j, mine);
            if (mine) reg_b_inv<R>(v, t, tw, buf);
        });
        __syncthreads();
    }
    with_n1<CLS>(p.n1, [&](auto len) {
        constexpr int R = decltype(len)::value;
        const bool mine = on && t < p.n2;
        C2 v[R];
        if (mine) {
            reg_a_inv<R>(v, t, buf);
            if constexpr (BLUE) {
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) v[m1] = cmulc(v[m1], __ldg(&chirp[min(p.n2 * m1 + t, p.n - 1)]));
            }
        }
        if (a.nsx == 2) {
            if (mine && px) {
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) {
                    const int i = p.n2 * m1 + t;
                    buf.at(m1, t) = cmulc(v[m1], cast<C2>(__ldg(&a.modP[BLUE ? min(i, p.n - 1) : i])));
                }
            }
            __syncthreads();
            if (mine && !px) {
                const RegLine<C2> odd{own + 2 * a.ls, p.n2 | 1, 1};
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) v[m1] = cadd(v[m1], odd.at(m1, t));
            }
        }
        if (mine && !px) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int i = p.n2 * m1 + t;
                const T2 w = cast<T2>(cscale(v[m1], (C)a.scale));
                if (i < rows) row[i] = w;
            }
        }
    });
}

// y-inverse: the lines of the y-forward, from W to y: inverse transform, demodulation, the sum over the y subbands
// through shared memory, cropped.
template <typename T, typename C, int CLS, bool BLUE>
__global__ void __launch_bounds__(RegShape<C, CLS>::threads, (RegShape<C, CLS>::blocks))
    k_reg_y_inv(const GridArgs<T> a, const RegPlan q, typename Cx<T>::T2* __restrict__ y) {
    using T2 = typename Cx<T>::T2;
    using C2 = typename Cx<C>::T2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    griddep_launch_dependents();
    const int c = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const int rows = a.rows[c], cols = a.cols[c];
    const int TI = a.ti, L = a.npy * TI;
    if ((int)blockIdx.x * TI >= rows) return;
    const int t = threadIdx.x / L, line = threadIdx.x - t * L;
    const int pyi = line / TI, i = blockIdx.x * TI + line - pyi * TI;
    const bool odd = (a.py0 + pyi) != 0, on = i < rows;
    const RegLine<C2> buf{reinterpret_cast<C2*>(smem_raw) + line, q.n2 * L, L};
    const C2* tw = RegTables<C2>::roots(q);
    const C2* chirp = RegTables<C2>::chirp(q);
    const T2* src = a.work + (int64_t)rhs * a.work_rhs + (int64_t)(pyi * a.ncomp + c) * a.Q * a.P + i;
    if constexpr (BLUE) {
        with_n1<CLS>(q.n1, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= q.n2) return;
            C2 v[R];
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int j = q.n2 * m1 + t;
                const C2 w = cast<C2>(j < q.n ? src[(int64_t)j * a.P] : czero<T2>());
                v[m1] = cmulc(w, __ldg(&chirp[min(j, q.n - 1)]));
            }
            reg_a_fwd<R>(v, t, tw, buf);
        });
        reg_convolve<CLS, true>(q, t, on, buf);
    } else {
        with_n2<CLS>(q.n2, [&](auto len) {
            constexpr int R = decltype(len)::value;
            if (!on || t >= q.n1) return;
            C2 v[R];
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) v[k2] = cast<C2>(src[(int64_t)(t + q.n1 * k2) * a.P]);
            reg_b_inv<R>(v, t, tw, buf);
        });
        __syncthreads();
    }
    T2* yr = y + (int64_t)rhs * a.n + a.off[c] + i;
    with_n1<CLS>(q.n1, [&](auto len) {
        constexpr int R = decltype(len)::value;
        const bool mine = on && t < q.n2;
        C2 v[R];
        if (mine) {
            reg_a_inv<R>(v, t, buf);
            if constexpr (BLUE) {
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) v[m1] = cmulc(v[m1], __ldg(&chirp[min(q.n2 * m1 + t, q.n - 1)]));
            }
            if (odd) {
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) {
                    const int j = q.n2 * m1 + t;
                    v[m1] = cmulc(v[m1], cast<C2>(__ldg(&a.modQ[BLUE ? min(j, q.n - 1) : j])));
                }
            }
        }
        if (a.npy == 2) {
            if (mine && pyi) {
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) buf.at(m1, t) = v[m1];
            }
            __syncthreads();
            if (mine && !pyi) {
                const RegLine<C2> other{buf.base + TI, q.n2 * L, L};
#pragma unroll
                for (int m1 = 0; m1 < R; ++m1) v[m1] = cadd(v[m1], other.at(m1, t));
            }
        }
        if (!mine || pyi) return;
        if (a.accumulate) {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int j = q.n2 * m1 + t;
                if (j < cols) yr[(int64_t)j * rows] = cadd(yr[(int64_t)j * rows], cast<T2>(v[m1]));
            }
        } else {
#pragma unroll
            for (int m1 = 0; m1 < R; ++m1) {
                const int j = q.n2 * m1 + t;
                if (j < cols) yr[(int64_t)j * rows] = cast<T2>(v[m1]);
            }
        }
    });
}

constexpr size_t kRegSmem = 200 * 1024;

template <typename T, typename C, int CLS, bool BLUE> int set_attrs() {
    static DeviceOnce once;
    return once([]() -> int {
        const int b = (int)kRegSmem;
        RTM_CUDA(cudaFuncSetAttribute(k_reg_y_fwd<T, C, CLS, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
        RTM_CUDA(cudaFuncSetAttribute(k_reg_x_mix<T, C, CLS, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
        RTM_CUDA(cudaFuncSetAttribute(k_reg_y_inv<T, C, CLS, BLUE>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
        return RTM_OK;
    });
}

}  // namespace

template <typename T, typename C, int CLS, bool BLUE>
int launch_reg_pass(int pass, GridArgs<T> a, const RegPlan& r, int nrhs, const void* x, void* y, cudaStream_t s) {
    using T2 = typename Cx<T>::T2;
    using C2 = typename Cx<C>::T2;
    RTM_TRY((set_attrs<T, C, CLS, BLUE>()));
    constexpr int kThreads = RegShape<C, CLS>::threads;
    if (pass == kRegXMix) {
        // as many y frequencies a CTA as its threads take, fewer while the launch would leave SMs without two CTAs
        const int per = 2 * a.nsx * r.n1;
        a.ls = r.n1 * (r.n2 | 1);
        int cb = std::max(1, std::min(a.Q, kThreads / per));
        while (cb > 1 && (int64_t)((a.Q + cb - 1) / cb) * a.npy * nrhs < 2 * kDeviceSms) --cb;
        a.cb = cb;
        const int threads = (cb * per + 31) / 32 * 32;
        const size_t smem = (size_t)cb * 2 * a.nsx * a.ls * sizeof(C2);
        RTM_CUDA(launch_dependent(k_reg_x_mix<T, C, CLS, BLUE>, dim3((a.Q + cb - 1) / cb, a.npy, nrhs), dim3(threads),
                                  smem, s, a, r));
    } else {
        // rows of TI columns: 64 bytes where the threads allow it
        int ti = sizeof(C) == 8 ? 4 : 8;
        while (ti > 1 && a.npy * ti * r.n1 > kThreads) ti /= 2;
        a.ti = ti;
        const int L = a.npy * ti, threads = (L * r.n1 + 31) / 32 * 32;
        const size_t smem = (size_t)L * r.m * sizeof(C2);
        const dim3 grid((std::max(a.rows[0], a.rows[1]) + ti - 1) / ti, 2, nrhs);
        if (pass == kRegYFwd)
            k_reg_y_fwd<T, C, CLS, BLUE><<<grid, threads, smem, s>>>(a, r, static_cast<const T2*>(x));
        else
            RTM_CUDA(launch_dependent(k_reg_y_inv<T, C, CLS, BLUE>, grid, dim3(threads), smem, s, a, r,
                                      static_cast<T2*>(y)));
    }
    count_launch();
    return RTM_OK;
}

// One form a translation unit (build.py), so that they compile side by side.
#if RTM_REG_FORM == 0
template int launch_reg_pass<double, double, 0, false>(int, GridArgs<double>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 1
template int launch_reg_pass<double, double, 1, false>(int, GridArgs<double>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 2
template int launch_reg_pass<double, double, 0, true>(int, GridArgs<double>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 3
template int launch_reg_pass<double, double, 1, true>(int, GridArgs<double>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 4
template int launch_reg_pass<float, float, 0, false>(int, GridArgs<float>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 5
template int launch_reg_pass<float, float, 1, false>(int, GridArgs<float>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 6
template int launch_reg_pass<float, double, 0, true>(int, GridArgs<float>, const RegPlan&, int, const void*, void*, cudaStream_t);
#elif RTM_REG_FORM == 7
template int launch_reg_pass<float, double, 1, true>(int, GridArgs<float>, const RegPlan&, int, const void*, void*, cudaStream_t);
#endif

}  // namespace rtm
