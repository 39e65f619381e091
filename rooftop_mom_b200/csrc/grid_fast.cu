// Power-of-two split products with register-resident line transforms.
//
// The same product as k_grid_y_fwd / k_grid_x_mix / k_grid_y_inv in grid.cu (the reference's
// src/+rooftopMoM/+assembler/+greensMatrix/@SplitFFTApplicator/applyBothDirections_.m:14-85) for
// transform sizes that are powers of two. A line of n = R1 R2 points is transformed by a group of R2
// threads, each holding R1 values in registers (four-step form, decimation in time):
//   thread m2 holds x[R2 m1 + m2], m1 < R1
//   -> R1-point DFT over m1 in registers -> twiddle w_n^(m2 k1)
//   -> one exchange through shared memory
//   -> R1 / R2 DFTs of R2 points over m2 -> X[k1 + R1 k2], thread t holding k1 = t + R2 s (s < R1 / R2)
//      for every k2, at register s R2 + k2.
// The inverse runs the same steps backwards from that layout. The x-mix multiplies the spectra in this
// layout without reordering; every global load and store is coalesced (consecutive threads touch
// consecutive elements). The line buffers are padded (row stride R2 + 1) against bank conflicts.
#include <algorithm>

#include "grid.h"
#include "grid_args.cuh"
#include "bulk.cuh"
#include "pdl.cuh"

namespace rtm {
namespace {

// CTA size: FP32 256 threads, FP64 128. How many CTAs an SM holds (the launch bound, which sets the
// registers a thread may use) is part of the schedule a product runs with (FastSchedule, grid.h).
template <typename T> struct Fast {
    static constexpr int threads = sizeof(T) == 8 ? 128 : 256;
};

template <int N> struct Shape;
template <> struct Shape<32> { static constexpr int R1 = 8, R2 = 4; };
template <> struct Shape<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct Shape<128> { static constexpr int R1 = 16, R2 = 8; };
template <> struct Shape<256> { static constexpr int R1 = 16, R2 = 16; };
template <> struct Shape<512> { static constexpr int R1 = 32, R2 = 16; };
template <> struct Shape<1024> { static constexpr int R1 = 32, R2 = 32; };

// cos(pi k / 16) for k = 0 .. 8 (the real parts of the 32nd roots of unity).
__host__ __device__ constexpr double cos_pi16(int k) {
    return k == 0 ? 1.0 : k == 1 ? 0.980785280403230449126182236134239 : k == 2 ? 0.923879532511286756128183189396788
         : k == 3 ? 0.831469612302545237078788377617906 : k == 4 ? 0.707106781186547524400844362104849
         : k == 5 ? 0.555570233019602224742830813948533 : k == 6 ? 0.382683432365089771728459984030399
         : k == 7 ? 0.195090322016128267848284868477022 : 0.0;
}
// The forward root w_32^k = exp(-i pi k / 16) = (cos, -sin), k < 16, as compile-time constants.
__host__ __device__ constexpr double root32_re(int k) { return k <= 8 ? cos_pi16(k) : -cos_pi16(16 - k); }
__host__ __device__ constexpr double root32_im(int k) { return k <= 8 ? -cos_pi16(8 - k) : -cos_pi16(k - 8); }

// In-register DFT of R points, natural order in and out. R = 32 splits by decimation in frequency
// into two 16-point transforms with the roots w_32^k (constants, no table reads).
template <int R, bool INV, typename T2> __device__ __forceinline__ void dft_reg(T2 (&v)[R]) {
    if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        dft8<INV>(v);
    } else if constexpr (R == 16) {
        dft16<INV>(v);
    } else {
        static_assert(R == 32, "radix");
        using S = decltype(v[0].x);
        T2 a[16], b[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            a[k] = cadd(v[k], v[k + 16]);
            b[k] = csub(v[k], v[k + 16]);
            if (k) b[k] = twc<INV>(b[k], (S)root32_re(k), (S)root32_im(k));
        }
        dft16<INV>(a);
        dft16<INV>(b);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            v[2 * k] = a[k];
            v[2 * k + 1] = b[k];
        }
    }
}

template <typename T2> __device__ __forceinline__ T2 make_vec2(decltype(T2{}.x) x, decltype(T2{}.x) y) {
    T2 r;
    r.x = x;
    r.y = y;
    return r;
}

// Element (r, c) of a line buffer at base[r * RS + c * CS].
template <typename T2> struct LineBuf {
    T2* base;
    int RS, CS;
    __device__ __forceinline__ T2& at(int r, int c) const { return base[r * RS + c * CS]; }
};

// Forward transform of the group's line, steps before the exchange: v[m1] = x[R2 m1 + t] in,
// written to buf(k1, t). ta, tb (inv_first): the twiddles in the two orders of FftTables (n1 = R1, n2 = R2).
template <int N, typename T2>
__device__ __forceinline__ void fwd_first(T2 (&v)[Shape<N>::R1], int t, const T2* __restrict__ ta,
                                          const LineBuf<T2>& buf) {
    constexpr int R1 = Shape<N>::R1;
    dft_reg<R1, false>(v);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
        const T2 w = k1 ? cmul(v[k1], __ldg(&ta[k1 * Shape<N>::R2 + t])) : v[k1];
        buf.at(k1, t) = w;
    }
}

// After the exchange: v[s R2 + k2] = X[(t + R2 s) + R1 k2].
template <int N, typename T2>
__device__ __forceinline__ void fwd_second(T2 (&v)[Shape<N>::R1], int t, const LineBuf<T2>& buf) {
    constexpr int R1 = Shape<N>::R1, R2 = Shape<N>::R2, S = R1 / R2;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        T2 u[R2];
#pragma unroll
        for (int m2 = 0; m2 < R2; ++m2) u[m2] = buf.at(t + R2 * s, m2);
        dft_reg<R2, false>(u);
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) v[s * R2 + k2] = u[k2];
    }
}

// Inverse from the transformed layout, steps before the exchange: written to buf(k1, m2) twiddled.
template <int N, typename T2>
__device__ __forceinline__ void inv_first(T2 (&v)[Shape<N>::R1], int t, const T2* __restrict__ tb,
                                          const LineBuf<T2>& buf) {
    constexpr int R1 = Shape<N>::R1, R2 = Shape<N>::R2, S = R1 / R2;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        T2 u[R2];
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) u[k2] = v[s * R2 + k2];
        dft_reg<R2, true>(u);
        const int k1 = t + R2 * s;
#pragma unroll
        for (int m2 = 0; m2 < R2; ++m2) buf.at(k1, m2) = m2 ? cmulc(u[m2], __ldg(&tb[m2 * R1 + k1])) : u[m2];
    }
}

// After the exchange: v[m1] = N x[R2 m1 + t] (unnormalised).
template <int N, typename T2>
__device__ __forceinline__ void inv_second(T2 (&v)[Shape<N>::R1], int t, const LineBuf<T2>& buf) {
    constexpr int R1 = Shape<N>::R1;
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) v[k1] = buf.at(k1, t);
    dft_reg<R1, true>(v);
}

// Lines in three steps, for N = R1 64 (R1 = 4, 8, 16): the TL threads of a line hold V = N / TL values of two transforms,
// which share the twiddles. With r = 8 t1 + t0, k = k1 + R1 k2 + 8 R1 k3 and a buffer of elements (k1, r), the steps run
// over units of R1, 8 and 8 points, a thread taking unit number thread + TL u:
//   unit r            x[64 a + r]; DFT over a, twiddle wN^(r k1), written to (k1, r);
//   unit 8 k1 + t0    reads (k1, 8 t1 + t0), DFT over t1, twiddle w64^(t0 k2), written back to (k1, 8 k2 + t0);
//   unit k1 + R1 k2   reads (k1, 8 k2 + t0), DFT over t0: X[k], consecutive threads on consecutive frequencies.
// The inverse runs backwards. Every thread writes where it has read, so a step needs one barrier, among its line's threads.
// ES: the stride of the buffer's elements (lines of a CTA may be interleaved); its second transform lies LB ES further.
template <typename T, int N, int ES> struct Lines3 {
    using T2 = typename Cx<T>::T2;
    static constexpr int R1 = N / 64;
    static constexpr int V = R1 <= 8 ? 8 : R1, TL = N / V;  // values and threads a line
    static constexpr int UA = 64 / TL, UB = V / 8;          // units a thread: first step, second and third
    // Element (k1, 8 r1 + r0) at LS k1 + PK r1 + r0: the 8 (FP64) or 16 lanes that share a wavefront meet in different
    // banks in the third step for every R1, and nearly so in the others.
    static constexpr int PK = R1 == 4 ? 9 : 8, LS = R1 == 4 ? (sizeof(T) == 8 ? 74 : 76) : 65;
    static constexpr int LB = R1 * LS;  // buffer elements of one transform
    static constexpr int CS = LB * ES;

    template <int R, bool INV> static __device__ __forceinline__ void dft(T2* v) {
        if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
        else if constexpr (R == 8) dft8<INV>(v);
        else dft16<INV>(v);
    }
    // Value R1 u + e of a thread is element 64 e + tid + TL u of the line; transformed, value 8 u + k3 is frequency
    // tid + TL u + 8 R1 k3.
    static __device__ __forceinline__ int elem(int tid, int u, int e) { return 64 * e + tid + TL * u; }
    static __device__ __forceinline__ int freq(int tid, int u, int k3) { return tid + TL * u + 8 * R1 * k3; }
    static __device__ __forceinline__ T2* first(T2* buf, int tid) { return buf + (PK * (tid / 8) + tid % 8) * ES; }
    static __device__ __forceinline__ T2* third(T2* buf, int tid) {
        return buf + (LS * (tid % R1) + PK * (tid / R1)) * ES;
    }

    template <typename Sync>
    static __device__ __forceinline__ void forward(T2 (&v)[2][V], int tid, T2* buf, const T2* __restrict__ t3, Sync sync) {
        const T2* w64 = t3 + N;  // [k2][t0]
#pragma unroll
        for (int u = 0; u < UA; ++u) {
            T2* at = first(buf, tid) + PK * (TL / 8) * u * ES;
            dft<R1, false>(v[0] + R1 * u);
            dft<R1, false>(v[1] + R1 * u);
#pragma unroll
            for (int k1 = 0; k1 < R1; ++k1) {
                T2* d = at + LS * k1 * ES;
                if (k1) {
                    const T2 w = __ldg(&t3[64 * k1 + tid + TL * u]);
                    d[0] = cmul(v[0][R1 * u + k1], w);
                    d[CS] = cmul(v[1][R1 * u + k1], w);
                } else {
                    d[0] = v[0][R1 * u];
                    d[CS] = v[1][R1 * u];
                }
            }
        }
        sync();
        const int lo = tid % 8, mk = tid / 8;
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const T2* mid = buf + (LS * (mk + TL / 8 * u) + lo) * ES;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[c][8 * u + e] = mid[c * CS + PK * e * ES];
                dft<8, false>(v[c] + 8 * u);
            }
        }
#pragma unroll
        for (int k2 = 0; k2 < 8; ++k2) {
            const T2 w = k2 ? __ldg(&w64[8 * k2 + lo]) : czero<T2>();
#pragma unroll
            for (int u = 0; u < UB; ++u) {
                T2* d = buf + (LS * (mk + TL / 8 * u) + lo + PK * k2) * ES;
                d[0] = k2 ? cmul(v[0][8 * u + k2], w) : v[0][8 * u];
                d[CS] = k2 ? cmul(v[1][8 * u + k2], w) : v[1][8 * u];
            }
        }
        sync();
        const T2* own = third(buf, tid);
#pragma unroll
        for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[c][8 * u + e] = own[c * CS + (PK * (TL / R1) * u + e) * ES];
                dft<8, false>(v[c] + 8 * u);
            }
    }

    template <typename Sync>
    static __device__ __forceinline__ void inverse(T2 (&v)[2][V], int tid, T2* buf, const T2* __restrict__ t3, Sync sync) {
        const T2* w64 = t3 + N;
        T2* own = third(buf, tid);
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            dft<8, true>(v[0] + 8 * u);
            dft<8, true>(v[1] + 8 * u);
            const int k2 = tid / R1 + TL / R1 * u;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                T2* d = own + (PK * (TL / R1) * u + e) * ES;
                if (e) {
                    const T2 w = __ldg(&w64[8 * k2 + e]);
                    d[0] = cmulc(v[0][8 * u + e], w);
                    d[CS] = cmulc(v[1][8 * u + e], w);
                } else {
                    d[0] = v[0][8 * u];
                    d[CS] = v[1][8 * u];
                }
            }
        }
        sync();
        const int lo = tid % 8, mk = tid / 8;
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int k1 = mk + TL / 8 * u;
            T2* mid = buf + (LS * k1 + lo) * ES;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[c][8 * u + e] = mid[c * CS + PK * e * ES];
                dft<8, true>(v[c] + 8 * u);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const T2 w = __ldg(&t3[64 * k1 + 8 * e + lo]);
                mid[PK * e * ES] = cmulc(v[0][8 * u + e], w);
                mid[CS + PK * e * ES] = cmulc(v[1][8 * u + e], w);
            }
        }
        sync();
        const T2* at = first(buf, tid);
#pragma unroll
        for (int u = 0; u < UA; ++u)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
#pragma unroll
                for (int k1 = 0; k1 < R1; ++k1) v[c][R1 * u + k1] = at[c * CS + (PK * (TL / 8) * u + LS * k1) * ES];
                dft<R1, true>(v[c] + R1 * u);
            }
    }
};

// --------------------------------------------------------------------------------------------
// y-forward: TI x-columns of one component; a group per (column, y subband). Thread index
// l + TI (py + 2 t): consecutive threads take consecutive columns, so rows of TI elements are read
// and written at once. W[py][c][k][i] = FFT_y(x_c(i, j) mod_y(j)^py).
template <typename T, int NQ, int MINB>
__global__ void __launch_bounds__(Fast<T>::threads, MINB) k_fast_y_fwd(const GridArgs<T> a, const typename Cx<T>::T2* __restrict__ x) {
    using T2 = typename Cx<T>::T2;
    constexpr int R1 = Shape<NQ>::R1, R2 = Shape<NQ>::R2, TI = Fast<T>::threads / (2 * R2), G = 2 * TI;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T2* sm = reinterpret_cast<T2*>(smem_raw);
    griddep_wait();
    const int c = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const PlateDesc<T> pd = plate_of(a, rhs);
    const int rows = pd.rows[c], cols = pd.cols[c];
    if ((int)blockIdx.x * TI >= rows) return;  // a smaller plate of a batch
    const int l = threadIdx.x % TI, py = (threadIdx.x / TI) % 2, t = threadIdx.x / (2 * TI);
    const int g = l + TI * py;
    const int i = blockIdx.x * TI + l;
    const bool on = i < rows;
    const LineBuf<T2> buf{sm + g, (R2 + 1) * G, G};
    const T2* xr = x + (int64_t)rhs * a.n + pd.off[c];
    T2 v[R1];
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) {
        const int j = R2 * m1 + t;
        T2 e = (on && j < cols) ? xr[i + (int64_t)j * rows] : czero<T2>();
        if (py) e = cmul(e, __ldg(&a.modQ[j]));
        v[m1] = e;
    }
    fwd_first<NQ>(v, t, a.taQ, buf);
    __syncthreads();
    fwd_second<NQ>(v, t, buf);
    if (!on) return;
    T2* dst = a.work + (int64_t)rhs * a.work_rhs + (int64_t)(py * a.ncomp + c) * NQ * a.P + i;
#pragma unroll
    for (int s = 0; s < R1 / R2; ++s)
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) dst[(int64_t)((t + R2 * s) + R1 * k2) * a.P] = v[s * R2 + k2];
}

// The spectra of a generator are even in both frequencies (its embedding is even): of the subband with parity p
// on n frequencies, f = 2 m + p, entry m equals entry n - m - p (mod n). The x-mix reads the lower of the two,
// so of the 12 P Q stored values a product touches 3 P Q, which stay in L2 between products (FP32 1024 x 1024:
// 25 MB instead of 100).
__device__ __forceinline__ int even_freq(int m, int p, int n) { return min(m, n - m - p); }

// The R2 <= 32 threads of an x line are lanes of one warp, so its exchanges need no CTA barrier. FP32 takes that, and
// shuffles for the partner's values (products of 256 x 256: 12.1 us, 12.6 with barriers, four vectors 23.2 against
// 24.7; 64 x 64 7.4 against 7.9; 128 x 128 alone 13.2 against 12.9). FP64, whose CTAs hold four warps with up to 255
// registers, keeps the barriers: its warps then share the twiddle and spectra lines (512 x 512 in two steps: 47 us, 51
// without them).
template <typename T> __device__ __forceinline__ void line_sync() {
    if constexpr (sizeof(T) == 8) __syncthreads();
    else __syncwarp();
}

// x-mix, direct form (one CTA per TEAMS y frequencies; inputs loaded straight into registers, the spectra
// read in the mix): teams of four groups (component c, x subband px) per y frequency j of subband py. Thread
// index t + R2 (team * 4 + 2 px + c). Forward transform along x of W mod_x^px, the 2x2 block mix
// with the subband spectra (the two components of a group pair meet through shared memory), inverse
// transform, demodulation, the sum over px, scaled by 1 / (PQ), in place in W.
template <typename T, int NP, int MINB>
__global__ void __launch_bounds__(Fast<T>::threads, MINB) k_fast_x_mix_direct(const GridArgs<T> a) {
    using T2 = typename Cx<T>::T2;
    constexpr int R1 = Shape<NP>::R1, R2 = Shape<NP>::R2, S = R1 / R2;
    constexpr int TEAMS = Fast<T>::threads / (4 * R2), LB = R1 * (R2 + 1);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T2* sm = reinterpret_cast<T2*>(smem_raw);
    griddep_wait();
    const int py = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const PlateDesc<T> pd = plate_of(a, rhs);
    const int t = threadIdx.x % R2, gid = threadIdx.x / R2;
    const int team = gid / 4, c = gid % 2, px = (gid / 2) % 2;
    const int j = blockIdx.x * TEAMS + team;
    const bool on = j < a.Q;
    const int Q = a.Q;
    const int64_t QP = (int64_t)Q * NP;
    const LineBuf<T2> buf{sm + gid * LB, R2 + 1, 1};
    const int rows = pd.rows[c];
    T2* row = a.work + (int64_t)rhs * a.work_rhs + (int64_t)(py * a.ncomp + c) * QP + (int64_t)(on ? j : 0) * NP;
    T2 v[R1];
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) {
        const int i = R2 * m1 + t;
        T2 e = (on && i < rows) ? row[i] : czero<T2>();
        if (px) e = cmul(e, __ldg(&a.modP[i]));
        v[m1] = e;
    }
    fwd_first<NP>(v, t, a.taP, buf);
    line_sync<T>();
    fwd_second<NP>(v, t, buf);
    // The partner's values come by warp shuffles where both lines share a warp (FP32; an FP64 value takes four: the
    // 256 x 256 product 17.2 us with them, 16.1 without), else through the buffers.
    constexpr bool kShuffle = R2 <= 16 && sizeof(T) == 4;
    T2* own = sm + gid * LB;
    const T2* partner = sm + (gid ^ 1) * LB;
    if constexpr (!kShuffle) {
        line_sync<T>();  // the line's buffer is read; it now carries the spectra values to the partner
#pragma unroll
        for (int r = 0; r < R1; ++r) own[r * R2 + t] = v[r];
        __syncthreads();
    }
    if (kShuffle || on) {
        const int sub = px + 2 * py;
        const int jc = on ? j : 0;
        const T2* spec = pd.spec + (int64_t)(sub * 3) * QP + (int64_t)even_freq(jc, py, Q) * NP;
        const T2* ux = px ? a.ux1 : a.ux0;
        const T2 vv = __ldg(&(py ? a.vy1 : a.vy0)[jc]);
        const T cv = (vv.x * vv.x + vv.y * vv.y) * pd.inv_b2;
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) {
                const int k = (t + R2 * s) + R1 * k2;
                const int ke = even_freq(k, px, NP);
                const T2 E = __ldg(&spec[ke]);
                const T2 M = __ldg(&spec[(1 + c) * QP + ke]);
                const T2 uu = __ldg(&ux[k]);
                const T cu = (uu.x * uu.x + uu.y * uu.y) * pd.inv_a2;
                // qc = -u conj(v) / (ab): XY = qc E, YX = conj(qc) E
                T2 qc = cmulc(uu, vv);
                qc.x = -qc.x * pd.inv_ab;
                qc.y = -qc.y * pd.inv_ab;
                const T2 coupling = c ? cconj(qc) : qc;
                const T cself = c ? cv : cu;
                const T2 me = v[s * R2 + k2];
                T2 other;
                if constexpr (kShuffle) {
                    other.x = __shfl_xor_sync(0xffffffffu, me.x, R2);
                    other.y = __shfl_xor_sync(0xffffffffu, me.y, R2);
                } else {
                    other = partner[(s * R2 + k2) * R2 + t];
                }
                // M me - cself E me + coupling E other = M me + E (coupling other - cself me)
                const T2 cp = cmul(coupling, other);
                const T2 d = make_vec2<T2>(cp.x - cself * me.x, cp.y - cself * me.y);
                v[s * R2 + k2] = cadd(cmul(M, me), cmul(E, d));
            }
    }
    if constexpr (!kShuffle) __syncthreads();  // the partner values are read
    inv_first<NP>(v, t, a.tbP, buf);
    line_sync<T>();
    inv_second<NP>(v, t, buf);
    if (px) {
        // in the thread's own column of the buffer, which no other one has read
#pragma unroll
        for (int m1 = 0; m1 < R1; ++m1) buf.at(m1, t) = cmulc(v[m1], __ldg(&a.modP[R2 * m1 + t]));
    }
    __syncthreads();
    if (px || !on) return;
    const LineBuf<T2> odd{sm + (gid + 2) * LB, R2 + 1, 1};
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) {
        const int i = R2 * m1 + t;
        if (i < rows) row[i] = cscale(cadd(v[m1], odd.at(m1, t)), a.scale);
    }
}

// The lengths that run in three steps by default when both lengths of a split product are powers of two, a thread
// holding both components of an x line (they share the twiddles, the phases and E, and meet in registers) or both subbands
// of a column; the small radices need half the registers. The L1 pipe bounds both forms of the x-mix (FP64 512 x 512 with
// four vectors: 49 % busy in two steps at 8 warps an SM, 70 % in three). Product, two steps -> three, one vector and four:
// FP64 256 x 256 15.9 -> 13.5 us and 42.9 -> 36.8; 512 x 512 46.6 -> 37.2 and 185 -> 139; FP32 512 x 512 29.6 -> 25.2 and
// 94 -> 81; 1024 x 1024 104 -> 89 and 382 -> 345. FP32 256 x 256 stays on two steps (x-mix in three: 12.5 against 12.4 us,
// 24.9 against 23.4): its lines exchange within their warps there; shorter lines leave too few threads for three steps.
constexpr bool three_step(int n, bool fp64) { return fp64 ? n == 256 || n == 512 : n == 512 || n == 1024; }

// SUB: the subbands along x (2: a split product, 1: an embedding or a circulant).
template <typename T, int NP, int SUB> struct XMix3 {
    using L = Lines3<T, NP, 1>;
    static constexpr int threads = 128, teams = threads / (SUB * L::TL);  // y frequencies a CTA
    static constexpr int smem_elems = teams * SUB * 2 * L::LB;
};

template <typename T, int NP, int SUB, int MINB>
__global__ void __launch_bounds__((XMix3<T, NP, SUB>::threads), MINB) k_fast_x_mix_3(const GridArgs<T> a) {
    using T2 = typename Cx<T>::T2;
    using L = Lines3<T, NP, 1>;
    constexpr int R1 = L::R1, TL = L::TL, LB = L::LB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    const int py = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const PlateDesc<T> pd = plate_of(a, rhs);
    const int tid = threadIdx.x % TL, line = threadIdx.x / TL, px = SUB == 2 ? line % 2 : 0;
    const int j = blockIdx.x * XMix3<T, NP, SUB>::teams + line / SUB;
    const bool on = j < a.Q;
    const int64_t QP = (int64_t)a.Q * NP;
    T2* buf = reinterpret_cast<T2*>(smem_raw) + line * 2 * LB;
    T2* row = a.work + (int64_t)rhs * a.work_rhs + (int64_t)(py * 2) * QP + (int64_t)(on ? j : 0) * NP;
    auto sync = [line]() {
        if constexpr (TL == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;\n" ::"r"(1 + line), "n"(TL) : "memory");
    };
    T2 v[2][L::V];
#pragma unroll
    for (int u = 0; u < L::UA; ++u)
#pragma unroll
        for (int e = 0; e < R1; ++e) {
            const int i = L::elem(tid, u, e);
#pragma unroll
            for (int c = 0; c < 2; ++c) v[c][R1 * u + e] = on && i < pd.rows[c] ? row[c * QP + i] : czero<T2>();
            if (px) {
                const T2 m = __ldg(&a.modP[i]);
                v[0][R1 * u + e] = cmul(v[0][R1 * u + e], m);
                v[1][R1 * u + e] = cmul(v[1][R1 * u + e], m);
            }
        }
    L::forward(v, tid, buf, a.t3P, sync);
    if (SUB == 1 && a.mode == kBlock4) {
        // blocks XX, XY, YX, YY
        const T2* spec = pd.spec + (int64_t)(on ? j : 0) * NP;
#pragma unroll
        for (int u = 0; u < L::UB; ++u)
#pragma unroll
            for (int k3 = 0; k3 < 8; ++k3) {
                const int k = L::freq(tid, u, k3);
                const T2 mx = v[0][8 * u + k3], my = v[1][8 * u + k3];
                v[0][8 * u + k3] = cadd(cmul(__ldg(&spec[k]), mx), cmul(__ldg(&spec[QP + k]), my));
                v[1][8 * u + k3] = cadd(cmul(__ldg(&spec[3 * QP + k]), my), cmul(__ldg(&spec[2 * QP + k]), mx));
            }
    } else {
        const int jc = on ? j : 0;
        const T2* spec = pd.spec + (int64_t)((px + SUB * py) * 3) * QP + (int64_t)even_freq(jc, py, a.Q) * NP;
        const T2* ux = px ? a.ux1 : a.ux0;
        const T2 vv = __ldg(&(py ? a.vy1 : a.vy0)[jc]);
        const T cv = (vv.x * vv.x + vv.y * vv.y) * pd.inv_b2;
#pragma unroll
        for (int u = 0; u < L::UB; ++u)
#pragma unroll
            for (int k3 = 0; k3 < 8; ++k3) {
                const int k = L::freq(tid, u, k3), ke = even_freq(k, px, NP);
                const T2 E = __ldg(&spec[ke]);
                const T2 uu = __ldg(&ux[k]);
                const T cu = (uu.x * uu.x + uu.y * uu.y) * pd.inv_a2;
                // qc = -u conj(v) / (ab): XY = qc E, YX = conj(qc) E
                T2 qc = cmulc(uu, vv);
                qc.x = -qc.x * pd.inv_ab;
                qc.y = -qc.y * pd.inv_ab;
                const T2 me[2] = {v[0][8 * u + k3], v[1][8 * u + k3]};
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const T2 M = __ldg(&spec[(1 + c) * QP + ke]);
                    const T cself = c ? cv : cu;
                    // M me - cself E me + coupling E other = M me + E (coupling other - cself me)
                    const T2 cp = cmul(c ? cconj(qc) : qc, me[1 - c]);
                    const T2 d = make_vec2<T2>(cp.x - cself * me[c].x, cp.y - cself * me[c].y);
                    v[c][8 * u + k3] = cadd(cmul(M, me[c]), cmul(E, d));
                }
            }
    }
    L::inverse(v, tid, buf, a.t3P, sync);
    if constexpr (SUB == 1) {
        if (!on) return;
#pragma unroll
        for (int u = 0; u < L::UA; ++u)
#pragma unroll
            for (int e = 0; e < R1; ++e) {
                const int i = L::elem(tid, u, e);
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    if (i < pd.rows[c]) row[c * QP + i] = cscale(v[c][R1 * u + e], a.scale);
            }
        return;
    }
    // the even subband's threads finish component 0 of the sum, the odd one's component 1
    T2* mine = L::first(buf, tid) + (1 - px) * LB;
#pragma unroll
    for (int u = 0; u < L::UA; ++u)
#pragma unroll
        for (int e = 0; e < R1; ++e) {
            const int o = R1 * u + e;
            if (px) {
                const T2 m = __ldg(&a.modP[L::elem(tid, u, e)]);
                v[0][o] = cmulc(v[0][o], m);
                v[1][o] = cmulc(v[1][o], m);
            }
            mine[L::PK * (TL / 8) * u + L::LS * e] = px ? v[0][o] : v[1][o];
        }
    __syncthreads();
    if (!on) return;
    const T2* theirs = L::first(reinterpret_cast<T2*>(smem_raw) + (line ^ 1) * 2 * LB, tid) + px * LB;
#pragma unroll
    for (int u = 0; u < L::UA; ++u)
#pragma unroll
        for (int e = 0; e < R1; ++e) {
            const int i = L::elem(tid, u, e), o = R1 * u + e;
            const T2 got = theirs[L::PK * (TL / 8) * u + L::LS * e];
            const T2 even = px ? got : v[0][o], odd = px ? v[1][o] : got;
            if (i < pd.rows[px]) row[px * QP + i] = cscale(cadd(even, odd), a.scale);
        }
}

// x-mix, pipelined form: persistent CTAs. A CTA takes the iterations it = blockIdx.x, blockIdx.x + gridDim.x, ...; an
// iteration is TEAMS consecutive y frequencies j of one (right-hand side, y subband py). Its inputs are
// copied into shared memory one iteration ahead by bulk asynchronous copies (one thread issues them): the
// W rows of both components (contiguous for consecutive j) as soon as the current ones are in registers,
// and the subband spectra rows (E, MXX, MYY of both x subbands) as soon as the current mix has read them,
// so the global-memory latency of both overlaps the transforms. Per y frequency, a team of four groups
// (component c, x subband px), thread index t + R2 (team * 4 + 2 px + c): forward transform along x of
// W mod_x^px, the 2x2 block mix with the subband spectra (the two components of a group pair meet through
// shared memory), inverse transform, demodulation, the sum over px, scaled by 1 / (PQ), in place in W.
// A bulk-copy wait that runs out records RTM_ERR_TIMEOUT in the fault word and ends the CTA.
template <typename T, int NP> struct MixShape {
    static constexpr int R1 = Shape<NP>::R1, R2 = Shape<NP>::R2;
    static constexpr int TEAMS = Fast<T>::threads / (4 * R2), LB = R1 * (R2 + 1);
    using T2 = typename Cx<T>::T2;
    // line buffers [4 TEAMS][LB], W rows [2 c][TEAMS][NP], spectra rows [2 px][3 kind][TEAMS][NS], the lower half
    // of each row (even_freq), padded to 16 bytes
    static constexpr int NS = NP / 2 + 2;
    static constexpr size_t lines = (size_t)4 * TEAMS * LB * sizeof(T2);
    static constexpr size_t wrows = (size_t)2 * TEAMS * NP * sizeof(T2);
    static constexpr size_t srows = (size_t)6 * TEAMS * NS * sizeof(T2);
    static constexpr size_t smem = lines + wrows + srows;
    static constexpr int blocks = 2 * smem <= 220 * 1024 ? 2 : 1;  // CTAs per SM the registers are sized for
};

template <typename T, int NP>
__global__ void __launch_bounds__(Fast<T>::threads, (MixShape<T, NP>::blocks)) k_fast_x_mix_pipe(const GridArgs<T> a, int iters) {
    using M = MixShape<T, NP>;
    using T2 = typename Cx<T>::T2;
    constexpr int R1 = M::R1, R2 = M::R2, S = R1 / R2, TEAMS = M::TEAMS, LB = M::LB, NS = M::NS;
    constexpr unsigned BLOCK = TEAMS * NP * sizeof(T2);  // TEAMS consecutive rows of one grid
    constexpr unsigned HALF = NS * sizeof(T2);           // the lower half of a spectra row
    static_assert(BLOCK % 16 == 0 && HALF % 16 == 0 && M::lines % 16 == 0 && M::wrows % 16 == 0,
                  "bulk copies need 16-byte units");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T2* sm = reinterpret_cast<T2*>(smem_raw);
    T2* wst = reinterpret_cast<T2*>(smem_raw + M::lines);
    T2* sst = reinterpret_cast<T2*>(smem_raw + M::lines + M::wrows);
    __shared__ __align__(8) uint64_t bar[2];  // 0: W rows, 1: spectra rows
    griddep_wait();
    const int Q = a.Q, per_py = Q / TEAMS, per_rhs = 2 * per_py;
    const int64_t QP = (int64_t)Q * NP;
    const int tid = threadIdx.x;
    const int t = tid % R2, gid = tid / R2;
    const int team = gid / 4, c = gid % 2, px = (gid / 2) % 2;
    auto live = [&](int it) {
        while (it < iters && skipped(a, it / per_rhs)) it += gridDim.x;
        return it;
    };
    // copies issued (thread 0) and barrier phases completed (every thread), per barrier
    unsigned issued[2] = {0, 0}, done[2] = {0, 0};
    auto issue = [&](int it, bool w, bool spectra) {
        const int rhs = it / per_rhs, r = it % per_rhs, py = r / per_py, j0 = (r % per_py) * TEAMS;
        if (w) {
            ++issued[0];
            mbar_expect_tx(&bar[0], 2 * BLOCK);
            for (int cc = 0; cc < 2; ++cc)
                bulk_load(wst + cc * TEAMS * NP,
                          a.work + rhs * a.work_rhs + (int64_t)(py * a.ncomp + cc) * QP + (int64_t)j0 * NP, BLOCK,
                          &bar[0]);
        }
        if (spectra) {
            ++issued[1];
            mbar_expect_tx(&bar[1], 6 * TEAMS * HALF);
            const T2* sp = a.plates ? a.plates[rhs].spec : a.spec;
            for (int q = 0; q < 2; ++q)
                for (int kind = 0; kind < 3; ++kind)
                    for (int e = 0; e < TEAMS; ++e)
                        bulk_load(sst + ((q * 3 + kind) * TEAMS + e) * NS,
                                  sp + (int64_t)((q + 2 * py) * 3 + kind) * QP +
                                      (int64_t)even_freq(j0 + e, py, Q) * NP,
                                  HALF, &bar[1]);
        }
    };
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    int it = live(blockIdx.x);
    if (tid == 0 && it < iters) issue(it, true, true);
    const LineBuf<T2> buf{sm + gid * LB, R2 + 1, 1};
    T2* own = sm + gid * LB;
    const T2* partner = sm + (gid ^ 1) * LB;
    const LineBuf<T2> odd{sm + (gid + 2) * LB, R2 + 1, 1};
    const T2* ux = px ? a.ux1 : a.ux0;
    while (it < iters) {
        const int nxt = live(it + gridDim.x);
        const int rhs = it / per_rhs, r = it % per_rhs, py = r / per_py, j = (r % per_py) * TEAMS + team;
        const PlateDesc<T> pd = plate_of(a, rhs);
        const int rows = pd.rows[c];
        if (__syncthreads_or(!mbar_wait(&bar[0], done[0] & 1, a.fault))) break;
        ++done[0];
        T2 v[R1];
        const T2* wrow = wst + (c * TEAMS + team) * NP;
#pragma unroll
        for (int m1 = 0; m1 < R1; ++m1) {
            const int i = R2 * m1 + t;
            T2 e = i < rows ? wrow[i] : czero<T2>();
            if (px) e = cmul(e, __ldg(&a.modP[i]));
            v[m1] = e;
        }
        __syncthreads();  // the W rows are in registers: the next iteration's may come in
        if (tid == 0 && nxt < iters) issue(nxt, true, false);
        fwd_first<NP>(v, t, a.taP, buf);
        __syncwarp();
        fwd_second<NP>(v, t, buf);
        __syncwarp();  // the line's buffer is read; it now carries the spectra values to the partner
#pragma unroll
        for (int q = 0; q < R1; ++q) own[q * R2 + t] = v[q];
        if (__syncthreads_or(!mbar_wait(&bar[1], done[1] & 1, a.fault))) break;
        ++done[1];
        {
            const T2* Es = sst + (px * 3 * TEAMS + team) * NS;
            const T2* Ms = sst + ((px * 3 + 1 + c) * TEAMS + team) * NS;
            const T2 vv = __ldg(&(py ? a.vy1 : a.vy0)[j]);
            const T cv = (vv.x * vv.x + vv.y * vv.y) * pd.inv_b2;
#pragma unroll
            for (int s = 0; s < S; ++s)
#pragma unroll
                for (int k2 = 0; k2 < R2; ++k2) {
                    const int k = (t + R2 * s) + R1 * k2;
                    const int ke = even_freq(k, px, NP);
                    const T2 E = Es[ke];
                    const T2 Mk = Ms[ke];
                    const T2 uu = __ldg(&ux[k]);
                    const T cu = (uu.x * uu.x + uu.y * uu.y) * pd.inv_a2;
                    // qc = -u conj(v) / (ab): XY = qc E, YX = conj(qc) E
                    T2 qc = cmulc(uu, vv);
                    qc.x = -qc.x * pd.inv_ab;
                    qc.y = -qc.y * pd.inv_ab;
                    const T2 coupling = c ? cconj(qc) : qc;
                    const T cself = c ? cv : cu;
                    const T2 me = v[s * R2 + k2], other = partner[(s * R2 + k2) * R2 + t];
                    // Mk me - cself E me + coupling E other = Mk me + E (coupling other - cself me)
                    const T2 cp = cmul(coupling, other);
                    const T2 d = make_vec2<T2>(cp.x - cself * me.x, cp.y - cself * me.y);
                    v[s * R2 + k2] = cadd(cmul(Mk, me), cmul(E, d));
                }
        }
        __syncthreads();  // the spectra and the partner values are read
        if (tid == 0 && nxt < iters) issue(nxt, false, true);
        inv_first<NP>(v, t, a.tbP, buf);
        __syncwarp();
        inv_second<NP>(v, t, buf);
        if (px) {
#pragma unroll
            for (int m1 = 0; m1 < R1; ++m1) buf.at(m1, t) = cmulc(v[m1], __ldg(&a.modP[R2 * m1 + t]));
        }
        __syncthreads();
        if (!px) {
            T2* row = a.work + rhs * a.work_rhs + (int64_t)(py * a.ncomp + c) * QP + (int64_t)j * NP;
#pragma unroll
            for (int m1 = 0; m1 < R1; ++m1) {
                const int i = R2 * m1 + t;
                if (i < rows) row[i] = cscale(cadd(v[m1], odd.at(m1, t)), a.scale);
            }
        }
        it = nxt;
    }
    // A wait ran out: let the copies still in flight into this CTA's shared memory land (each wait
    // bounded) before the CTA ends.
    if (tid == 0)
        for (int q = 0; q < 2; ++q)
            for (; done[q] < issued[q]; ++done[q]) mbar_wait(&bar[q], done[q] & 1, nullptr);
}

// Zeros behind a plate's rooftops in its vector of a batch, by the CTAs of a y-inverse (a launch of its own took 2.1 us,
// of the 41 of an iteration on sixteen plates of 33 to 64 faces a side).
template <typename T>
__device__ __forceinline__ void zero_tail(const GridArgs<T>& a, const PlateDesc<T>& pd, typename Cx<T>::T2* yr) {
    if (!a.plates) return;
    const int64_t from = pd.off[1] + (int64_t)pd.rows[1] * pd.cols[1];
    for (int64_t i = from + (int64_t)(blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; i < a.n;
         i += (int64_t)gridDim.y * gridDim.x * blockDim.x)
        yr[i] = czero<typename Cx<T>::T2>();
}

// y-inverse: TI columns of one component, a group per (column, y subband); inverse transform along y,
// demodulation, the sum over py through shared memory, cropped into y.
template <typename T, int NQ, int MINB>
__global__ void __launch_bounds__(Fast<T>::threads, MINB) k_fast_y_inv(const GridArgs<T> a, typename Cx<T>::T2* __restrict__ y) {
    using T2 = typename Cx<T>::T2;
    constexpr int R1 = Shape<NQ>::R1, R2 = Shape<NQ>::R2, TI = Fast<T>::threads / (2 * R2), G = 2 * TI;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T2* sm = reinterpret_cast<T2*>(smem_raw);
    griddep_wait();
    const int c = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const PlateDesc<T> pd = plate_of(a, rhs);
    zero_tail(a, pd, y + (int64_t)rhs * a.n);
    const int rows = pd.rows[c], cols = pd.cols[c];
    if ((int)blockIdx.x * TI >= rows) return;  // a smaller plate of a batch
    const int l = threadIdx.x % TI, py = (threadIdx.x / TI) % 2, t = threadIdx.x / (2 * TI);
    const int g = l + TI * py;
    const int i = blockIdx.x * TI + l;
    const bool on = i < rows;
    const LineBuf<T2> buf{sm + g, (R2 + 1) * G, G};
    const T2* src = a.work + (int64_t)rhs * a.work_rhs + (int64_t)(py * a.ncomp + c) * NQ * a.P + (on ? i : 0);
    T2 v[R1];
#pragma unroll
    for (int s = 0; s < R1 / R2; ++s)
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2)
            v[s * R2 + k2] = on ? src[(int64_t)((t + R2 * s) + R1 * k2) * a.P] : czero<T2>();
    inv_first<NQ>(v, t, a.tbQ, buf);
    __syncthreads();
    inv_second<NQ>(v, t, buf);
    __syncthreads();
    if (py) {
#pragma unroll
        for (int m1 = 0; m1 < R1; ++m1) buf.at(m1, t) = cmulc(v[m1], __ldg(&a.modQ[R2 * m1 + t]));
    }
    __syncthreads();
    if (py || !on) return;
    const LineBuf<T2> odd{sm + g + TI, (R2 + 1) * G, G};
    T2* yr = y + (int64_t)rhs * a.n + pd.off[c];
#pragma unroll
    for (int m1 = 0; m1 < R1; ++m1) {
        const int j = R2 * m1 + t;
        if (j < cols) yr[i + (int64_t)j * rows] = cadd(v[m1], odd.at(m1, t));
    }
}

// The y passes in three steps: a thread holds both subbands of a column, which share its loads and twiddles and, in the
// inverse, sum in registers; without subbands (SUB = 1) two columns TI apart. TI columns a CTA, interleaved in the buffer:
// thread l + TI tid.
template <typename T, int NQ> struct Y3 {
    static constexpr int TI = 64 / sizeof(typename Cx<T>::T2);
    using L = Lines3<T, NQ, TI>;
    static constexpr int threads = TI * L::TL;
    static constexpr size_t smem = (size_t)2 * L::CS * sizeof(typename Cx<T>::T2);
};

struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

template <typename T, int NQ, int SUB, int MINB>
__global__ void __launch_bounds__((Y3<T, NQ>::threads), MINB)
    k_fast_y_fwd_3(const GridArgs<T> a, const typename Cx<T>::T2* __restrict__ x) {
    using T2 = typename Cx<T>::T2;
    using L = typename Y3<T, NQ>::L;
    constexpr int R1 = L::R1, TI = Y3<T, NQ>::TI;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    const int c = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const PlateDesc<T> pd = plate_of(a, rhs);
    const int rows = pd.rows[c], cols = pd.cols[c];
    if ((int)blockIdx.x * TI * (3 - SUB) >= rows) return;  // a smaller plate of a batch
    const int l = threadIdx.x % TI, tid = threadIdx.x / TI;
    const int i = blockIdx.x * TI * (3 - SUB) + l;
    // the second transform: the odd subband of the column, or the column TI further
    const bool on = i < rows, on2 = SUB == 1 && i + TI < rows;
    const T2* xr = x + (int64_t)rhs * a.n + pd.off[c] + i;
    T2 v[2][L::V];
#pragma unroll
    for (int u = 0; u < L::UA; ++u)
#pragma unroll
        for (int e = 0; e < R1; ++e) {
            const int j = L::elem(tid, u, e);
            v[0][R1 * u + e] = (on && j < cols) ? xr[(int64_t)j * rows] : czero<T2>();
            if (SUB == 1) v[1][R1 * u + e] = (on2 && j < cols) ? xr[(int64_t)j * rows + TI] : czero<T2>();
        }
    if (SUB == 2) {
#pragma unroll
    for (int u = 0; u < L::UA; ++u)
#pragma unroll
        for (int e = 0; e < R1; ++e) v[1][R1 * u + e] = cmul(v[0][R1 * u + e], __ldg(&a.modQ[L::elem(tid, u, e)]));
    }
    L::forward(v, tid, reinterpret_cast<T2*>(smem_raw) + l, a.t3Q, CtaSync{});
    if (!on) return;
    const int64_t QP = (int64_t)NQ * a.P;
    const int64_t second = SUB == 2 ? 2 * QP : TI;
    T2* dst = a.work + (int64_t)rhs * a.work_rhs + c * QP + i;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (SUB == 1 && h && !on2) return;
#pragma unroll
        for (int u = 0; u < L::UB; ++u)
#pragma unroll
            for (int k3 = 0; k3 < 8; ++k3) dst[h * second + (int64_t)L::freq(tid, u, k3) * a.P] = v[h][8 * u + k3];
    }
}

template <typename T, int NQ, int SUB, int MINB>
__global__ void __launch_bounds__((Y3<T, NQ>::threads), MINB)
    k_fast_y_inv_3(const GridArgs<T> a, typename Cx<T>::T2* __restrict__ y) {
    using T2 = typename Cx<T>::T2;
    using L = typename Y3<T, NQ>::L;
    constexpr int R1 = L::R1, TI = Y3<T, NQ>::TI;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep_wait();
    const int c = blockIdx.y, rhs = blockIdx.z;
    if (skipped(a, rhs)) return;
    const PlateDesc<T> pd = plate_of(a, rhs);
    zero_tail(a, pd, y + (int64_t)rhs * a.n);
    const int rows = pd.rows[c], cols = pd.cols[c];
    if ((int)blockIdx.x * TI * (3 - SUB) >= rows) return;  // a smaller plate of a batch
    const int l = threadIdx.x % TI, tid = threadIdx.x / TI;
    const int i = blockIdx.x * TI * (3 - SUB) + l;
    // the second transform: the odd subband of the column, or the column TI further
    const bool on = i < rows, on2 = SUB == 1 && i + TI < rows;
    const int64_t QP = (int64_t)NQ * a.P;
    const int64_t second = SUB == 2 ? 2 * QP : TI;
    const T2* src = a.work + (int64_t)rhs * a.work_rhs + c * QP + (on ? i : 0);
    T2 v[2][L::V];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < L::UB; ++u)
#pragma unroll
            for (int k3 = 0; k3 < 8; ++k3)
                v[h][8 * u + k3] =
                    (SUB == 1 && h ? on2 : on) ? src[h * second + (int64_t)L::freq(tid, u, k3) * a.P] : czero<T2>();
    L::inverse(v, tid, reinterpret_cast<T2*>(smem_raw) + l, a.t3Q, CtaSync{});
    if (!on) return;
    T2* yr = y + (int64_t)rhs * a.n + pd.off[c] + i;
#pragma unroll
    for (int u = 0; u < L::UA; ++u)
#pragma unroll
        for (int e = 0; e < R1; ++e) {
            const int j = L::elem(tid, u, e), o = R1 * u + e;
            if (SUB == 2) {
                const T2 odd = cmulc(v[1][o], __ldg(&a.modQ[j]));
                if (j < cols) yr[(int64_t)j * rows] = cadd(v[0][o], odd);
            } else {
                if (j < cols) yr[(int64_t)j * rows] = v[0][o];
                if (on2 && j < cols) yr[(int64_t)j * rows + TI] = v[1][o];
            }
        }
}

template <typename T, int NQ> size_t y_smem() {
    constexpr int R1 = Shape<NQ>::R1, R2 = Shape<NQ>::R2, TI = Fast<T>::threads / (2 * R2);
    return (size_t)2 * TI * R1 * (R2 + 1) * sizeof(typename Cx<T>::T2);
}
template <typename T, int NQ, int MINB> int launch_y_b(const GridArgs<T>& a, int nrhs, const void* x, void* y,
                                                       bool fwd, cudaStream_t s) {
    using T2 = typename Cx<T>::T2;
    constexpr int TI = Fast<T>::threads / (2 * Shape<NQ>::R2);
    const size_t smem = y_smem<T, NQ>();
    static DeviceOnce once;
    RTM_TRY(once([smem]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_fast_y_fwd<T, NQ, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        RTM_CUDA(cudaFuncSetAttribute(k_fast_y_inv<T, NQ, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        return RTM_OK;
    }));
    const int rows_max = a.rows[0] > a.rows[1] ? a.rows[0] : a.rows[1];
    const dim3 grid((rows_max + TI - 1) / TI, 2, nrhs);
    if (fwd)
        RTM_CUDA(launch_dependent(k_fast_y_fwd<T, NQ, MINB>, grid, dim3(Fast<T>::threads), smem, s, a,
                                  static_cast<const T2*>(x)));
    else
        RTM_CUDA(launch_dependent(k_fast_y_inv<T, NQ, MINB>, grid, dim3(Fast<T>::threads), smem, s, a,
                                  static_cast<T2*>(y)));
    count_launch();
    return RTM_OK;
}

template <typename T, int NQ, int SUB> int launch_y_3(const GridArgs<T>& a, int nrhs, const void* x, void* y, bool fwd,
                                             cudaStream_t s) {
    using T2 = typename Cx<T>::T2;
    using S = Y3<T, NQ>;
    // CTAs an SM; with TI columns of 64 bytes (FP64 512 x 512 with four vectors: 139 us; 2 columns and 3 CTAs 150, one
    // CTA 155; FP32 1024 x 1024: 345, 4 columns and 2 CTAs 352).
    constexpr int MINB = sizeof(T) == 8 ? (NQ == 256 ? 3 : 2) : (NQ == 1024 ? 1 : 2);
    static DeviceOnce once;
    RTM_TRY(once([]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_fast_y_fwd_3<T, NQ, SUB, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem));
        RTM_CUDA(cudaFuncSetAttribute(k_fast_y_inv_3<T, NQ, SUB, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem));
        return RTM_OK;
    }));
    const int rows_max = a.rows[0] > a.rows[1] ? a.rows[0] : a.rows[1];
    constexpr int columns = S::TI * (3 - SUB);
    const dim3 grid((rows_max + columns - 1) / columns, 2, nrhs);
    if (fwd)
        RTM_CUDA(launch_dependent(k_fast_y_fwd_3<T, NQ, SUB, MINB>, grid, dim3(S::threads), S::smem, s, a,
                                  static_cast<const T2*>(x)));
    else
        RTM_CUDA(launch_dependent(k_fast_y_inv_3<T, NQ, SUB, MINB>, grid, dim3(S::threads), S::smem, s, a, static_cast<T2*>(y)));
    count_launch();
    return RTM_OK;
}

template <typename T, int NQ> int launch_y(const GridArgs<T>& a, int nrhs, const void* x, void* y, bool fwd,
                                           int minb, cudaStream_t s) {
    if (minb <= 1) {
        if constexpr (three_step(NQ, sizeof(T) == 8)) return launch_y_3<T, NQ, 2>(a, nrhs, x, y, fwd, s);
        else return launch_y_b<T, NQ, 1>(a, nrhs, x, y, fwd, s);
    }
    if constexpr (sizeof(T) == 8) {
        if (minb >= 3) return launch_y_b<T, NQ, 3>(a, nrhs, x, y, fwd, s);
    }
    return launch_y_b<T, NQ, 2>(a, nrhs, x, y, fwd, s);
}

template <typename T, int NP> size_t x_direct_smem() {
    constexpr int R1 = Shape<NP>::R1, R2 = Shape<NP>::R2, TEAMS = Fast<T>::threads / (4 * R2);
    return (size_t)4 * TEAMS * R1 * (R2 + 1) * sizeof(typename Cx<T>::T2);
}

template <typename T, int NP, int MINB> int launch_x_direct(const GridArgs<T>& a, int nrhs, cudaStream_t s) {
    constexpr int TEAMS = Fast<T>::threads / (4 * Shape<NP>::R2);
    const size_t smem = x_direct_smem<T, NP>();
    static DeviceOnce once;
    RTM_TRY(once([smem]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_fast_x_mix_direct<T, NP, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        return RTM_OK;
    }));
    const dim3 grid((a.Q + TEAMS - 1) / TEAMS, 2, nrhs);
    RTM_CUDA(launch_dependent(k_fast_x_mix_direct<T, NP, MINB>, grid, dim3(Fast<T>::threads), smem, s, a));
    count_launch();
    return RTM_OK;
}

template <typename T, int NP, int SUB> int launch_x_3(const GridArgs<T>& a, int nrhs, cudaStream_t s) {
    using S = XMix3<T, NP, SUB>;
    // CTAs an SM, one less and one more: FP64 2 (512 x 512 product 37.2 us, with 3 or 4 spills: 40.4, 37.6), FP32 512
    // 4 (27.9; 5: 28.3), FP32 1024 3 (alone 93; 2: 98, 4: 105).
    constexpr int MINB = sizeof(T) == 8 ? 2 : NP == 1024 ? 3 : 4;
    const size_t smem = (size_t)S::smem_elems * sizeof(typename Cx<T>::T2);
    static DeviceOnce once;
    RTM_TRY(once([smem]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_fast_x_mix_3<T, NP, SUB, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        return RTM_OK;
    }));
    RTM_CUDA(launch_dependent(k_fast_x_mix_3<T, NP, SUB, MINB>, dim3((a.Q + S::teams - 1) / S::teams, SUB, nrhs), dim3(S::threads), smem, s, a));
    count_launch();
    return RTM_OK;
}

template <typename T, int NP> int launch_x_pipe(const GridArgs<T>& a, int nrhs, cudaStream_t s) {
    using M = MixShape<T, NP>;
    static DeviceOnce once;
    static int per_sm[64] = {};
    int dev = 0;
    RTM_CUDA(cudaGetDevice(&dev));
    RTM_TRY(once([dev]() -> int {
        RTM_CUDA(cudaFuncSetAttribute(k_fast_x_mix_pipe<T, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)M::smem));
        int blocks = 0, sms = 0;
        RTM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_fast_x_mix_pipe<T, NP>, Fast<T>::threads,
                                                               M::smem));
        RTM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        if (dev >= 0 && dev < 64) per_sm[dev] = std::max(1, blocks) * sms;
        return RTM_OK;
    }));
    const int iters = nrhs * 2 * (a.Q / M::TEAMS);
    const int resident = dev >= 0 && dev < 64 && per_sm[dev] > 0 ? per_sm[dev] : kDeviceSms;
    const int grid = std::max(1, std::min(iters, resident));
    RTM_CUDA(launch_dependent(k_fast_x_mix_pipe<T, NP>, dim3(grid), dim3(Fast<T>::threads), M::smem, s, a, iters));
    count_launch();
    return RTM_OK;
}

template <typename T, int NP> int launch_x(const GridArgs<T>& a, int nrhs, int kind, cudaStream_t s) {
    if (kind == kMixPipelined) return launch_x_pipe<T, NP>(a, nrhs, s);
    if (kind == kMixDirect2) return launch_x_direct<T, NP, 2>(a, nrhs, s);
    if constexpr (sizeof(T) == 8) {
        if (kind == kMixDirect3) return launch_x_direct<T, NP, 3>(a, nrhs, s);
    }
    if constexpr (three_step(NP, sizeof(T) == 8)) return launch_x_3<T, NP, 2>(a, nrhs, s);
    else return launch_x_direct<T, NP, 1>(a, nrhs, s);
}

template <typename T> int dispatch_y(const GridArgs<T>& a, int nrhs, const void* x, void* y, bool fwd, int minb,
                                     cudaStream_t s) {
    switch (a.Q) {
        case 32: return launch_y<T, 32>(a, nrhs, x, y, fwd, minb, s);
        case 64: return launch_y<T, 64>(a, nrhs, x, y, fwd, minb, s);
        case 128: return launch_y<T, 128>(a, nrhs, x, y, fwd, minb, s);
        case 256: return launch_y<T, 256>(a, nrhs, x, y, fwd, minb, s);
        case 512: return launch_y<T, 512>(a, nrhs, x, y, fwd, minb, s);
        default:
            if constexpr (sizeof(T) == 4) return launch_y<T, 1024>(a, nrhs, x, y, fwd, minb, s);
            return fail(RTM_ERR_UNSUPPORTED, "transform size");
    }
}

template <typename T> int dispatch_x(const GridArgs<T>& a, int nrhs, int kind, cudaStream_t s) {
    switch (a.P) {
        case 32: return launch_x<T, 32>(a, nrhs, kind, s);
        case 64: return launch_x<T, 64>(a, nrhs, kind, s);
        case 128: return launch_x<T, 128>(a, nrhs, kind, s);
        case 256: return launch_x<T, 256>(a, nrhs, kind, s);
        case 512: return launch_x<T, 512>(a, nrhs, kind, s);
        default:
            if constexpr (sizeof(T) == 4) return launch_x<T, 1024>(a, nrhs, kind, s);
            return fail(RTM_ERR_UNSUPPORTED, "transform size");
    }
}

}  // namespace

// The lengths whose passes run in three steps where the other choice is the register-resident lines of grid_reg.cu, with
// no two-step form beside them: FP32 256 gains there too. Circulants, lines of grid_reg.cu -> three steps: FP64 256 x 256
// 20.5 -> 11.3 us, 512 x 512 35.2 -> 17.3; FP32 17.9 -> 10.1, 27.9 -> 15.4, 1024 x 1024 110 -> 36. FP32 split products with
// one length of 256, one vector and four: 256 x 35 17.6 -> 8.4 and 19.6 -> 12.7, 256 x 700 33.0 -> 29.5 and 80.7 ->
// 68.2, 100 x 256 16.9 -> 12.4 and 19.9 -> 18.0.
bool three_step_length(int n, bool fp64) { return n == 256 || n == 512 || (!fp64 && n == 1024); }

namespace {
template <typename T, int N> int three_step_of(int pass, const GridArgs<T>& a, int nrhs, const void* x, void* y, cudaStream_t s) {
    if (pass == kRegXMix) return a.nsx == 2 ? launch_x_3<T, N, 2>(a, nrhs, s) : launch_x_3<T, N, 1>(a, nrhs, s);
    return a.nsy == 2 ? launch_y_3<T, N, 2>(a, nrhs, x, y, pass == kRegYFwd, s)
                      : launch_y_3<T, N, 1>(a, nrhs, x, y, pass == kRegYFwd, s);
}
}  // namespace

template <typename T>
int launch_three_step(int pass, const GridArgs<T>& a, int nrhs, const void* x, void* y, cudaStream_t s) {
    switch (pass == kRegXMix ? a.P : a.Q) {
        case 256: return three_step_of<T, 256>(pass, a, nrhs, x, y, s);
        case 512: return three_step_of<T, 512>(pass, a, nrhs, x, y, s);
        default:
            if constexpr (sizeof(T) == 4) return three_step_of<T, 1024>(pass, a, nrhs, x, y, s);
            return fail(RTM_ERR_UNSUPPORTED, "transform size");
    }
}
template int launch_three_step<double>(int, const GridArgs<double>&, int, const void*, void*, cudaStream_t);
template int launch_three_step<float>(int, const GridArgs<float>&, int, const void*, void*, cudaStream_t);

bool fast_split_eligible(int P, int Q, bool fp64) {
    auto ok = [&](int n) { return n >= 32 && n <= (fp64 ? 512 : 1024) && (n & (n - 1)) == 0; };
    return ok(P) && ok(Q);
}

FastSchedule default_fast_schedule(int P, int Q, bool fp64) {
    FastSchedule f;
    // Three steps where the lengths have them; else the y passes take FP32 two CTAs of 256 threads an SM (128 registers),
    // FP64 three of 128, and the x-mix the direct form, which keeps more warps resident than the pipelined one.
    f.y_blocks = three_step(Q, fp64) ? 1 : fp64 ? 3 : 2;
    f.x_kind = three_step(P, fp64) ? kMixDirect1 : fp64 ? kMixDirect3 : kMixDirect2;
    return f;
}

template <typename T>
int launch_fast_split(const GridArgs<T>& a, int nrhs, const void* x, void* y, const FastSchedule& f, cudaStream_t s) {
    RTM_TRY(dispatch_y<T>(a, nrhs, x, y, true, f.y_blocks, s));
    RTM_TRY(dispatch_x<T>(a, nrhs, f.x_kind, s));
    RTM_TRY(dispatch_y<T>(a, nrhs, x, y, false, f.y_blocks, s));
    RTM_CUDA(cudaGetLastError());
    return RTM_OK;
}

template int launch_fast_split<float>(const GridArgs<float>&, int, const void*, void*, const FastSchedule&,
                                      cudaStream_t);
template int launch_fast_split<double>(const GridArgs<double>&, int, const void*, void*, const FastSchedule&,
                                       cudaStream_t);

}  // namespace rtm
