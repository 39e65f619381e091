// Sources and launch arguments of the spectra builders (grid.cu, gen_reg.cu).
#pragma once

#include "fft.cuh"

namespace rtm {

enum SourceKind { kSrcEmbed = 0, kSrcCirculant = 1, kSrcTwoSided = 2, kSrcPart = 3 };
enum Window { kWinStrang = 0, kWinTChan = 1, kWinRChan = 2, kWinHuckle = 3 };
constexpr int kMaxItems = 12;

struct GenItem {
    const double2* g;  // generator, column-major rows x cols (two-sided sources: (2P - 1) x (2Q - 1))
    int rows, cols;
    int px, py;        // subband parities; part (m, n) of kSrcPart
    double2* dst;      // P x Q output (column-major, x fastest)
};

struct GenArgs {
    int P, Q;
    int kind;
    int Lx, Ly;        // mirror periods of the embedding
    int nsx, nsy;      // folded copies (2 for split directions)
    double scale;
    int window, bw_x, bw_y;
    int realify;
    int ti;
    FftPlan planP, planQ;
    const double2* twP;
    const double2* twQ;
    const double2* modP;
    const double2* modQ;
    int nitems;
    GenItem items[kMaxItems];
};

__device__ __forceinline__ int mirror_index(int i, int rows, int L) {
    if (i < rows) return i;
    const int m = L - i;
    return (m >= 0 && m < rows) ? m : -1;
}

__device__ __forceinline__ double window_weight(int w, int o, int n, int bw) {
    const int ao = o < 0 ? -o : o;
    switch (w) {
        case kWinStrang: return (2 * ao < n) ? 1.0 : (2 * ao == n ? 0.5 : 0.0);
        case kWinTChan: return (double)(n - ao) / (double)n;
        case kWinRChan: return 1.0;
        default: return fmax(0.0, 1.0 - (double)ao / (double)bw);
    }
}

// The source of an item at (i, j); x_mod false: without the x subband's modulation.
__device__ __forceinline__ double2 gen_value(const GenArgs& a, const GenItem& it, int i, int j, bool x_mod = true) {
    double re = 0, im = 0;
    if (a.kind == kSrcEmbed) {
        for (int ca = 0; ca < a.nsx; ++ca) {
            const int mx = mirror_index(i + ca * a.P, it.rows, a.Lx);
            if (mx < 0) continue;
            const double sa = (it.px && ca) ? -1.0 : 1.0;
            for (int cb = 0; cb < a.nsy; ++cb) {
                const int my = mirror_index(j + cb * a.Q, it.cols, a.Ly);
                if (my < 0) continue;
                const double sb = (it.py && cb) ? -1.0 : 1.0;
                const double2 g = it.g[mx + (int64_t)my * it.rows];
                re += sa * sb * g.x;
                im += sa * sb * g.y;
            }
        }
        double2 v = make_double2(re * a.scale, im * a.scale);
        if (it.px && x_mod) v = cmul(v, a.modP[i]);
        if (it.py) v = cmul(v, a.modQ[j]);
        return v;
    }
    if (a.kind == kSrcTwoSided || a.kind == kSrcPart) {
        // A two-sided source, offsets -(P-1)..P-1 by -(Q-1)..Q-1. kSrcTwoSided: the windowed fold onto the
        // face grid (foldGenerator.m:47-60). kSrcPart: part (m, n) of generatePartSpectra.m:15-49, the
        // halved sum (m = 0) or difference (m = 1) of the offsets i and i - P, likewise along y, times
        // exp(i pi i / P) for m = 1 and exp(i pi j / Q) for n = 1.
        const bool part = a.kind == kSrcPart;
        for (int ca = 0; ca < 2; ++ca) {
            if (ca == 1 && i == 0) continue;
            const int ox = ca ? i - a.P : i;
            const double wa = part ? ((it.px && ca) ? -0.5 : 0.5) : window_weight(a.window, ox, a.P, a.bw_x);
            for (int cb = 0; cb < 2; ++cb) {
                if (cb == 1 && j == 0) continue;
                const int oy = cb ? j - a.Q : j;
                const double wb = part ? ((it.py && cb) ? -0.5 : 0.5) : window_weight(a.window, oy, a.Q, a.bw_y);
                const double2 g = it.g[(ox + a.P - 1) + (int64_t)(oy + a.Q - 1) * it.rows];
                re += wa * wb * g.x;
                im += wa * wb * g.y;
            }
        }
        double2 v = make_double2(re, im);
        if (part && it.px) v = cmulc(v, a.modP[i]);
        if (part && it.py) v = cmulc(v, a.modQ[j]);
        return v;
    }
    // Circulant fold of the even generator onto the face grid (foldGenerator.m:38-45).
    for (int ca = 0; ca < 2; ++ca) {
        if (ca == 1 && i == 0) continue;
        const int mx = ca ? a.P - i : i;
        if (mx >= it.rows) continue;
        const double wa = window_weight(a.window, ca ? i - a.P : i, a.P, a.bw_x);
        for (int cb = 0; cb < 2; ++cb) {
            if (cb == 1 && j == 0) continue;
            const int my = cb ? a.Q - j : j;
            if (my >= it.cols) continue;
            const double wb = window_weight(a.window, cb ? j - a.Q : j, a.Q, a.bw_y);
            const double2 g = it.g[mx + (int64_t)my * it.rows];
            re += wa * wb * g.x;
            im += wa * wb * g.y;
        }
    }
    return make_double2(re, im);
}

// One pass of run_gen on lines with a register-resident split (gen_reg.cu): CLS the plan's codelet class, BLUE a
// Bluestein convolution. The sources even in both directions (kSrcEmbed, kSrcCirculant) take half the columns along y
// and half the rows along x. x false: the y pass, plan of a.Q; true: the x pass, plan of a.P.
template <int CLS, bool BLUE> int launch_reg_gen(bool x, const GenArgs& a, const RegPlan& r, cudaStream_t s);

}  // namespace rtm
