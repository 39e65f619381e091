// Green's-matrix generator assembly on the device.
//
// Follows the reference's
//   src/+rooftopMoM/+assembler/+greensMatrix/@MomentAssembler/generate.m:10-59
//   src/+rooftopMoM/+assembler/+greensMatrix/@MomentAssembler/private/integrateLattice_.m:17-127
//   src/+rooftopMoM/+assembler/+greensMatrix/@MomentAssembler/private/countNearOffsets_.m:1-11
//   src/+rooftopMoM/+assembler/+greensMatrix/+utils/generateReducedRule.m:21-66
//   src/+rooftopMoM/+assembler/+greensMatrix/+utils/integrateMoments.m:17-39
//   src/+rooftopMoM/+assembler/+greensMatrix/+utils/accumulateMoments.m:27-133
//   src/+rooftopMoM/+assembler/+singularIntegrals/evaluateRemainder.m:13-14
//
// Kernels:
//   k_far_blocks  - the kernel exp(-ikR)/R on the far lattice: block (m, n) holds the order^2
//                   points x = a (p - m), y = b (p - n); each block's four quadrant sums of the 7
//                   moment weights (28 complex numbers) are written out.
//   k_near        - one CTA per near offset: 7 weighted sums over the near rule, the remainder of
//                   the singularity extraction on the touching offsets plus their closed form.
//   k_terms       - per offset: the moments (near, or four quadrant sums of the far blocks) and
//                   the 7 scaled combinations of accumulateMoments.m:43-49.
//   k_gather      - per generator entry: E at e; XX at e from e, e + u (rising, doubled at
//                   dX = 1), e - u (falling); YY likewise along y.
#include <cmath>
#include <vector>

#include "fft.cuh"
#include "grid.h"

namespace rtm {

static constexpr double kZ0 = 376.730313668;  // Constants.m:11
static constexpr double kPi = 3.141592653589793238462643383279502884;

// The moment weights are products of one-dimensional ones (generateReducedRule.m:33): of the nodes of an axis
// ([4] columns W00, W10, W01, W11), M00, M10, M01, M11 are W00(eta) W..(nu) and N10, N01, N11 are W..(eta) W00(nu).
__device__ __forceinline__ double moment_weight(int m, const double* wx, int sx, const double* wy, int sy) {
    return m < 4 ? wy[0] * wx[m * sx] : wy[(m - 3) * sy] * wx[0];
}

struct FarArgs {
    int cx, cy;        // faces; blocks are 0..cx x 0..cy
    int order;
    int square;        // square faces: block (n, m) mirrors block (m, n)
    int staged;        // the rule in shared memory
    int64_t nblocks;   // blocks evaluated
    double a, b, k;
    const double* points;   // order far points p in (0, 1)
    const double* weights;  // [2 halves][4][order], of one axis
    double2* sums;          // [28][(cx+1)(cy+1)], block index m + (cx+1) n
};

// The evaluated blocks in order: all of them, or with square faces those of m >= n and the rows n > cx, whose mirror
// images lie outside.
__device__ __forceinline__ void far_block(const FarArgs& f, int64_t t, int& m, int& n) {
    const int64_t W = f.cx + 1;
    if (!f.square) {
        n = (int)(t / W);
        m = (int)(t - n * W);
        return;
    }
    const int64_t last = min(f.cx, f.cy) + (int64_t)1;          // triangular rows: row n holds W - n blocks
    const int64_t tri = last * W - last * (last - 1) / 2;
    if (t >= tri) {
        n = (int)(last + (t - tri) / W);
        m = (int)((t - tri) % W);
        return;
    }
    // the largest n with n W - n (n - 1) / 2 <= t, from the quadratic's root, corrected for its rounding
    const double h = W + 0.5;
    int64_t q = (int64_t)(h - sqrt(fmax(0.0, h * h - 2.0 * (double)t)));
    q = max((int64_t)0, min(q, last - 1));
    while (q > 0 && q * W - q * (q - 1) / 2 > t) --q;
    while (q + 1 < last && (q + 1) * W - (q + 1) * q / 2 <= t) ++q;
    n = (int)q;
    m = (int)(t - (q * W - q * (q - 1) / 2) + q);
}

// A thread per (block, row of points py) evaluates the kernel at its row's points and sums them with the weights along
// x (2 halves x 4 columns) in registers; a thread per (block, quadrant) then sums those along y. Against a thread per
// (block, quadrant) over all points and weights that is 1472 multiply-adds a block instead of 3584, at order 8, and
// no kernel value goes through shared memory; square faces evaluate half the blocks. Bound: the FP64 square root,
// sine, cosine and reciprocal of 64 points a block. 256 x 256 blocks: 33 us, 66 in that form.
constexpr int kFarThreads = 256, kFarRows = 32;  // rows of points a pass takes at most

__global__ void __launch_bounds__(kFarThreads) k_far_blocks(const FarArgs f, int py_threads) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int o = f.order, nb = kFarThreads / py_threads;  // blocks of the CTA
    double2* A = reinterpret_cast<double2*>(smem_raw);      // [py_threads][2 x 4][nb]
    const double* w = f.weights;  // [2][4][order], in shared memory where they fit
    const double* pts = f.points;
    if (f.staged) {
        double* sw = reinterpret_cast<double*>(A + (size_t)py_threads * 8 * nb);
        double* sp = sw + 8 * o;
        for (int t = threadIdx.x; t < 8 * o; t += kFarThreads) sw[t] = f.weights[t];
        for (int t = threadIdx.x; t < o; t += kFarThreads) sp[t] = f.points[t];
        w = sw;
        pts = sp;
    }
    const int64_t first = (int64_t)blockIdx.x * nb, W = f.cx + 1, total = W * (f.cy + 1);
    const int bl = threadIdx.x % nb, row = threadIdx.x / nb;  // block of the CTA; row of points
    const bool in = first + bl < f.nblocks;
    int m = 0, n = 0;
    if (in) far_block(f, first + bl, m, n);
    double2 M[7];
#pragma unroll
    for (int e = 0; e < 7; ++e) M[e] = make_double2(0, 0);
    const int hx = row & 1, hy = (row >> 1) & 1;  // this thread's quadrant in the second part (rows 0 to 3)
    __syncthreads();
    for (int p0 = 0; p0 < o; p0 += py_threads) {
        const int py = p0 + row;
        double2 S[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) S[e] = make_double2(0, 0);
        if (in && py < o) {
            const double y = f.b * (pts[py] - n), y2 = y * y;
            for (int px = 0; px < o; ++px) {
                const double x = f.a * (pts[px] - m);
                const double R = sqrt(x * x + y2);
                double s, c;
                sincos(f.k * R, &s, &c);
                const double inv = 1.0 / R;
                const double kr = c * inv, ki = -s * inv;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    S[e].x = fma(w[e * o + px], kr, S[e].x);
                    S[e].y = fma(w[e * o + px], ki, S[e].y);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) A[(row * 8 + e) * nb + bl] = S[e];
        __syncthreads();
        if (row < 4) {
            const int rows = min(py_threads, o - p0);
            // Last row first: either order has the same error (4e-15 against 64 bits), but the last bits decide how
            // many iterations an unpreconditioned solve of hundreds takes, and in this order they stay nearer the
            // oracle's count (COCG on 12 x 12 faces to 1e-6 within 2 of its 52, 47 in the other).
            for (int q = rows - 1; q >= 0; --q) {
                const double* wy = w + hy * 4 * o + p0 + q;
                double2 a[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) a[e] = A[(q * 8 + hx * 4 + e) * nb + bl];
#pragma unroll
                for (int e = 0; e < 7; ++e) {
                    const double ww = e < 4 ? wy[0] : wy[(e - 3) * o];
                    const double2 v = e < 4 ? a[e] : a[0];
                    M[e].x = fma(ww, v.x, M[e].x);
                    M[e].y = fma(ww, v.y, M[e].y);
                }
            }
        }
        __syncthreads();
    }
    if (row >= 4 || !in) return;
    const int64_t at = m + W * n;
    const int q = hx + 2 * hy;
#pragma unroll
    for (int e = 0; e < 7; ++e) f.sums[(int64_t)(q * 7 + e) * total + at] = M[e];
    if (f.square && m != n && n <= f.cx && m <= f.cy) {
        // x and y exchanged: quadrant (hy, hx) of block (n, m), the M.. and the N.. (M00 is its own image)
        const int64_t mirror = n + W * m;
        const int qm = hy + 2 * hx;
#pragma unroll
        for (int e = 0; e < 7; ++e) f.sums[(int64_t)(qm * 7 + (e == 0 ? 0 : e < 4 ? e + 3 : e - 3)) * total + mirror] = M[e];
    }
}

struct NearArgs {
    int near_x, near_y;
    int px_count, py_count;   // nodes of the near rule along x and y
    double a, b, k;
    const double* nodes_x;
    const double* nodes_y;
    const double* weights_x;  // [px_count][4], [py_count][4]
    const double* weights_y;
    const double* extracted;  // [7][4] closed-form moments at (0,0), (1,0), (0,1), (1,1)
    int count_x, count_y;
    double2* moments;         // [near_x * near_y][7], offset dX + near_x dY
};

__device__ __forceinline__ double2 remainder_kernel(double R, double k) {
    // exp(-ikR)/R - (1/R - k^2 R / 2 + k^4 R^3 / 24), with exp(-ikR) - 1 = -2 sin^2(kR/2) - i sin(kR).
    double sh, ch;
    sincos(0.5 * k * R, &sh, &ch);
    const double em1_re = -2.0 * sh * sh;
    const double em1_im = -2.0 * sh * ch;
    const double k2 = k * k;
    return make_double2(em1_re / R + 0.5 * k2 * R - k2 * k2 / 24.0 * R * R * R, em1_im / R);
}

__global__ void __launch_bounds__(256) k_near(const NearArgs f) {
    const int off = blockIdx.x;
    const int dX = off % f.near_x, dY = off / f.near_x;
    const bool touching = dX <= 1 && dY <= 1;
    const int npts = f.px_count * f.py_count;
    double re[7], im[7];
#pragma unroll
    for (int m = 0; m < 7; ++m) re[m] = im[m] = 0.0;
    for (int p = threadIdx.x; p < npts; p += blockDim.x) {
        const int ix = p % f.px_count, iy = p / f.px_count;
        const double x = f.a * (f.nodes_x[ix] - dX);
        const double y = f.b * (f.nodes_y[iy] - dY);
        const double R = sqrt(x * x + y * y);
        double2 kv;
        if (touching) {
            kv = remainder_kernel(R, f.k);
        } else {
            double s, c;
            sincos(f.k * R, &s, &c);
            kv = make_double2(c / R, -s / R);
        }
#pragma unroll
        for (int m = 0; m < 7; ++m) {
            const double w = moment_weight(m, f.weights_x + 4 * ix, 1, f.weights_y + 4 * iy, 1);
            re[m] = fma(w, kv.x, re[m]);
            im[m] = fma(w, kv.y, im[m]);
        }
    }
    __shared__ double red[7][2][8];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
#pragma unroll
    for (int m = 0; m < 7; ++m) {
        double r = re[m], i = im[m];
        for (int o = 16; o > 0; o >>= 1) {
            r += __shfl_down_sync(0xffffffffu, r, o);
            i += __shfl_down_sync(0xffffffffu, i, o);
        }
        if (lane == 0) {
            red[m][0][warp] = r;
            red[m][1][warp] = i;
        }
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int m = threadIdx.x;
        double r = 0, i = 0;
        for (int w = 0; w < (int)(blockDim.x / 32); ++w) {
            r += red[m][0][w];
            i += red[m][1][w];
        }
        // The closed-form moments of the extracted part on the touching pairs (generate.m:45-52);
        // only offsets inside the grid exist here.
        if (touching && dX < f.count_x && dY < f.count_y) r += f.extracted[m * 4 + dX + 2 * dY];
        f.moments[(int64_t)off * 7 + m] = make_double2(r, i);
    }
}

struct TermArgs {
    int cx, cy;
    int near_x, near_y;
    const double2* near;     // [near_x*near_y][7]
    const double2* sums;     // [28][(cx+1)(cy+1)]
    double2 scale_e, scale_m;
    double2* terms;          // [7][cx*cy], offset dX + cx dY
};

// accumulateMoments.m:43-49: E; XX at e, e - u, e + u; YY at e, e - u, e + u.
__constant__ double c_combine[7][7] = {
    {1, 0, 0, 0, 0, 0, 0},  {1, -1, -1, 2, 0, 0, 0}, {0, 1, 0, -1, 0, 0, 0}, {0, 0, 1, -1, 0, 0, 0},
    {1, 0, 0, 0, -1, -1, 2}, {0, 0, 0, 0, 1, 0, -1}, {0, 0, 0, 0, 0, 1, -1}};

__global__ void k_terms(const TermArgs t) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t G = (int64_t)t.cx * t.cy;
    if (idx >= G) return;
    const int dX = (int)(idx % t.cx), dY = (int)(idx / t.cx);
    double2 M[7];
    if (dX < t.near_x && dY < t.near_y) {
#pragma unroll
        for (int m = 0; m < 7; ++m) M[m] = t.near[(int64_t)(dX + t.near_x * dY) * 7 + m];
    } else {
        const int64_t nb = (int64_t)(t.cx + 1) * (t.cy + 1);
#pragma unroll
        for (int m = 0; m < 7; ++m) M[m] = make_double2(0, 0);
        // Quadrant (hx, hy) takes the block of the offset plus (hx == 0, hy == 0).
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int sx = (q % 2) == 0 ? 1 : 0, sy = (q / 2) == 0 ? 1 : 0;
            const int64_t blk = (dX + sx) + (int64_t)(t.cx + 1) * (dY + sy);
#pragma unroll
            for (int m = 0; m < 7; ++m) {
                const double2 v = t.sums[(int64_t)(q * 7 + m) * nb + blk];
                M[m].x += v.x;
                M[m].y += v.y;
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 7; ++r) {
        double sr = 0, si = 0;
#pragma unroll
        for (int m = 0; m < 7; ++m) {
            sr += c_combine[r][m] * M[m].x;
            si += c_combine[r][m] * M[m].y;
        }
        const double2 sc = r == 0 ? t.scale_e : t.scale_m;
        t.terms[(int64_t)r * G + idx] = make_double2(sc.x * sr - sc.y * si, sc.x * si + sc.y * sr);
    }
}

__global__ void k_gather(int cx, int cy, const double2* __restrict__ terms, double2* __restrict__ E,
                         double2* __restrict__ XX, double2* __restrict__ YY) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t G = (int64_t)cx * cy;
    if (idx >= G) return;
    const int r = (int)(idx % cx), c = (int)(idx / cx);
    auto T = [&](int k, int rr, int cc) { return terms[(int64_t)k * G + rr + (int64_t)cx * cc]; };
    E[idx] = T(0, r, c);
    if (XX && r <= cx - 2) {
        double2 v = T(1, r, c);
        const double f = (r + 1 == 1) ? 2.0 : 1.0;  // the reflected pair at dX = -1
        const double2 rising = T(2, r + 1, c);
        v.x += f * rising.x;
        v.y += f * rising.y;
        if (r >= 1) {
            const double2 falling = T(3, r - 1, c);
            v.x += falling.x;
            v.y += falling.y;
        }
        XX[r + (int64_t)(cx - 1) * c] = v;
    }
    if (YY && c <= cy - 2) {
        double2 v = T(4, r, c);
        const double f = (c + 1 == 1) ? 2.0 : 1.0;
        const double2 rising = T(5, r, c + 1);
        v.x += f * rising.x;
        v.y += f * rising.y;
        if (c >= 1) {
            const double2 falling = T(6, r, c - 1);
            v.x += falling.x;
            v.y += falling.y;
        }
        YY[r + (int64_t)cx * c] = v;
    }
}

// generateReducedRule.m:36-66 along one axis: nodes and the columns W00, W10, W01, W11.
static void reduced_axis(int order, int parts, std::vector<double>& nodes, std::vector<double>& w /* P x 4 */) {
    std::vector<double> pts, pw;
    gauss_legendre(order, 0.0, 1.0, pts, pw);
    const int P = 2 * order * parts;
    nodes.resize(P);
    w.resize((size_t)P * 4);
    for (int half = 0; half < 2; ++half)
        for (int p = 0; p < parts; ++p)
            for (int i = 0; i < order; ++i) {
                const int idx = half * order * parts + p * order + i;
                const double right = (pts[i] + p) / parts;
                const double nu = half == 0 ? right - 1.0 : right;
                nodes[idx] = nu;
                const double g = pw[i] / parts;
                const bool left = nu < 0;
                const double d = std::fabs(nu);
                const double w10 = left ? (1 + nu) * (1 + nu) / 2 : (1 - nu * nu) / 2;
                const double w01 = left ? (1 - nu * nu) / 2 : (1 - nu) * (1 - nu) / 2;
                w[(size_t)idx * 4 + 0] = g * (1 - d);
                w[(size_t)idx * 4 + 1] = g * w10;
                w[(size_t)idx * 4 + 2] = g * w01;
                w[(size_t)idx * 4 + 3] = g * (1 - d) * (1 - d) * (2 + d) / 6;
            }
}

static int count_near(int count, double size, double longest) {
    int n = 0;
    for (int d = 0; d < count; ++d)
        if (std::max(d - 1, 0) * size < 3 * longest) ++n;
    return n;
}

int assemble_generators(int cx, int cy, double a, double b, double k, int near_order, int far_order,
                        DeviceGenerators& out, cudaStream_t s) {
    if (cx < 1 || cy < 1 || (cx == 1 && cy == 1)) return fail(RTM_ERR_ARG, "A single face carries no rooftop.");
    if (!(a > 0) || !(b > 0) || !(k > 0) || !std::isfinite(a) || !std::isfinite(b) || !std::isfinite(k))
        return fail(RTM_ERR_ARG, "face sizes and the wavenumber must be positive and finite");
    if (near_order < 1 || far_order < 1) return fail(RTM_ERR_ARG, "quadrature orders must be positive");
    out.count_x = cx;
    out.count_y = cy;
    const int64_t nxr = (int64_t)(cx - 1) * cy, nyr = (int64_t)cx * (cy - 1);
    out.content = (nxr > 0 && nyr > 0) ? RTM_BOTH : nxr > 0 ? RTM_XONLY : RTM_YONLY;
    out.is_real = false;
    const int64_t G = (int64_t)cx * cy;
    RTM_TRY(out.e.alloc(G * sizeof(double2)));
    if (nxr > 0) RTM_TRY(out.xx.alloc(nxr * sizeof(double2)));
    if (nyr > 0) RTM_TRY(out.yy.alloc(nyr * sizeof(double2)));

    // generate.m:20: i Z0 / (4 pi) (ab)^2 [1/k, k].
    const double base = kZ0 / (4 * kPi) * (a * b) * (a * b);
    const double2 scale_e = make_double2(0.0, base / k), scale_m = make_double2(0.0, base * k);
    const double longest = std::max(a, b);
    const int near_x = count_near(cx, a, longest), near_y = count_near(cy, b, longest);
    const double shortest = std::min(a, b);
    const int parts_x = (int)std::floor(a / shortest + 0.5), parts_y = (int)std::floor(b / shortest + 0.5);

    // The rules of both passes and the closed forms, uploaded together.
    std::vector<double> host;
    auto put = [&](const std::vector<double>& v) {
        const size_t at = host.size();
        host.insert(host.end(), v.begin(), v.end());
        return at;
    };
    std::vector<double> nnx, nny, nwx, nwy, fnx, fw;
    reduced_axis(near_order, parts_x, nnx, nwx);
    reduced_axis(near_order, parts_y, nny, nwy);
    reduced_axis(far_order, 1, fnx, fw);
    double ext[7][4];
    extracted_moments(a, b, k, ext);
    const int o = far_order;
    std::vector<double> axis((size_t)8 * o);  // [half][column][point] of the far rule, whose axes are alike
    for (int h = 0; h < 2; ++h)
        for (int c = 0; c < 4; ++c)
            for (int i = 0; i < o; ++i) axis[(size_t)(h * 4 + c) * o + i] = fw[(size_t)(h * o + i) * 4 + c];
    const size_t at_nx = put(nnx), at_ny = put(nny), at_wx = put(nwx), at_wy = put(nwy),
                 at_ext = put(std::vector<double>(&ext[0][0], &ext[0][0] + 28)),
                 at_pts = put(std::vector<double>(fnx.begin() + o, fnx.end())), at_axis = put(axis);
    const int64_t nblocks = (int64_t)(cx + 1) * (cy + 1);
    DeviceBuffer d_host, d_near, d_sums, d_terms;
    StreamSyncGuard guard(s);
    RTM_TRY(d_host.alloc(host.size() * sizeof(double)));
    RTM_TRY(d_near.alloc((size_t)near_x * near_y * 7 * sizeof(double2)));
    RTM_TRY(d_sums.alloc((size_t)28 * nblocks * sizeof(double2)));
    RTM_CUDA(cudaMemcpyAsync(d_host.ptr, host.data(), d_host.bytes, cudaMemcpyHostToDevice, s));
    const double* dev = d_host.as<double>();

    // Near pass.
    NearArgs na{};
    na.near_x = near_x;
    na.near_y = near_y;
    na.px_count = (int)nnx.size();
    na.py_count = (int)nny.size();
    na.a = a;
    na.b = b;
    na.k = k;
    na.nodes_x = dev + at_nx;
    na.nodes_y = dev + at_ny;
    na.weights_x = dev + at_wx;
    na.weights_y = dev + at_wy;
    na.extracted = dev + at_ext;
    na.count_x = cx;
    na.count_y = cy;
    na.moments = d_near.as<double2>();
    k_near<<<near_x * near_y, 256, 0, s>>>(na);
    count_launch();
    RTM_CUDA(cudaGetLastError());

    // Far lattice (quadrant weights of the far rule, one part per direction).
    FarArgs fa{};
    fa.cx = cx;
    fa.cy = cy;
    fa.order = o;
    fa.square = a == b;
    fa.nblocks = nblocks;
    if (fa.square) {
        const int64_t last = std::min(cx, cy) + (int64_t)1;
        fa.nblocks -= last * (last - 1) / 2;  // the blocks that mirror another one
    }
    fa.a = a;
    fa.b = b;
    fa.k = k;
    fa.points = dev + at_pts;
    fa.weights = dev + at_axis;
    fa.sums = d_sums.as<double2>();
    // a power of two of point rows, at least the four a block's quadrants need
    int py_threads = 4;
    while (py_threads < std::min(o, kFarRows)) py_threads *= 2;
    const int64_t per_cta = kFarThreads / py_threads;
    const size_t values = (size_t)kFarThreads * 8 * sizeof(double2), rule = (size_t)9 * o * sizeof(double);
    fa.staged = values + rule <= 48 * 1024;  // orders up to 227; longer rules are read through the caches
    const size_t far_smem = values + (fa.staged ? rule : 0);
    k_far_blocks<<<(unsigned)((fa.nblocks + per_cta - 1) / per_cta), kFarThreads, far_smem, s>>>(fa, py_threads);
    count_launch();
    RTM_CUDA(cudaGetLastError());

    RTM_TRY(d_terms.alloc((size_t)7 * G * sizeof(double2)));
    TermArgs ta{};
    ta.cx = cx;
    ta.cy = cy;
    ta.near_x = near_x;
    ta.near_y = near_y;
    ta.near = d_near.as<double2>();
    ta.sums = d_sums.as<double2>();
    ta.scale_e = scale_e;
    ta.scale_m = scale_m;
    ta.terms = d_terms.as<double2>();
    k_terms<<<(unsigned)((G + 255) / 256), 256, 0, s>>>(ta);
    k_gather<<<(unsigned)((G + 255) / 256), 256, 0, s>>>(cx, cy, d_terms.as<double2>(), out.e.as<double2>(),
                                                        out.xx.as<double2>(), out.yy.as<double2>());
    count_launch(2);
    RTM_CUDA(cudaGetLastError());
    RTM_CUDA(cudaStreamSynchronize(s));
    return RTM_OK;
}

}  // namespace rtm
