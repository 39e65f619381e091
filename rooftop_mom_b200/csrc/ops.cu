// Dense operator and block-Jacobi preconditioner.
//
// The Green's-matrix entry between rooftops p and q follows the definition the reference's tests use
// (tests/+unit/Base.m:83-113): the magnetic generator of their direction at the offset of their first
// faces, minus sum over the two faces of each of div_p(f) E(f - f') div_q(f'), with the divergence
// +1/h on the first face and -1/h on the second (h the face size along the rooftop).
#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "fft.cuh"
#include "grid.h"
#include "ops.h"
#include "pdl.cuh"

namespace rtm {

__global__ void k_dense(const double2* __restrict__ A, const double2* __restrict__ x, double2* __restrict__ y, int64_t n,
                        const int* skip, int stride) {
    const int rhs = blockIdx.y;
    if (skip && skip[(int64_t)rhs * stride]) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double2* xr = x + rhs * n;
    double re = 0, im = 0;
    for (int64_t j = 0; j < n; ++j) {
        const double2 a = A[i + j * n], v = xr[j];
        re += a.x * v.x - a.y * v.y;
        im += a.x * v.y + a.y * v.x;
    }
    y[rhs * n + i] = make_double2(re, im);
}

struct DenseOp : LinearOp {
    DeviceBuffer A;
    int apply(const void* x, void* y, int nrhs, cudaStream_t s, SkipFlags skip) override {
        dim3 g((unsigned)((n + 127) / 128), nrhs);
        k_dense<<<g, 128, 0, s>>>(A.as<double2>(), static_cast<const double2*>(x), static_cast<double2*>(y), n,
                                  skip.ptr, skip.stride);
        count_launch();
        RTM_CUDA(cudaGetLastError());
        return RTM_OK;
    }
    double stored_bytes() const override { return (double)A.bytes; }
};

std::unique_ptr<LinearOp> make_dense_op(const double2* device_matrix, int64_t n, int* status) {
    auto op = std::make_unique<DenseOp>();
    op->n = n;
    op->precision = RTM_FP64;
    *status = op->A.alloc((size_t)n * n * sizeof(double2));
    if (*status != RTM_OK) return nullptr;
    if (cudaMemcpy(op->A.ptr, device_matrix, (size_t)n * n * sizeof(double2), cudaMemcpyDeviceToDevice) != cudaSuccess) {
        *status = fail(RTM_ERR_CUDA, "copy of the dense matrix failed");
        return nullptr;
    }
    return op;
}

// ---------------------------------------------------------------------------------------------
// Block-Jacobi. A block's matrix depends on the offsets between its rooftops alone, and only the last block
// column and the last block row lack rooftops (their last faces are no first faces), so a plate has four
// distinct block matrices at most: class (last column) + 2 (last row). Four inverses are formed and stored; the
// apply reads them from the caches instead of one inverse per block (the 256 x 256 plate's 16.8 MB).
constexpr int kMaxBlockUnknowns = 16;
constexpr int kBlockClasses = 4;

__device__ double2 green_entry(const BjShape& g, const double2* E, const double2* XX, const double2* YY, double a,
                               double b, int dp, int ip, int jp, int dq, int iq, int jq) {
    double re = 0, im = 0;
    if (dp == dq) {
        const int dx = abs(ip - iq), dy = abs(jp - jq);
        const double2 m = dp == 0 ? XX[dx + (int64_t)(g.cx - 1) * dy] : YY[dx + (int64_t)g.cx * dy];
        re = m.x;
        im = m.y;
    }
    const double hp = dp == 0 ? a : b, hq = dq == 0 ? a : b;
    for (int s = 0; s < 2; ++s) {
        const int fi = ip + (s && dp == 0), fj = jp + (s && dp == 1);
        for (int t = 0; t < 2; ++t) {
            const int gi = iq + (t && dq == 0), gj = jq + (t && dq == 1);
            const double2 e = E[abs(fi - gi) + (int64_t)g.cx * abs(fj - gj)];
            const double w = ((s == t) ? 1.0 : -1.0) / (hp * hq);
            re -= w * e.x;
            im -= w * e.y;
        }
    }
    return make_double2(re, im);
}

// The unknowns of a block with wx x wy faces, rx of its faces with an x-directed rooftop per row and ry rows of
// faces with y-directed ones: x-directed rooftops first, i fastest.
struct BlockLayout {
    int wx, wy, rx, ry;
    __host__ __device__ int count() const { return rx * wy + wx * ry; }
    // direction and first face (within the block) of unknown r < count()
    __device__ void unknown(int r, int& dir, int& i, int& j) const {
        dir = r >= rx * wy;
        const int q = dir ? r - rx * wy : r, w = dir ? wx : rx;
        j = q / w;
        i = q - j * w;
    }
};
// Layout of the blocks in column class lx and row class ly (1: the last one).
__host__ __device__ inline BlockLayout block_layout(const BjShape& g, int lx, int ly) {
    BlockLayout l;
    l.wx = lx ? g.cx - (g.nbx - 1) * g.bx : g.bx;
    l.wy = ly ? g.cy - (g.nby - 1) * g.by : g.by;
    l.rx = lx ? l.wx - 1 : g.bx;
    l.ry = ly ? l.wy - 1 : g.by;
    return l;
}

// One CTA per class, a thread per entry of [A | B]: forms the block of the Green's matrix and inverts it by
// Gauss-Jordan elimination with partial pivoting in shared memory; a chain of at most 16 columns, latency bound
// (one thread per block of the plate had taken 175 us on the 256 x 256 plate). Writes the inverse packed
// column-major with S = 2 bx by unknowns (entry (r, c) at class S^2 + c S + r).
constexpr int kBuildThreads = kMaxBlockUnknowns * kMaxBlockUnknowns;
template <typename T2>
__global__ void __launch_bounds__(kBuildThreads) k_bj_build(const BjShape g, const double2* __restrict__ E,
                                                            const double2* __restrict__ XX,
                                                            const double2* __restrict__ YY, double a, double b,
                                                            T2* __restrict__ out, int* __restrict__ singular) {
    __shared__ double2 A[kMaxBlockUnknowns][kMaxBlockUnknowns + 1], B[kMaxBlockUnknowns][kMaxBlockUnknowns + 1];
    __shared__ int pivot;
    const int lx = blockIdx.x & 1, ly = blockIdx.x >> 1;
    T2* dst = out + (int64_t)blockIdx.x * g.S * g.S;
    const int r = threadIdx.x % kMaxBlockUnknowns, c = threadIdx.x / kMaxBlockUnknowns;
    const bool present = (lx || g.nbx > 1) && (ly || g.nby > 1);  // some block of the plate is of this class
    const BlockLayout l = block_layout(g, lx, ly);
    const int cnt = present ? l.count() : 0;
    if (r < g.S && c < g.S) dst[c * g.S + r] = czero<T2>();
    const bool in = r < cnt && c < cnt;
    if (in) {
        int dp, ip, jp, dq, iq, jq;
        l.unknown(r, dp, ip, jp);
        l.unknown(c, dq, iq, jq);
        A[r][c] = green_entry(g, E, XX, YY, a, b, dp, ip, jp, dq, iq, jq);
        B[r][c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    for (int col = 0; col < cnt; ++col) {
        if (threadIdx.x == 0) {
            int piv = col;
            double best = -1;
            for (int q = col; q < cnt; ++q) {
                const double v = A[q][col].x * A[q][col].x + A[q][col].y * A[q][col].y;
                if (v > best) { best = v; piv = q; }
            }
            pivot = best > 0 ? piv : -1;
        }
        __syncthreads();
        const int piv = pivot;
        if (piv < 0) {
            if (threadIdx.x == 0) atomicExch(singular, 1);
            return;
        }
        // row `col` after the exchange and its scaling, and every row's factor, read before anything is written
        double2 pa, pb, f, own_a, own_b;
        if (in) {
            const double2 p = A[piv][col];
            const double d = p.x * p.x + p.y * p.y;
            const double2 inv = make_double2(p.x / d, -p.y / d);
            pa = cmul(A[piv][c], inv);
            pb = cmul(B[piv][c], inv);
            const int src = r == piv ? col : r;  // the row that stands at r after the exchange
            f = A[src][col];
            own_a = A[src][c];
            own_b = B[src][c];
        }
        __syncthreads();
        if (in) {
            A[r][c] = r == col ? pa : csub(own_a, cmul(f, pa));
            B[r][c] = r == col ? pb : csub(own_b, cmul(f, pb));
        }
        __syncthreads();
    }
    if (in) dst[c * g.S + r] = cmake<T2>(B[r][c].x, B[r][c].y);
}

// y(idx_r) = sum_c inv(r, c) x(idx_c) over the block's unknowns, one thread per (block, row). Where S divides
// the warp (blocks of 1, 2, 4, 8 or 16 unknowns, 2 x 2 faces among them), the S threads of a block each gather
// their own x(idx_r) and pass it to the others by warp shuffles, so a thread issues one vector load instead of S;
// the sum runs over c in the same order either way. Bound: the vectors (read and written once); the inverses
// stay in L1. The 256 x 256 plate, FP64: 7.2 us with an inverse and an index list per block, 5.4 with a
// class's (cold caches; 3.1 warm).
template <typename T2, int SC>  // SC: S as a compile-time constant (the loops unroll), or 0
__device__ __forceinline__ void bj_rows(const BjShape& g, const T2* __restrict__ xr, T2* __restrict__ yr, int64_t t) {
    const int S = SC ? SC : g.S;
    const int nblocks = g.nbx * g.nby;
    const int blk = (int)(t / S), r = (int)(t % S);
    const bool in = t < (int64_t)nblocks * S;
    const int J = in ? blk / g.nbx : 0, I = in ? blk - J * g.nbx : 0;
    const int lx = I == g.nbx - 1, ly = J == g.nby - 1;
    const BlockLayout l = block_layout(g, lx, ly);
    const int cnt = in ? l.count() : 0;
    const T2* inv = static_cast<const T2*>(g.inv) + (lx + 2 * ly) * S * S;
    auto index = [&](int u) -> int64_t {
        int dir, i, j;
        l.unknown(u, dir, i, j);
        i += I * g.bx;
        j += J * g.by;
        return dir ? g.nx_roof + i + (int64_t)g.cx * j : i + (int64_t)(g.cx - 1) * j;
    };
    const bool row = r < cnt;
    if ((32 % S) == 0) {
        // every lane reaches the shuffles: blocks past the end and rows past a block's count carry zeros
        const int64_t at = row ? index(r) : 0;
        const T2 mine = row ? xr[at] : czero<T2>();
        const int base = (int)(threadIdx.x & 31) - r;  // the block's first lane (blocks align with warps)
        T2 acc = czero<T2>();
#pragma unroll 16
        for (int c = 0; c < S; ++c) {
            T2 v;
            v.x = __shfl_sync(0xffffffffu, mine.x, base + c);
            v.y = __shfl_sync(0xffffffffu, mine.y, base + c);
            if (c < cnt && row) acc = cadd(acc, cmul(__ldg(&inv[c * S + r]), v));
        }
        if (row) yr[at] = acc;
        return;
    }
    if (!row) return;
    T2 acc = czero<T2>();
    // unrolled so that the loads of all columns are in flight together (the order of the sum is unchanged)
#pragma unroll 8
    for (int c = 0; c < cnt; ++c) acc = cadd(acc, cmul(__ldg(&inv[c * S + r]), xr[index(c)]));
    yr[index(r)] = acc;
}

template <typename T2>
__global__ void k_bj_apply(const BjShape g, const T2* __restrict__ x, T2* __restrict__ y, int64_t n, const int* skip,
                           int stride) {
    griddep_wait();
    const int rhs = blockIdx.y;
    if (skip && skip[(int64_t)rhs * stride]) return;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g.S == 8) bj_rows<T2, 8>(g, x + rhs * n, y + rhs * n, t);
    else bj_rows<T2, 0>(g, x + rhs * n, y + rhs * n, t);
}

// k_bj_apply for a batch of block-Jacobi operators: right-hand side k takes entry k's blocks, and its vector is zero behind
// the entry's rooftops.
template <typename T2>
__global__ void k_bj_apply_batch(const BjShape* __restrict__ entries, const T2* __restrict__ x, T2* __restrict__ y,
                                 int64_t stride, const int* skip, int skip_stride) {
    griddep_wait();
    const int rhs = blockIdx.y;
    if (skip && skip[(int64_t)rhs * skip_stride]) return;
    const BjShape e = entries[rhs];
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    for (int64_t i = (int64_t)(e.cx - 1) * e.cy + (int64_t)e.cx * (e.cy - 1) + t; i < stride;
         i += (int64_t)gridDim.x * blockDim.x)
        y[rhs * stride + i] = T2{};
    if (e.S == 8) bj_rows<T2, 8>(e, x + rhs * stride, y + rhs * stride, t);
    else bj_rows<T2, 0>(e, x + rhs * stride, y + rhs * stride, t);
}

int apply_block_jacobi_batch(const BjShape* entries, int count, int max_blocks, int S, int precision, const void* x,
                             void* y, int64_t stride, cudaStream_t s, SkipFlags skip) {
    const int64_t threads = (int64_t)max_blocks * S;
    const dim3 g((unsigned)((threads + 255) / 256), count);
    if (precision == RTM_FP64)
        RTM_CUDA(launch_dependent(k_bj_apply_batch<double2>, g, dim3(256), 0, s, entries, static_cast<const double2*>(x),
                                  static_cast<double2*>(y), stride, skip.ptr, skip.stride));
    else
        RTM_CUDA(launch_dependent(k_bj_apply_batch<float2>, g, dim3(256), 0, s, entries, static_cast<const float2*>(x),
                                  static_cast<float2*>(y), stride, skip.ptr, skip.stride));
    count_launch();
    RTM_CUDA(cudaGetLastError());
    return RTM_OK;
}

struct BlockJacobi : LinearOp {
    BjShape shape;
    DeviceBuffer inv;  // [kBlockClasses][S][S]
    int apply(const void* x, void* y, int nrhs, cudaStream_t s, SkipFlags skip) override {
        const int64_t threads = (int64_t)shape.nbx * shape.nby * shape.S;
        dim3 g((unsigned)((threads + 255) / 256), nrhs);
        if (precision == RTM_FP64)
            RTM_CUDA(launch_dependent(k_bj_apply<double2>, g, dim3(256), 0, s, shape, static_cast<const double2*>(x),
                                      static_cast<double2*>(y), n, skip.ptr, skip.stride));
        else
            RTM_CUDA(launch_dependent(k_bj_apply<float2>, g, dim3(256), 0, s, shape, static_cast<const float2*>(x),
                                      static_cast<float2*>(y), n, skip.ptr, skip.stride));
        count_launch();
        RTM_CUDA(cudaGetLastError());
        return RTM_OK;
    }
    double stored_bytes() const override { return (double)inv.bytes; }
};

bool block_jacobi_entry(const LinearOp* op, BjShape* out) {
    const auto* bj = dynamic_cast<const BlockJacobi*>(op);
    if (!bj) return false;
    *out = bj->shape;
    return true;
}

std::unique_ptr<LinearOp> make_block_jacobi(const DeviceGenerators& gen, double size_x, double size_y, int bx, int by,
                                            int precision, cudaStream_t s, int* status) {
    if (bx < 1 || by < 1 || 2 * bx * by > kMaxBlockUnknowns) {
        *status = fail(RTM_ERR_UNSUPPORTED, "block-Jacobi blocks hold at most 8 faces in this build");
        return nullptr;
    }
    auto op = std::make_unique<BlockJacobi>();
    const int cx = gen.count_x, cy = gen.count_y;
    const int64_t nx_roof = (int64_t)(cx - 1) * cy, ny_roof = (int64_t)cx * (cy - 1);
    op->n = nx_roof + ny_roof;
    op->precision = precision;
    BjShape& g = op->shape;
    g.cx = cx;
    g.cy = cy;
    g.bx = bx;
    g.by = by;
    g.nbx = (cx + bx - 1) / bx;
    g.nby = (cy + by - 1) / by;
    g.S = 2 * bx * by;
    g.nx_roof = nx_roof;
    DeviceBuffer flag;
    StreamSyncGuard guard(s);
    const size_t entries = (size_t)kBlockClasses * g.S * g.S;
    if ((*status = op->inv.alloc(entries * (precision == RTM_FP64 ? sizeof(double2) : sizeof(float2)))) != RTM_OK)
        return nullptr;
    if ((*status = flag.alloc(sizeof(int))) != RTM_OK) return nullptr;
    if ((*status = check_cuda(cudaMemsetAsync(flag.ptr, 0, sizeof(int), s), "block-Jacobi flag")) != RTM_OK)
        return nullptr;
    g.inv = op->inv.ptr;
    const double2 *E = gen.e.as<double2>(), *XX = gen.xx.as<double2>(), *YY = gen.yy.as<double2>();
    if (precision == RTM_FP64)
        k_bj_build<double2><<<kBlockClasses, kBuildThreads, 0, s>>>(g, E, XX, YY, size_x, size_y,
                                                                    op->inv.as<double2>(), flag.as<int>());
    else
        k_bj_build<float2><<<kBlockClasses, kBuildThreads, 0, s>>>(g, E, XX, YY, size_x, size_y, op->inv.as<float2>(),
                                                                   flag.as<int>());
    count_launch();
    if ((*status = check_cuda(cudaGetLastError(), "block-Jacobi build launch")) != RTM_OK) return nullptr;
    int bad = 0;
    if ((*status = check_cuda(cudaMemcpyAsync(&bad, flag.ptr, sizeof(int), cudaMemcpyDeviceToHost, s),
                              "block-Jacobi flag")) != RTM_OK)
        return nullptr;
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        *status = cuda_fail(e, "block-Jacobi build");
        return nullptr;
    }
    if (bad) {
        *status = fail(RTM_ERR_SINGULAR, "a block of the block-Jacobi preconditioner is singular");
        return nullptr;
    }
    *status = RTM_OK;
    return op;
}

}  // namespace rtm
