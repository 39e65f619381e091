// A GMRES solve whose device-side barriers may not be polled at all, so that every wait gives up at once: the call
// returns RTM_ERR_TIMEOUT, and the same solve with the default limit then succeeds on the same stream. The solver's source
// is part of this unit, since the limit is no part of the C ABI. Prints "<name> <status> <converged> <residual>" a line.
#include <cstdio>

#include "../../rooftop_mom_b200/csrc/krylov.cu"

namespace rtm {
// strip_solve.cu, which no dense operator reaches
template <typename T>
int strip_cocg(LinearOp*, LinearOp*, const SolveConfig&, const void*, const void*, void*, int64_t, int, SolveResult&,
               cudaStream_t, bool* taken) {
    *taken = false;
    return RTM_OK;
}
template int strip_cocg<float>(LinearOp*, LinearOp*, const SolveConfig&, const void*, const void*, void*, int64_t, int,
                               SolveResult&, cudaStream_t, bool*);
template int strip_cocg<double>(LinearOp*, LinearOp*, const SolveConfig&, const void*, const void*, void*, int64_t, int,
                                SolveResult&, cudaStream_t, bool*);
}  // namespace rtm

// y = (3 + i) x_i + x_(i - 1) + x_(i + 1): well conditioned, and no Krylov space of few columns holds its solution.
__global__ void k_tridiagonal(const double2* x, double2* y, int64_t n, const int* skip, int stride) {
    if (skip && skip[(int64_t)blockIdx.y * stride]) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    x += blockIdx.y * n;
    y += blockIdx.y * n;
    double2 s = make_double2(3 * x[i].x - x[i].y, 3 * x[i].y + x[i].x);
    if (i > 0) s = make_double2(s.x + x[i - 1].x, s.y + x[i - 1].y);
    if (i + 1 < n) s = make_double2(s.x + x[i + 1].x, s.y + x[i + 1].y);
    y[i] = s;
}

struct Tridiagonal : rtm::LinearOp {
    int apply(const void* x, void* y, int nrhs, cudaStream_t s, rtm::SkipFlags skip) override {
        k_tridiagonal<<<dim3((unsigned)((n + 127) / 128), nrhs), 128, 0, s>>>(
            static_cast<const double2*>(x), static_cast<double2*>(y), n, skip.ptr, skip.stride);
        return cudaGetLastError() == cudaSuccess ? RTM_OK : RTM_ERR_CUDA;
    }
};

int main() {
    constexpr int64_t n = 5000;
    constexpr int nrhs = 2;
    Tridiagonal op;
    op.n = n;
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    std::vector<double2> host(n * nrhs);
    for (int64_t i = 0; i < n * nrhs; ++i) host[i] = make_double2(std::cos(0.37 * i), std::sin(0.11 * i * i));
    double2 *b = nullptr, *x = nullptr;
    if (cudaMalloc(&b, n * nrhs * sizeof(double2)) != cudaSuccess || cudaMalloc(&x, n * nrhs * sizeof(double2)) != cudaSuccess)
        return 1;
    cudaMemcpy(b, host.data(), n * nrhs * sizeof(double2), cudaMemcpyHostToDevice);
    rtm::SolveConfig cfg;
    cfg.method = RTM_METHOD_GMRES;
    cfg.restart = 20;
    cfg.tolerance = 1e-10;
    for (int pass = 0; pass < 2; ++pass) {
        rtm::SolveConfig c = cfg;
        if (pass == 0) c.barrier_polls = 0;
        rtm::SolveResult res;
        const int status = rtm::solve(&op, nullptr, c, b, nullptr, x, n, nrhs, res, s);
        std::printf("%s %d %d %.3e\n", pass ? "default" : "unpolled", status,
                    res.stats.empty() ? -1 : res.stats[0].converged && res.stats[1].converged,
                    res.stats.empty() ? -1.0 : std::max(res.stats[0].residual_norm, res.stats[1].residual_norm));
    }
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
