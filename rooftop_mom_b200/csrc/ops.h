// Linear operators on rooftop vectors, as the solvers see them.
#pragma once

#include <initializer_list>
#include <memory>

#include "internal.h"

namespace rtm {

// Per-right-hand-side skip flags: an operator skips the vectors whose flag is nonzero.
struct SkipFlags {
    const int* ptr = nullptr;  // device; flag of rhs r at ptr[r * stride]
    int stride = 1;
};

struct LinearOp {
    int64_t n = 0;
    int precision = RTM_FP64;
    virtual ~LinearOp() = default;
    // y = A x for nrhs vectors of length n in the operator's precision, both on the device.
    virtual int apply(const void* x, void* y, int nrhs, cudaStream_t s, SkipFlags skip) = 0;
    // Makes room for nrhs vectors in one apply (outside of any stream capture).
    virtual int reserve(int nrhs) { (void)nrhs; return RTM_OK; }
    virtual double stored_bytes() const { return 0; }
    virtual double working_bytes() const { return 0; }
    // Whether a wait of the operator's kernels has run out since the last call (their stream synchronised before).
    virtual bool take_fault() { return false; }
};

// Synchronises the stream and takes the operators' faults (null entries aside): RTM_ERR_TIMEOUT if there was one.
int fault_check(cudaStream_t s, std::initializer_list<LinearOp*> ops);

// Dense n x n complex FP64 matrix (column-major).
std::unique_ptr<LinearOp> make_dense_op(const double2* device_matrix, int64_t n, int* status);

struct DeviceGenerators;
// Block-Jacobi over blocks of bx x by faces, inverted on the device.
std::unique_ptr<LinearOp> make_block_jacobi(const DeviceGenerators& g, double size_x, double size_y, int bx, int by,
                                            int precision, cudaStream_t s, int* status);

// A block-Jacobi operator as its apply needs it: faces, blocks of bx x by faces in nbx columns and nby rows, the
// packed size S = 2 bx by, the x-directed rooftops, and the inverses of the four block classes
// ([class][S][S], column-major; class (last column) + 2 (last row)) in the operator's precision.
struct BjShape {
    int cx = 0, cy = 0, bx = 1, by = 1, nbx = 0, nby = 0, S = 0;
    int64_t nx_roof = 0;
    const void* inv = nullptr;
};
// False when op is not a block-Jacobi operator.
bool block_jacobi_entry(const LinearOp* op, BjShape* out);
// y = M_k x for count block-Jacobi operators at once (one launch; entry k's vectors start at k * stride),
// entries a device table; max_blocks the most blocks of an entry.
int apply_block_jacobi_batch(const BjShape* entries, int count, int max_blocks, int S, int precision, const void* x,
                             void* y, int64_t stride, cudaStream_t s, SkipFlags skip);

// Precision conversion of complex vectors on the device.
void convert_to_fp32(const double2* in, float2* out, int64_t n, cudaStream_t s);
void convert_to_fp64(const float2* in, double2* out, int64_t n, cudaStream_t s);

}  // namespace rtm
