// Internal interface of the RMSNorm + INT4 linear kernel of decode steps (int4_norm.cu).
#pragma once

#include "common.cuh"
#include "int4_epilogue.cuh"

namespace kfb {
namespace normed {

// Whether the kernel takes epilogue(RMSNorm(x[M, K]) . W[N, K]^T), fp16.
bool fits(int M, int N, int K, int group);

// Arguments as checked by the caller: non-null, x, packed and the norm weight 16-byte aligned, fits().
int run(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K, int group, cudaStream_t stream,
        const gemv::Fusion& fu);

}  // namespace normed
}  // namespace kfb
