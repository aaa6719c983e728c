// Internal interface of the tcgen05 INT4 GEMM (int4_gemm.cu).
#pragma once

#include "common.cuh"

namespace kfb {
namespace gemm {

size_t ws_bytes(int M, int N, int K, int group);
// y [M, N] = x W_hat^T (+ bias) in fp16 or bf16; checks its arguments.
int run(const void* x, const void* packed, const void* scales, const void* bias, void* y, int M, int N, int K, int group, bool bf16,
        void* ws, size_t ws_bytes, cudaStream_t stream);

}  // namespace gemm
}  // namespace kfb
