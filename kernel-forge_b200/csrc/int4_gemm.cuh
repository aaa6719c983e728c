// Internal interface of the tcgen05 INT4 GEMM (int4_gemm.cu).
#pragma once

#include "common.cuh"

namespace kfb {
namespace gemm {

size_t ws_bytes(int M, int N, int K, int group, bool bf16);
// y [M, N] = x W_hat^T (+ bias) in fp16 or bf16; checks its arguments.  silu (fp16, N % 4 == 0): rows 2j, 2j + 1 of the weight
// are gate and up of one feature and y is [M, N / 2] = silu(gate) * up.
int run(const void* x, const void* packed, const void* scales, const void* bias, void* y, int M, int N, int K, int group, bool bf16,
        bool silu, void* ws, size_t ws_bytes, cudaStream_t stream);

}  // namespace gemm
}  // namespace kfb
