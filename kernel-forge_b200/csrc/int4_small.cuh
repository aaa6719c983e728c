// Internal interface of the small-batch INT4 linear kernel (int4_small.cu).
#pragma once

#include "common.cuh"
#include "int4_epilogue.cuh"

namespace kfb {
namespace small {

constexpr int kMaxM = 32;

// Arguments as checked by the caller: non-null, x and packed 16-byte aligned, K a multiple of `group` (64 or 128).
// The pair epilogues of `fu` are fp16 only.
int run(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K, int group, bool bf16, cudaStream_t stream,
        const gemv::Fusion& fu);

}  // namespace small
}  // namespace kfb
