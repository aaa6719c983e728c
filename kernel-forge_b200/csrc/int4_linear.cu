// The dispatcher of the INT4 linear: which kernel serves (M, N, K, dtype).  Host code only.
//
// The reference's dispatcher (kernelforge/ops.py:193-214) knows a GEMV up to M = 7 and a GEMM above; here:
//   M = 1                 CUDA-core GEMV (int4_gemv.cu): one row of activations, nothing for an MMA to share
//   fp16, N >= 75776      persistent streaming kernel (int4_gemv_mma.cuh) up to M = 16, where it has no bias to add
//   M <= 32               small-batch kernel (int4_small.cu), but for few rows of a long K above M = 16
//   otherwise             tcgen05 GEMM (int4_gemm.cu)
#include "int4_gemm.cuh"
#include "int4_small.cuh"

using namespace kfb;

namespace {

enum class Route { kGemv, kStream, kSmall, kGemm };

// Where the lines lie (graph of L2-cold calls, us):
//   M = 1: GEMV / small-batch kernel 5632x2048 4.1/4.7, 1536x8960 5.2/6.2, 2560x2048 3.7/3.7, but 8960x1536 5.0/4.8,
//     11264x2048 8.0/7.3: the GEMV's four or eight rows per warp leave it too few warps there.
//   16 < M <= 32: small-batch kernel / GEMM, M = 32, 5632x2048 10.2/10.7, 8960x1536 9.1/10.2, 2048x8192 9.7/11.1, 4096x4096 9.6/11.8,
//     11264x2048 14.9/12.1, 16384x2048 19.6/12.6; its activation reads grow with M * N, the GEMM's time hardly with M.  Few rows and a
//     long K leave a warp too many groups one after the other, while the GEMM splits K over the chip: M = 17 / 24 / 32, 512x8192 8.8/8.3,
//     9.1/8.4, 10.0/8.5, 512x12288 10.8/9.2, 11.5/9.4, 12.8/9.5, 1280x12288 11.4/10.8, 11.7/11.1, 12.8/11.2; bf16, whose unpacking
//     costs more: 512x6144 7.6/8.4, 7.8/8.6, 8.5/8.7, 512x8192 9.4/8.7, 9.8/8.9, 10.6/9.0.
//     Both lines were drawn before K was walked in blocks of 64, which made the small-batch kernel faster, and are too low for it in
//     places: on the GEMM's side it would be the faster one at M = 17 of 11264x2048 (12.2/13.1; not of 16384x2048, 16.1/13.4), at
//     M = 24 and 32 of 1536x8960 (9.5/10.1, 10.1/10.5; M = 17, on its own side, 9.2/9.7), and for bf16 probably from some N between
//     512 and 1536 on (2048x8192, on its own side, 8.8/12.0, 9.0/11.9, 9.6/12.1).
Route route(int M, int N, int K, int dtype, bool bias) {
  const bool fp16 = dtype == KFB_F16;
  if (fp16 && N >= 75776 && !bias && M <= 16) return M <= 8 ? Route::kGemv : Route::kStream;
  if (fp16 && M == 1 && N < 8192) return Route::kGemv;
  if (M > 32 || (M > 16 && (long long)N * K > 16LL << 20)) return Route::kGemm;
  if (M > 16 && N <= 1536 && K >= 8192 && (!fp16 || (long long)K * (M + 8) > 8192 * 32)) return Route::kGemm;
  return Route::kSmall;
}

}  // namespace

extern "C" int kfb_int4_linear_route(int M, int N, int K, int dtype, int with_bias) {
  if (M < 1 || N < 1 || K < 1 || (dtype != KFB_F16 && dtype != KFB_BF16)) return fail(KFB_ERR_INVALID, "no such linear: M=%d N=%d K=%d", M, N, K);
  return (int)route(M, N, K, dtype, with_bias != 0);
}

extern "C" size_t kfb_int4_linear_ws_bytes(int M, int N, int K, int group, int dtype) {
  return M <= 16 ? 0 : route(M, N, K, dtype, false) == Route::kGemm ? gemm::ws_bytes(M, N, K, group, dtype == KFB_BF16) : 0;
}

namespace {

int check_small(const void* x, const void* packed, int N, int K, int group) {
  if (int rc = require_sm100()) return rc;
  if (group != 64 && group != 128) return fail(KFB_ERR_INVALID, "group_size must be one of (64, 128), got %d", group);
  if (N < 1 || K < group || K % group) return fail(KFB_ERR_INVALID, "K=%d is not a multiple of group_size=%d", K, group);
  if (!aligned16(x) || !aligned16(packed)) return fail(KFB_ERR_ALIGNMENT, "x and packed must be 16-byte aligned");
  return KFB_OK;
}

}  // namespace

extern "C" int kfb_int4_linear(const void* x, const void* packed, const void* scales, const void* bias, void* y, int M, int N,
                               int K, int group, int dtype, void* ws, size_t ws_bytes, void* stream) {
  if (dtype != KFB_F16 && dtype != KFB_BF16) return fail(KFB_ERR_INVALID, "int4_linear takes fp16 or bf16 activations");
  if (!x || !packed || !scales || !y) return fail(KFB_ERR_INVALID, "null pointer");
  if (M < 1) return fail(KFB_ERR_INVALID, "int4_linear needs M >= 1, got M=%d", M);
  switch (route(M, N, K, dtype, bias != nullptr)) {
    case Route::kGemv:
      if (bias) return kfb_int4_gemv_fused(x, packed, scales, y, M, N, K, group, 0, nullptr, 0.0f, bias, nullptr, 0, stream);
      return kfb_int4_gemv(x, packed, scales, y, M, N, K, group, 0, stream);
    case Route::kStream: return kfb_int4_small_batch(x, packed, scales, y, M, N, K, group, 0, stream);
    case Route::kSmall: {
      if (int rc = check_small(x, packed, N, K, group)) return rc;
      gemv::Fusion fu = {};
      fu.bias = static_cast<const __half*>(bias);
      return small::run(x, packed, scales, y, M, N, K, group, dtype == KFB_BF16, (cudaStream_t)stream, fu);
    }
    default: return gemm::run(x, packed, scales, bias, y, M, N, K, group, dtype == KFB_BF16, false, ws, ws_bytes, (cudaStream_t)stream);
  }
}

extern "C" int kfb_int4_linear_silu_pairs(const void* x, const void* packed, const void* scales, void* act, int M, int N, int K, int group,
                                          void* ws, size_t ws_bytes, void* stream) {
  if (!x || !packed || !scales || !act) return fail(KFB_ERR_INVALID, "null pointer");
  if (M < 1 || N < 4 || N % 4) return fail(KFB_ERR_INVALID, "int4_linear_silu_pairs needs M >= 1 and N a multiple of 4, got M=%d N=%d", M, N);
  const Route r = route(M, N, K, KFB_F16, true);
  if (r == Route::kGemm) return gemm::run(x, packed, scales, nullptr, act, M, N, K, group, false, true, ws, ws_bytes, (cudaStream_t)stream);
  if (r == Route::kGemv) return kfb_int4_gemv_silu_pair(x, packed, scales, act, M, N, K, group, 0, nullptr, 0.0f, 0, stream);
  if (int rc = check_small(x, packed, N, K, group)) return rc;
  gemv::Fusion fu = {};
  fu.epi = gemv::kEpiSiluPair;
  return small::run(x, packed, scales, act, M, N, K, group, false, (cudaStream_t)stream, fu);
}
