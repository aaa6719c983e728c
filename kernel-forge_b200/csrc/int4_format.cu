// INT4 weight format on the GPU: quantise+pack, pack, unpack, dequantise.
//
// Bit-exact with the torch implementation of the reference (kernelforge/quantize.py:61-114):
// every step is an IEEE fp32 operation (division, rint = round-half-to-even, one RN to fp16),
// so no fast-math flag may be applied to this file.  The kernels stream the weight once
// (HBM-bound: 4 B read + 0.52 B written per weight for fp32 input).
#include "common.cuh"

namespace kfb {
namespace {

// nibble position (bits 4p..4p+3) of k-offset o inside its 8-weight word:
// positions 0..7 hold offsets 0,2,4,6,1,3,5,7 (kernelforge/quantize.py:34).
__device__ __forceinline__ int nibble_pos(int o) { return (o >> 1) + ((o & 1) << 2); }

// The 8 weights of one packed word as FP32.
__device__ __forceinline__ void load8(const float* w, float (&v)[8]) {
  const float4 a = __ldcs(reinterpret_cast<const float4*>(w)), b = __ldcs(reinterpret_cast<const float4*>(w) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __half* w, float (&v)[8]) {
  const uint4 a = __ldcs(reinterpret_cast<const uint4*>(w));
  const __half2* h = reinterpret_cast<const __half2*>(&a);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void load8(const __nv_bfloat16* w, float (&v)[8]) {
  const uint4 a = __ldcs(reinterpret_cast<const uint4*>(w));
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&a);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}

// The packed word by definition: clamp(rint(v / s), -8, 7) + 8 with the quotient rounded to FP32 first.
struct Eight {   // by value: an array whose address is taken would live in local memory for everybody
  float v[8];
};
__device__ __noinline__ uint32_t pack_exact(Eight w, float s) {
  uint32_t word = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    word |= (uint32_t)((int)fminf(fmaxf(rintf(__fdiv_rn(w.v[j], s)), -8.0f), 7.0f) + 8) << (4 * nibble_pos(j));
  return word;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Largest magnitude of three (one instruction on sm_100); NaN only if all are.
__device__ __forceinline__ float max_abs3(float a, float b, float c) {
  float y;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// One lane per packed word (8 consecutive k); G / 8 neighbouring lanes share a group.  Words and groups are contiguous
// over the whole tensor, so a CTA takes a run of kUnroll * 256 flat word indices and knows no rows.
//
// HBM-bound by design (2.5 bytes per fp16 weight), bound by issue slots in fact.  One IEEE division per weight (a dozen
// instructions) and 8-byte loads took 42.8 us for 11264 x 2048 fp16; this kernel takes 14.9 us (3.9 TB/s; with one weight per
// floating-point instruction 15.1, bf16 16.8 and now 16.3).  A weight is
// multiplied with the group's reciprocal and rounded by the magic-number addition of one FMA.  The product is off by at
// most 2^-22 of itself, so the result can only differ from the definition's next to a half integer; a lane that sees such
// a weight (or a quotient above 7.4, infinity, NaN) packs its word by the definition.
constexpr int kQuantThreads = 256;
constexpr int kQuantUnroll = 2;   // words per lane, requested at once (1 or 4: 5 % slower)

template <typename T, int G>
__global__ void __launch_bounds__(kQuantThreads, 8) quantize_pack_kernel(const T* __restrict__ w, uint32_t* __restrict__ packed,
                                                                         __half* __restrict__ scales, long long words) {
  constexpr int kLanes = G / 8;
  pdl_wait(w);   // (the successor is not released early: it may read these weights before its own wait)
  // a group's lanes all have a word or none, since `words` is a multiple of kLanes
  const long long first = (long long)blockIdx.x * (kQuantUnroll * kQuantThreads);
  const int left = (int)min(words - first, (long long)(kQuantUnroll * kQuantThreads));
  w += first * 8;
  packed += first;
  scales += first / kLanes;
  float v[kQuantUnroll][8];
#pragma unroll
  for (int u = 0; u < kQuantUnroll; ++u) {
    const int i = u * kQuantThreads + threadIdx.x;
    load8(w + 8 * min(i, left - 1), v[u]);   // past the end: the last word again, not stored
  }
#pragma unroll
  for (int u = 0; u < kQuantUnroll; ++u) {
    const int i = u * kQuantThreads + threadIdx.x;
    float amax = max_abs3(max_abs3(v[u][0], v[u][1], v[u][2]), max_abs3(v[u][3], v[u][4], v[u][5]), max_abs3(v[u][6], v[u][7], v[u][7]));
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    // scale = fp16(max(absmax / 7, smallest normal fp16)); exactly 1 for an all-zero group
    __half sh = __float2half_rn(fmaxf(__fdiv_rn(amax, 7.0f), 6.103515625e-05f));
    if (amax == 0.0f) sh = __float2half_rn(1.0f);
    const float s32 = __half2float(sh), inv = rcp_approx(s32);
    // v * inv + 1.5 * 2^23 has rint(v / s) in its low bits (ties to even).  Rounding it with a slightly smaller and a
    // slightly larger reciprocal tells whether the error of inv could matter.  The words of the sums are kBits + rint;
    // the constant part, and the + 8 of every nibble, come in through kSum, so no masks are needed.
    constexpr float kMagic = 12582912.0f;
    constexpr uint32_t kBits = 0x4B400000u, kSum = 0u - (kBits - 8u) * 0x11111111u;
    const float lo = inv * (1.0f - 1.0f / 1048576.0f), hi = inv * (1.0f + 1.0f / 1048576.0f);
    const float2 lo2 = make_float2(lo, lo), hi2 = make_float2(hi, hi), magic2 = make_float2(kMagic, kMagic);
    uint32_t word = kSum, differ = 0;
    float2 sum = make_float2(0.0f, 0.0f);   // not finite if any weight is (amax does not see NaN)
#pragma unroll
    for (int j = 0; j < 8; j += 2) {   // two weights per floating-point instruction
      const float2 w2 = make_float2(v[u][j], v[u][j + 1]);
      const float2 t = __ffma2_rn(w2, lo2, magic2), q = __ffma2_rn(w2, hi2, magic2);
      const uint32_t a0 = __float_as_uint(t.x), a1 = __float_as_uint(t.y);
      sum = __fadd2_rn(sum, t);
      differ |= a0 ^ __float_as_uint(q.x);
      differ |= a1 ^ __float_as_uint(q.y);
      word += a0 << (4 * nibble_pos(j));
      word += a1 << (4 * nibble_pos(j + 1));
    }
    if (!(differ == 0 && amax * inv < 7.4f && sum.x + sum.y < 1e9f)) {
      Eight w8;
#pragma unroll
      for (int j = 0; j < 8; ++j) w8.v[j] = v[u][j];
      word = pack_exact(w8, s32);
    }
    if (i < left) {
      packed[i] = word;
      if ((threadIdx.x & (kLanes - 1)) == 0) scales[i / kLanes] = sh;
    }
  }
}

// One thread per packed word.
__global__ void __launch_bounds__(256) unpack_kernel(const uint32_t* __restrict__ packed, int8_t* __restrict__ q,
                                                     long long words) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < words;
       i += (long long)gridDim.x * blockDim.x) {
    const uint32_t w = packed[i];
    uint32_t lo = 0, hi = 0;  // bytes k0..k3, k4..k7
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const uint32_t b = (((w >> (4 * nibble_pos(o))) & 0xFu) - 8u) & 0xFFu;
      if (o < 4) lo |= b << (8 * o); else hi |= b << (8 * (o - 4));
    }
    reinterpret_cast<uint2*>(q)[i] = make_uint2(lo, hi);
  }
}

__global__ void __launch_bounds__(256) pack_kernel(const int8_t* __restrict__ q, uint32_t* __restrict__ packed,
                                                   long long words) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < words;
       i += (long long)gridDim.x * blockDim.x) {
    const uint2 b = reinterpret_cast<const uint2*>(q)[i];
    uint32_t w = 0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const uint32_t byte = ((o < 4 ? b.x : b.y) >> (8 * (o & 3))) & 0xFFu;
      w |= ((byte + 8u) & 0xFu) << (4 * nibble_pos(o));
    }
    packed[i] = w;
  }
}

// One thread per packed word; writes 8 consecutive outputs.
template <typename OutT>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint32_t* __restrict__ packed,
                                                         const __half* __restrict__ scales, OutT* __restrict__ out,
                                                         int N, int K, int G) {
  const long long words = (long long)N * (K / 8);
  const int wpr = K / 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < words;
       i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / wpr;
    const int j = (int)(i - row * wpr);
    const uint32_t w = packed[i];
    const __half sh = scales[row * (K / G) + (j * 8) / G];
    __align__(16) OutT vals[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const int qv = (int)((w >> (4 * nibble_pos(o))) & 0xFu) - 8;
      if constexpr (sizeof(OutT) == 2) {
        vals[o] = __hmul(__int2half_rn(qv), sh);  // one fp16 multiply, as the reference's fp16 path
      } else {
        vals[o] = __fmul_rn((float)qv, __half2float(sh));
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + row * K + (long long)j * 8);
    const uint4* srcv = reinterpret_cast<const uint4*>(vals);
#pragma unroll
    for (int t = 0; t < (int)(sizeof(OutT) * 8 / 16); ++t) dst[t] = srcv[t];
  }
}

int check_format_args(const void* a, const void* b, int N, int K) {
  if (N < 1 || K < 8 || (K % 8) != 0) return fail(KFB_ERR_INVALID, "need N >= 1 and K a positive multiple of 8, got N=%d K=%d", N, K);
  if (!a || !b) return fail(KFB_ERR_INVALID, "null pointer");
  if (!aligned16(a) || !aligned16(b)) return fail(KFB_ERR_ALIGNMENT, "pointers must be 16-byte aligned");
  return KFB_OK;
}

int grid_for(long long items, int per_block) {
  long long blocks = (items + per_block - 1) / per_block;
  long long cap = (long long)sm_count() * 16;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace
}  // namespace kfb

using namespace kfb;

extern "C" int kfb_quantize_pack(const void* w, int w_dtype, int N, int K, int group, void* packed, void* scales,
                                 void* stream) {
  if (int rc = require_sm100()) return rc;
  if (group != 64 && group != 128) return fail(KFB_ERR_INVALID, "group_size must be one of (64, 128), got %d", group);
  if (N < 1 || K < group || K % group) return fail(KFB_ERR_INVALID, "K=%d is not a multiple of group_size=%d", K, group);
  if (!w || !packed || !scales) return fail(KFB_ERR_INVALID, "null pointer");
  if (!aligned16(w) || !aligned16(packed)) return fail(KFB_ERR_ALIGNMENT, "w and packed must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  const long long words = (long long)N * (K / 8);
  constexpr int kPerCta = kQuantUnroll * kQuantThreads;
  if (words > (1LL << 40)) return fail(KFB_ERR_INVALID, "weight too large");
#define KFB_Q(T, G)                                                                                                          \
  return launch_kernel("quantize_pack_kernel", quantize_pack_kernel<T, G>, dim3((unsigned)((words + kPerCta - 1) / kPerCta)), \
                       dim3(kQuantThreads), 0, s, (const T*)w, (uint32_t*)packed, (__half*)scales, words)
  if (w_dtype == KFB_F32) { if (group == 128) KFB_Q(float, 128); else KFB_Q(float, 64); }
  if (w_dtype == KFB_F16) { if (group == 128) KFB_Q(__half, 128); else KFB_Q(__half, 64); }
  if (w_dtype == KFB_BF16) { if (group == 128) KFB_Q(__nv_bfloat16, 128); else KFB_Q(__nv_bfloat16, 64); }
#undef KFB_Q
  return fail(KFB_ERR_INVALID, "w_dtype must be KFB_F16, KFB_BF16 or KFB_F32");
}

extern "C" int kfb_unpack_int4(const void* packed, int N, int K, void* q_out, void* stream) {
  if (int rc = require_sm100()) return rc;
  if (int rc = check_format_args(packed, q_out, N, K)) return rc;
  const long long words = (long long)N * (K / 8);
  unpack_kernel<<<grid_for(words, 256), 256, 0, (cudaStream_t)stream>>>((const uint32_t*)packed, (int8_t*)q_out, words);
  KFB_LAUNCH_CHECK("unpack_kernel");
  return KFB_OK;
}

extern "C" int kfb_pack_int4(const void* q, int N, int K, void* packed, void* stream) {
  if (int rc = require_sm100()) return rc;
  if (int rc = check_format_args(q, packed, N, K)) return rc;
  const long long words = (long long)N * (K / 8);
  pack_kernel<<<grid_for(words, 256), 256, 0, (cudaStream_t)stream>>>((const int8_t*)q, (uint32_t*)packed, words);
  KFB_LAUNCH_CHECK("pack_kernel");
  return KFB_OK;
}

extern "C" int kfb_dequantize(const void* packed, const void* scales, int N, int K, int group, void* out,
                              int out_dtype, void* stream) {
  if (int rc = require_sm100()) return rc;
  if (int rc = check_format_args(packed, out, N, K)) return rc;
  if (group != 64 && group != 128) return fail(KFB_ERR_INVALID, "group_size must be one of (64, 128), got %d", group);
  if (K % group) return fail(KFB_ERR_INVALID, "K=%d is not a multiple of group_size=%d", K, group);
  if (!scales) return fail(KFB_ERR_INVALID, "null pointer");
  const long long words = (long long)N * (K / 8);
  const int grid = grid_for(words, 256);
  cudaStream_t s = (cudaStream_t)stream;
  if (out_dtype == KFB_F16)
    dequantize_kernel<__half><<<grid, 256, 0, s>>>((const uint32_t*)packed, (const __half*)scales, (__half*)out, N, K, group);
  else if (out_dtype == KFB_F32)
    dequantize_kernel<float><<<grid, 256, 0, s>>>((const uint32_t*)packed, (const __half*)scales, (float*)out, N, K, group);
  else
    return fail(KFB_ERR_INVALID, "out_dtype must be KFB_F16 or KFB_F32");
  KFB_LAUNCH_CHECK("dequantize_kernel");
  return KFB_OK;
}
