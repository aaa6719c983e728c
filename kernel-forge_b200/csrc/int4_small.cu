// INT4 linear for small batches (M <= 32) on sm_100a, straight from the public packed format.
//
// Replaces the small-M side of the reference's dispatcher (csrc/gemm/dequant_gemv_kernel.cuh:38-109 up to M = 7, and the
// 64-row tiles of dequant_gemm_tc_kernel.cuh above).  At these sizes the product is bound by latency and by what the
// SMs keep in flight, not by HBM: 0.5 bytes per weight are read once.  So the kernel has nothing between a load and
// its use -- no shared-memory tile, no barrier before the products:
//
//   * A CTA owns 16 * RB rows; its KS warps split K in scale groups.  A warp requests its weights (kDepth groups at a
//     time) and multiplies them straight from registers; one shared-memory reduction over the warps, in order, ends it.
//   * K is walked in blocks of 64.  Of each row of a block, lane t of the four lanes of an MMA fragment row reads two
//     consecutive words, 16 k (a warp reads 32 contiguous bytes of each of 16 rows: whole sectors).  A dot product may
//     visit k in any order as long as both operands agree, so the lane multiplies nibble pair s of its two words
//     (fragment columns 2t, 2t + 1 and 2t + 8, 2t + 9) with the activations of the same k, which are 32 contiguous bytes
//     of the activation row.  (16 bytes of weights and 64 of activations per lane instead needs twice as many L1 lines
//     per activation load: 1536 x 8960, M = 16 9.0 us against 7.4.)
//   * Nibbles become exact integers q in fp16 (1024 + u or 1024 + 16 u through the magic number, one subtraction or
//     fused multiply-add) or bf16 (128 + u, one subtraction); mma.sync m16n8k16 accumulates a group in FP32, the scale
//     is applied in FP32 once per group, the result is rounded once.  The batch is the N = 8 of the MMA.
//
// Measured (graph of L2-cold calls, us; TMA / shared-memory kernels of int4_gemv_mma.cuh or the tcgen05 GEMM, whichever
// was faster -> this kernel):  5632 x 2048 M = 8 8.6 -> 5.5, M = 16 12.4 -> 5.9, M = 32 14.5 -> 10.1;  2048 x 5632 9.5 ->
// 4.8, 11.3 -> 5.6, 11.9 -> 7.4;  1536 x 8960 12.1 -> 6.3, 12.2 -> 7.3, 12.8 -> 10.1;  8960 x 1536 7.7 -> 5.1, 11.5 -> 6.2,
// 16.0 -> 9.1.
// Also built: activations staged in shared memory, K split over a cluster of CTAs and added up through distributed shared
// memory.  It reads fewer activation bytes, but the staging, two cluster barriers and the cluster launch cost 2-3 us:
// 5632 x 2048 M = 8 6.9 us, 1536 x 8960 M = 16 10.2 us.
#include "common.cuh"
#include "int4_epilogue.cuh"
#include "int4_small.cuh"

namespace kfb {
namespace small {
namespace {

template <int W>
struct Words {
  uint32_t w[W];
};
__device__ __forceinline__ void load_words(Words<4>& d, const uint32_t* p) {
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(d.w[0]), "=r"(d.w[1]) : "l"(p));
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(d.w[2]), "=r"(d.w[3]) : "l"(p + 8));
}
__device__ __forceinline__ void load_words(Words<2>& d, const uint32_t* p) {
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(d.w[0]), "=r"(d.w[1]) : "l"(p));
}

template <bool kBf16>
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

// nibble pairs 0..3 of a packed word -> the four half2 / bfloat162 (q[2s], q[2s + 1]), exact
template <bool kBf16>
__device__ __forceinline__ void unpack(uint32_t w, uint32_t (&q)[4]) {
  if constexpr (kBf16) {
    const __nv_bfloat162 k136 = __halves2bfloat162(__ushort_as_bfloat16(0x4308), __ushort_as_bfloat16(0x4308));
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      uint32_t v = ((w >> (4 * s)) & 0x000F000Fu) | 0x43004300u;   // (128 + u, 128 + u')
      __nv_bfloat162 b = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&v), k136);
      q[s] = *reinterpret_cast<uint32_t*>(&b);
    }
  } else {
    const uint32_t h = w >> 8;
    uint32_t v0 = (w & 0x000F000Fu) | 0x64006400u, v1 = (w & 0x00F000F0u) | 0x64006400u;   // 1024 + u, 1024 + 16 u
    uint32_t v2 = (h & 0x000F000Fu) | 0x64006400u, v3 = (h & 0x00F000F0u) | 0x64006400u;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(q[0]) : "r"(v0), "r"(0x64086408u));
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(q[1]) : "r"(v1), "r"(0x2C002C00u), "r"(0xD480D480u));   // v / 16 - 72
    asm("sub.f16x2 %0, %1, %2;" : "=r"(q[2]) : "r"(v2), "r"(0x64086408u));
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(q[3]) : "r"(v3), "r"(0x2C002C00u), "r"(0xD480D480u));
  }
}

// Rows n, n + 1 (n even) of batch column m.
template <bool kBf16>
__device__ __forceinline__ void store_rows(float a0, float a1, const gemv::Fusion& fu, uint16_t* __restrict__ y, int m, int n, int N) {
  if constexpr (kBf16) {
    const __nv_bfloat16* bias = reinterpret_cast<const __nv_bfloat16*>(fu.bias);
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(y) + (size_t)m * N + n;
    auto fin = [&](float v, int r) {
      const __nv_bfloat16 b = __float2bfloat16_rn(v);
      return bias ? __float2bfloat16_rn(__bfloat162float(b) + __bfloat162float(bias[r])) : b;
    };
    out[0] = fin(a0, n);
    if (n + 1 < N) out[1] = fin(a1, n + 1);
  } else {
    __half* out = reinterpret_cast<__half*>(y);
    switch (fu.epi) {   // uniform over the grid
      case gemv::kEpiSiluPair: gemv::store_pair<gemv::kEpiSiluPair>(a0, a1, fu, out, m, n, N); break;
      case gemv::kEpiRopeKv: gemv::store_pair<gemv::kEpiRopeKv>(a0, a1, fu, out, m, n, N); break;
      default:
        if ((N & 1) == 0 && (reinterpret_cast<uintptr_t>(y) & 3u) == 0) {   // one 4-byte store (n + 1 < N then)
          *reinterpret_cast<__half2*>(out + (size_t)m * N + n) =
              __halves2half2(gemv::finish(a0, fu, m, n, N), gemv::finish(a1, fu, m, n + 1, N));
        } else {
          gemv::store_pair<gemv::kEpiNone>(a0, a1, fu, out, m, n, N);
        }
    }
  }
}

// Resident CTAs per SM.  Registers decide it: the more column blocks, the fewer CTAs.
template <int KS, int RB, int MB>
constexpr int min_blocks() { return KS == 16 ? 1 : RB * MB == 1 ? 4 : RB == 1 && MB == 2 ? 3 : 2; }

// G: group size; KS: warps of a CTA = shares of K; RB: 16-row blocks per warp; MB: blocks of 8 batch columns; kHalves: see run.
template <int G, int KS, int RB, int MB, bool kBf16, bool kHalves>
__global__ void __launch_bounds__(KS * 32, min_blocks<KS, RB, MB>())
int4_small_kernel(const uint16_t* __restrict__ x, const uint32_t* __restrict__ packed, const __half* __restrict__ scales,
                  uint16_t* __restrict__ y, int M, int N, int K, const gemv::Fusion fu) {
  static_assert(!kHalves || G == 128, "a group of 64 is a block of 64");
  constexpr int U = kHalves ? 64 : G;               // K is walked in scale groups, or in blocks of 64
  constexpr int W = U / 32;                         // packed words per lane, row and unit; and 16-byte pieces of x
  constexpr int kDepth = (KS == 16 && MB == 1 ? 4 : 2) * (128 / U);   // units a warp keeps in flight
  constexpr int kRows = 16 * RB, kPad = kRows + 4;
  extern __shared__ float red[];                    // [warp][8 MB][kPad]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int warps = KS;
  const int g = lane >> 2, t = lane & 3;
  const int r0 = blockIdx.x * kRows;
  const int SG = K / G, KW = K / 8;
  const int units = K / U, g0 = (int)((long long)units * warp / warps), g1 = (int)((long long)units * (warp + 1) / warps);   // of this warp

  if (!fu.early) pdl_wait(x, packed, scales);   // (early: the weights are older than the kernel in front)
  const uint32_t* wrow[RB][2];
  const __half* srow[RB][2];
#pragma unroll
  for (int rb = 0; rb < RB; ++rb)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = min(r0 + 16 * rb + 8 * h + g, N - 1);   // rows past N: a valid row, never stored
      wrow[rb][h] = packed + (size_t)row * KW + 2 * t;
      srow[rb][h] = scales + (size_t)row * SG;
    }
  Words<W> wbuf[kDepth][RB][2];
  float sbuf[kDepth][RB][2];
  auto fetch = [&](int slot, int gi) {
    if (gi < g1) {
#pragma unroll
      for (int rb = 0; rb < RB; ++rb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          load_words(wbuf[slot][rb][h], wrow[rb][h] + (size_t)gi * (U / 8));
          sbuf[slot][rb][h] = __half2float(srow[rb][h][gi / (G / U)]);
        }
    }
  };

#pragma unroll
  for (int d = 0; d < kDepth; ++d) fetch(d, g0 + d);
  if (fu.early) pdl_wait(x);
  pdl_launch_dependents();
  if (!kBf16 && fu.residual != nullptr && threadIdx.x < M)   // what the epilogue adds: on its way while the product is computed
    asm volatile("prefetch.global.L1 [%0];" ::"l"(fu.residual + (size_t)threadIdx.x * N + r0));

  float acc[RB][MB][4];
#pragma unroll
  for (int rb = 0; rb < RB; ++rb)
#pragma unroll
    for (int j = 0; j < MB; ++j) acc[rb][j][0] = acc[rb][j][1] = acc[rb][j][2] = acc[rb][j][3] = 0.f;

  const uint16_t* xrow = x + (size_t)g * K + 16 * t;   // batch row 8 j + g of column block j
  auto group_product = [&](int slot, int gi) {
    uint4 xv[MB][W];
#pragma unroll
    for (int j = 0; j < MB; ++j) {
      const bool real = 8 * j + g < M;
      const uint4* p = reinterpret_cast<const uint4*>(xrow + (size_t)(8 * j) * K + (size_t)gi * U);
#pragma unroll
      for (int i = 0; i < W; ++i) xv[j][i] = real ? p[(i >> 1) * 8 + (i & 1)] : make_uint4(0u, 0u, 0u, 0u);
    }
    float c[RB][MB][4];
#pragma unroll
    for (int rb = 0; rb < RB; ++rb)
#pragma unroll
      for (int j = 0; j < MB; ++j) c[rb][j][0] = c[rb][j][1] = c[rb][j][2] = c[rb][j][3] = 0.f;
#pragma unroll
    for (int i = 0; i < W; i += 2)
#pragma unroll
      for (int rb = 0; rb < RB; ++rb) {
        uint32_t a0[4], a1[4], a2[4], a3[4];
        unpack<kBf16>(wbuf[slot][rb][0].w[i], a0);
        unpack<kBf16>(wbuf[slot][rb][1].w[i], a1);
        unpack<kBf16>(wbuf[slot][rb][0].w[i + 1], a2);
        unpack<kBf16>(wbuf[slot][rb][1].w[i + 1], a3);
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
          for (int j = 0; j < MB; ++j)
            mma16816<kBf16>(c[rb][j], a0[s], a1[s], a2[s], a3[s], reinterpret_cast<const uint32_t*>(&xv[j][i])[s],
                            reinterpret_cast<const uint32_t*>(&xv[j][i + 1])[s]);
      }
#pragma unroll
    for (int rb = 0; rb < RB; ++rb)
#pragma unroll
      for (int j = 0; j < MB; ++j) {
        acc[rb][j][0] = fmaf(sbuf[slot][rb][0], c[rb][j][0], acc[rb][j][0]);
        acc[rb][j][1] = fmaf(sbuf[slot][rb][0], c[rb][j][1], acc[rb][j][1]);
        acc[rb][j][2] = fmaf(sbuf[slot][rb][1], c[rb][j][2], acc[rb][j][2]);
        acc[rb][j][3] = fmaf(sbuf[slot][rb][1], c[rb][j][3], acc[rb][j][3]);
      }
  };
  for (int gi = g0; gi < g1; gi += kDepth) {
#pragma unroll
    for (int d = 0; d < kDepth; ++d)
      if (gi + d < g1) {
        group_product(d, gi + d);
        fetch(d, gi + d + kDepth);
      }
  }

  // ---- sum over the warps, in order
  {
    float* mine = red + (size_t)warp * (8 * MB) * kPad;
#pragma unroll
    for (int rb = 0; rb < RB; ++rb)
#pragma unroll
      for (int j = 0; j < MB; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) mine[(8 * j + 2 * t + (e & 1)) * kPad + 16 * rb + g + 8 * (e >> 1)] = acc[rb][j][e];
  }
  __syncthreads();
  constexpr int kPairs = kRows / 2;
  for (int idx = threadIdx.x; idx < M * kPairs; idx += KS * 32) {
    const int m = idx / kPairs, pr = idx % kPairs;
    const int n = r0 + 2 * pr;
    if (n >= N) continue;
    float v0 = 0.f, v1 = 0.f;
    const float* at = red + m * kPad + 2 * pr;
#pragma unroll 8
    for (int k = 0; k < warps; ++k) {
      const float2 o = *reinterpret_cast<const float2*>(at + (size_t)k * (8 * MB) * kPad);
      v0 += o.x;
      v1 += o.y;
    }
    store_rows<kBf16>(v0, v1, fu, y, m, n, N);
  }
}

template <int G, int KS, int RB, int MB, bool kBf16, bool kHalves = false>
int launch(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K,
           cudaStream_t stream, const gemv::Fusion& fu) {
  auto kernel = int4_small_kernel<G, KS, RB, MB, kBf16, kHalves>;
  constexpr size_t smem = (size_t)KS * (8 * MB) * (16 * RB + 4) * sizeof(float);
  static_assert(smem <= 48 * 1024, "no opt-in for more shared memory is made");
  return launch_kernel("int4_small_kernel", kernel, dim3(ceil_div(N, 16 * RB)), dim3(KS * 32), smem, stream,
                       (const uint16_t*)x, (const uint32_t*)packed, (const __half*)scales, (uint16_t*)y, M, N, K, fu);
}

}  // namespace

int run(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K, int group, bool bf16, cudaStream_t stream,
        const gemv::Fusion& given) {
  gemv::Fusion fu = given;
  fu.early = given.early || constants_are_old();
  // Few row blocks (at most one CTA per SM) and a long K: 16 shares of K instead of 8, so that a warp has half as many
  // groups one after the other (2048 x 5632, M = 8: 5.3 us against 6.1; at K = 2048 there is nothing to gain).
  // 9 <= M <= 16 and more row blocks than the three CTAs per SM hold: two row blocks per warp share the activations
  // (8960 x 1536, M = 16: 6.2 us against 9.0, which takes a second, nearly empty wave).
  const int row_blocks = ceil_div(N, 16), sms = sm_count();
  const bool long_k = row_blocks <= sms && K >= 4096;
  const bool two_rows = M > 8 && M <= 16 && row_blocks > 3 * sms;
  // Above M = 16 the activations of a group of 128 take 64 registers, which costs a resident CTA and loads in flight: with more than 48
  // row blocks K is walked in blocks of 64 (us, M = 19, 5824 x 1920 9.1 -> 7.5; M = 22, 6464 x 1536 bf16 9.1 -> 7.0; M = 23, 1600 x
  // 1792 4.7 -> 4.1; step of the 22-layer model at batch 32 952 -> 921).  Fewer row blocks (M = 22, 371 x 1792 3.8 and 3.9; M = 29, 512
  // x 2560 4.8 and 4.9) and smaller M (M = 16, 1536 x 8960 6.8 and 7.5; M = 4, 1216 x 2688 3.5 and 4.0) gain nothing from it.
  const bool halves = group == 128 && row_blocks > 48;
#define KFB_SMALL(G, ...) return launch<G, __VA_ARGS__>(x, packed, scales, y, M, N, K, stream, fu)
#define KFB_SMALL_KS(G, BF)                                                            \
  {                                                                                    \
    if (two_rows) KFB_SMALL(G, 8, 2, 2, BF);                                           \
    if (M <= 8) { if (long_k) KFB_SMALL(G, 16, 1, 1, BF); KFB_SMALL(G, 8, 1, 1, BF); } \
    if (M <= 16) { if (long_k) KFB_SMALL(G, 16, 1, 2, BF); KFB_SMALL(G, 8, 1, 2, BF); } \
    constexpr bool kHalves = G == 128;                                                 \
    if (long_k && halves) KFB_SMALL(G, 16, 1, 4, BF, kHalves);                         \
    if (halves) KFB_SMALL(G, 8, 1, 4, BF, kHalves);                                    \
    if (long_k) KFB_SMALL(G, 16, 1, 4, BF);                                            \
    KFB_SMALL(G, 8, 1, 4, BF);                                                         \
  }
  if (group == 128) { if (bf16) KFB_SMALL_KS(128, true) else KFB_SMALL_KS(128, false) }
  if (bf16) KFB_SMALL_KS(64, true) else KFB_SMALL_KS(64, false)
#undef KFB_SMALL_KS
#undef KFB_SMALL
}

}  // namespace small
}  // namespace kfb
