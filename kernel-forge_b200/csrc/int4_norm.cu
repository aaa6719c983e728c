// RMSNorm and the INT4 linear behind it as one kernel, for the one or two rows of a small decode step on sm_100a, straight from the
// public packed format:   epilogue(RMSNorm(x) . W^T),  epilogue: + bias, + residual | SiLU(gate) * up | RoPE + cache write.
//
// The kernels of a step run one after the other, each on the result of the one in front, on a few MB of weights: a step is
// bound by the path through each kernel from the moment its activations exist, not by HBM (with every layer of a 22-layer
// model reading the same weights from L2 the step took 532 us instead of 548).  Measured on that path: about 1 us from the
// last store of one kernel to the return of the next one's wait; 1.1 us for load, norm and two barriers; 26 clocks of a
// scheduler per packed word of a warp to unpack (18) and multiply (8).  So:
//   * RMSNorm sits in the prologue: two block barriers here, 1.9 us in a kernel of its own;
//   * all weights of the CTA and their scales are in registers before the wait for the kernel in front (a warp owns NG scale
//     groups of K and 16 RB rows, both known to the compiler: no loop, no address arithmetic between the loads), and with
//     RB = 1 they are unpacked by then;
//   * one CTA per SM where there are more than two blocks of 16 rows for each: a second wave would fetch its weights and
//     normalise after the first one has finished (11264 rows, step of 22 layers: 704 CTAs of one block 583 us, 235 of three
//     561, 141 of five 513).
//   * with RB > 1 the packed nibbles are multiplied as they are, subnormal fp16 numbers, which takes 10 clocks of unpacking per word
//     instead of 18 (unpack_tiny; step of 22 layers 484 us -> 477; the error against 64 bits is the same, 4.41e-4 of a SiLU output).
//     With one row block the product that makes up for the offset costs as much as it saves.  (RB = 5 with groups of 128 takes all
//     128 registers and spills 16 bytes, with NG = 2 groups of 64 32 bytes.)
// Weights staged in shared memory with asynchronous copies instead of registers were slower (+2 us per layer), and so was
// this structure without the norm (o and down projection: int4_small.cu, which has fewer and smaller CTAs there).
// Step of the 22-layer model at batch 1: 593 us with separate norm kernels and the CUDA-core GEMV -> 503.  At batch 2 the step
// with the norms apart on fragment-order copies of qkv and gate_up is the faster one (LlamaInt4Decoder decides).
// The fragment layout and the unpacking are those of int4_small.cu.
#include "common.cuh"
#include "int4_epilogue.cuh"
#include "int4_norm.cuh"

namespace kfb {
namespace normed {
namespace {

constexpr int kMaxWarps = 16, kMaxRB = 5;

__device__ __forceinline__ uint2 load_words(const uint32_t* p) {
  uint2 v;
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// nibble pairs 0..3 of a packed word -> the four half2 (q[2s], q[2s + 1]), exact
__device__ __forceinline__ void unpack(uint32_t w, uint32_t (&q)[4]) {
  const uint32_t h = w >> 8;
  const uint32_t v0 = (w & 0x000F000Fu) | 0x64006400u, v1 = (w & 0x00F000F0u) | 0x54005400u;   // 1024 + u, 64 + u
  const uint32_t v2 = (h & 0x000F000Fu) | 0x64006400u, v3 = (h & 0x00F000F0u) | 0x54005400u;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(q[0]) : "r"(v0), "r"(0x64086408u));   // - 1032
  asm("sub.f16x2 %0, %1, %2;" : "=r"(q[1]) : "r"(v1), "r"(0x54805480u));   // - 72
  asm("sub.f16x2 %0, %1, %2;" : "=r"(q[2]) : "r"(v2), "r"(0x64086408u));
  asm("sub.f16x2 %0, %1, %2;" : "=r"(q[3]) : "r"(v3), "r"(0x54805480u));
}

// The same pairs as subnormal fp16 numbers, u = q + 8 times 2^-24 (s even) or 2^-20 (s odd), exact: no additions.
__device__ __forceinline__ void unpack_tiny(uint32_t w, uint32_t (&q)[4]) {
  const uint32_t h = w >> 8;
  q[0] = w & 0x000F000Fu;
  q[1] = w & 0x00F000F0u;
  q[2] = h & 0x000F000Fu;
  q[3] = h & 0x00F000F0u;
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// One result by the definition, sum over the groups of scale * sum of q * x.  Taking the nibbles as they are is the same for finite
// activations only: u * x - 8 * x is NaN where x is infinite, q * x is infinite with the sign of the product (NaN for q = 0).  So a
// result that is not finite is taken again here, by one thread, from the activations in shared memory.  (Step of 22 layers at batch 1, 512
// keys, with that in the kernel 476.7 us -> 477.9, as a function that is called 480.)
__device__ __forceinline__ float by_definition(const uint32_t* __restrict__ packed, const __half* __restrict__ scales, const __half* x, int groups, int words) {
  float sum = 0.f;
  for (int i = 0; i < groups && sum == sum; ++i) {
    float c = 0.f;
#pragma unroll 1
    for (int w = i * words; w < (i + 1) * words; ++w) {
      const uint32_t word = packed[w];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int q = (int)((word >> (4 * (j >> 1) + 16 * (j & 1))) & 15u) - 8;
        c = fmaf((float)q, __half2float(x[8 * w + j]), c);
      }
    }
    sum = fmaf(__half2float(scales[i]), c, sum);
  }
  return sum;
}

// Shared memory: partial sums [warp][M][16 RB]; sums of squares [M][16]; the normalised activations, rows of K + 8 (the
// fragment reads of eight rows then hit distinct banks).
size_t smem_bytes(int warps, int rb, int M, int K) {
  return ((size_t)warps * M * 16 * rb + (size_t)M * kMaxWarps) * sizeof(float) + (size_t)M * (K + 8) * sizeof(__half);
}

// G: group size; NG: groups of K per warp (K = G * NG * warps); RB: blocks of 16 rows per CTA.
template <int G, int NG, int RB>
__global__ void __launch_bounds__(kMaxWarps * 32, RB == 1 ? 2 : 1)
int4_norm_kernel(const __half* __restrict__ x, const uint32_t* __restrict__ packed, const __half* __restrict__ scales,
                 __half* __restrict__ y, int M, int N, int K, const gemv::Fusion fu) {
  constexpr int H = G / 64;                         // blocks of 64 k per group
  constexpr int kRows = 16 * RB;
  constexpr bool kEarlyUnpack = RB == 1 && NG * G <= 128;
  extern __shared__ __align__(16) float red[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int r0 = blockIdx.x * kRows;
  const int KW = K / 8, SG = K / G;
  float* part = red + warps * M * kRows;
  __half* hx = reinterpret_cast<__half*>(part + M * kMaxWarps);

  // ---- before the wait: whatever does not depend on the kernel in front
  const __half* norm_w = fu.norm_w;
  if (!fu.early) pdl_wait(x, packed, scales, norm_w);   // (early: the weights are older than it)
  uint2 wv[RB][2][NG][H];
  __half sv[RB][2][NG];
#pragma unroll
  for (int rb = 0; rb < RB; ++rb)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = min(r0 + 16 * rb + 8 * h + g, N - 1);   // rows past N: a valid row, never stored
      const uint32_t* w = packed + (size_t)row * KW + warp * (NG * G / 8) + 2 * t;
      const __half* s = scales + (size_t)row * SG + warp * NG;
#pragma unroll
      for (int i = 0; i < NG; ++i) {
#pragma unroll
        for (int b = 0; b < H; ++b) wv[rb][h][i][b] = load_words(w + i * (G / 8) + b * 8);
        sv[rb][h][i] = s[i];
      }
    }
  uint32_t early[kEarlyUnpack ? H : 1][4][4];       // [64 k][word][pair]
  if constexpr (kEarlyUnpack) {
#pragma unroll
    for (int b = 0; b < H; ++b) {
      unpack(wv[0][0][0][b].x, early[b][0]);
      unpack(wv[0][1][0][b].x, early[b][1]);
      unpack(wv[0][0][0][b].y, early[b][2]);
      unpack(wv[0][1][0][b].y, early[b][3]);
    }
  }
  const int pieces = K / 8;                         // 16-byte pieces of a row of activations: at most two per thread
  const int c0 = threadIdx.x, c1 = threadIdx.x + blockDim.x;
  const uint4* nw = reinterpret_cast<const uint4*>(norm_w);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4 w0 = c0 < pieces ? nw[c0] : zero, w1 = c1 < pieces ? nw[c1] : zero;
  const float inv_k = 1.0f / (float)K;
  for (int i = threadIdx.x; i < M * kMaxWarps; i += blockDim.x) part[i] = 0.f;
  __syncthreads();
  if (fu.early) pdl_wait(x);
  pdl_launch_dependents();

  // ---- RMSNorm of the rows, every CTA for itself
  long long pos = -1;   // RoPE: the angles of this position are on their way while the product is computed
  if (fu.epi == gemv::kEpiRopeKv && threadIdx.x < kRows / 2) pos = fu.rope.pos[0];
  uint4 a = zero, b = zero;                         // row 0 stays in registers, the others wait in shared memory
#pragma unroll 2
  for (int m = M - 1; m >= 0; --m) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)m * K);
    if (c0 < pieces) a = xr[c0];
    if (c1 < pieces) b = xr[c1];
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = __half22float2(reinterpret_cast<const __half2*>(&a)[e]);
      const float2 f1 = __half22float2(reinterpret_cast<const __half2*>(&b)[e]);
      ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
      ss = fmaf(f1.x, f1.x, fmaf(f1.y, f1.y, ss));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    if (lane == 0) part[m * kMaxWarps + warp] = ss;
    if (m > 0) {
      uint4* hr = reinterpret_cast<uint4*>(hx + m * (K + 8));
      if (c0 < pieces) hr[c0] = a;
      if (c1 < pieces) hr[c1] = b;
    }
  }
  __syncthreads();
  if (pos >= 0 && pos < fu.rope.Lmax) {
    const size_t at = pos * fu.rope.D + ((r0 >> 1) + threadIdx.x) % (fu.rope.D / 2);   // (of a q or k head; harmless for v)
    asm volatile("prefetch.global.L1 [%0];" ::"l"(fu.rope.cos_t + at));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(fu.rope.sin_t + at));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(fu.rope.cos_t + at + fu.rope.D / 2));
    asm volatile("prefetch.global.L1 [%0];" ::"l"(fu.rope.sin_t + at + fu.rope.D / 2));
  }
  for (int m = 0; m < M; ++m) {
    const float4* pm = reinterpret_cast<const float4*>(part + m * kMaxWarps);
    float tot = 0.f;
#pragma unroll
    for (int q = 0; q < kMaxWarps / 4; ++q) tot += (pm[q].x + pm[q].y) + (pm[q].z + pm[q].w);
    const float inv = rsqrtf(tot * inv_k + fu.eps);
    uint4* hr = reinterpret_cast<uint4*>(hx + m * (K + 8));
    auto scaled = [&](uint4 v, const uint4& w) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        __half2& p = reinterpret_cast<__half2*>(&v)[e];
        const float2 f = __half22float2(p);
        p = __hmul2(__floats2half2_rn(f.x * inv, f.y * inv), reinterpret_cast<const __half2*>(&w)[e]);
      }
      return v;
    };
    if (c0 < pieces) hr[c0] = scaled(m == 0 ? a : hr[c0], w0);
    if (c1 < pieces) hr[c1] = scaled(m == 0 ? b : hr[c1], w1);
  }
  __syncthreads();

  // ---- the product; fragment columns past M repeat row M - 1 and are never stored
  const __half* xs = hx + min(g, M - 1) * (K + 8) + warp * (NG * G) + 16 * t;
  float acc[RB][4];
#pragma unroll
  for (int i = 0; i < NG; ++i) {
    uint4 xv[H][2];
#pragma unroll
    for (int b = 0; b < H; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) xv[b][e] = *reinterpret_cast<const uint4*>(xs + i * G + b * 64 + e * 8);
    // With several row blocks the unpacking is what a scheduler spends its time on; there the nibbles go into the product as they
    // are (unpack_tiny), and what that is too large by, 8 times the sum of the group's activations, is what the sums start with:
    // a product with a constant, once for all row blocks.  Even and odd pairs have a sum each, which differ by 2^4.
    float start[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (RB > 1) {
      constexpr uint32_t kMinusEight = 0x80088008u;   // -8 * 2^-24, twice
#pragma unroll
      for (int b = 0; b < H; ++b)
#pragma unroll
        for (int s = 0; s < 4; ++s)
          mma16816(start, kMinusEight, kMinusEight, kMinusEight, kMinusEight, reinterpret_cast<const uint32_t*>(&xv[b][0])[s],
                   reinterpret_cast<const uint32_t*>(&xv[b][1])[s]);
    }
#pragma unroll
    for (int rb = 0; rb < RB; ++rb) {
      float c[2][4] = {{start[0], start[1], start[2], start[3]}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int b = 0; b < H; ++b) {
        uint32_t q[4][4];
        if constexpr (!kEarlyUnpack) {
          auto take = [](uint32_t w, uint32_t (&to)[4]) {
            if constexpr (RB > 1) unpack_tiny(w, to);
            else unpack(w, to);
          };
          take(wv[rb][0][i][b].x, q[0]);
          take(wv[rb][1][i][b].x, q[1]);
          take(wv[rb][0][i][b].y, q[2]);
          take(wv[rb][1][i][b].y, q[3]);
        }
        const uint32_t (&u)[4][4] = kEarlyUnpack ? early[kEarlyUnpack ? b : 0] : q;
#pragma unroll
        for (int s = 0; s < 4; ++s)
          mma16816(c[RB > 1 ? s & 1 : 0], u[0][s], u[1][s], u[2][s], u[3][s], reinterpret_cast<const uint32_t*>(&xv[b][0])[s],
                   reinterpret_cast<const uint32_t*>(&xv[b][1])[s]);
      }
      constexpr float kUnit = RB > 1 ? 16777216.0f : 1.0f;
      const float s0 = __half2float(sv[rb][0][i]) * kUnit, s1 = __half2float(sv[rb][1][i]) * kUnit;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float v = RB > 1 ? fmaf(c[1][e], 0.0625f, c[0][e]) : c[0][e];
        acc[rb][e] = i == 0 ? (e < 2 ? s0 : s1) * v : fmaf(e < 2 ? s0 : s1, v, acc[rb][e]);
      }
    }
  }

  // ---- sum over the warps, in order
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if (2 * t + e < M) {
      float* mine = red + (warp * M + 2 * t + e) * kRows + g;
#pragma unroll
      for (int rb = 0; rb < RB; ++rb) {
        mine[16 * rb] = acc[rb][e];
        mine[16 * rb + 8] = acc[rb][2 + e];
      }
    }
  __syncthreads();
  constexpr int kPairs = kRows / 2;
  for (int idx = threadIdx.x; idx < M * kPairs; idx += blockDim.x) {
    const int m = idx / kPairs, pr = idx % kPairs;
    const int n = r0 + 2 * pr;
    if (n >= N) continue;
    float v0 = 0.f, v1 = 0.f;
    const float* at = red + m * kRows + 2 * pr;
#pragma unroll 8
    for (int k = 0; k < warps; ++k) {
      const float2 o = *reinterpret_cast<const float2*>(at + k * M * kRows);
      v0 += o.x;
      v1 += o.y;
    }
    if constexpr (RB > 1) {
      auto again = [&](int row) { return by_definition(packed + (size_t)row * KW, scales + (size_t)row * SG, hx + m * (K + 8), SG, G / 8); };
      if (!(fabsf(v0) < INFINITY)) v0 = again(n);
      if (!(fabsf(v1) < INFINITY)) v1 = again(min(n + 1, N - 1));
    }
    switch (fu.epi) {   // uniform over the grid
      case gemv::kEpiSiluPair: gemv::store_pair<gemv::kEpiSiluPair>(v0, v1, fu, y, m, n, N); break;
      case gemv::kEpiRopeKv: gemv::store_pair<gemv::kEpiRopeKv>(v0, v1, fu, y, m, n, N); break;
      default: gemv::store_pair<gemv::kEpiNone>(v0, v1, fu, y, m, n, N);
    }
  }
}

template <int G, int NG, int RB>
int launch(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K, cudaStream_t stream, const gemv::Fusion& fu) {
  const int warps = K / (G * NG);
  return launch_kernel("int4_norm_kernel", int4_norm_kernel<G, NG, RB>, dim3(ceil_div(N, 16 * RB)), dim3(warps * 32),
                       smem_bytes(warps, RB, M, K), stream, (const __half*)x, (const uint32_t*)packed, (const __half*)scales, (__half*)y, M,
                       N, K, fu);
}

// Groups per warp: the smallest share that divides K into at most 16 warps.
int groups_per_warp(int sg) {
  for (int ng = 1; ng <= 4; ++ng)
    if (sg % ng == 0 && sg / ng <= kMaxWarps) return ng;
  return 0;
}

// Blocks of 16 rows per CTA (see above).
int row_blocks(int N) {
  const int blocks = ceil_div(N, 16), sms = sm_count();
  return blocks <= 2 * sms ? 1 : ceil_div(blocks, sms) < kMaxRB ? ceil_div(blocks, sms) : kMaxRB;
}

}  // namespace

// Up to 128 k per warp (K <= 2048) every N that keeps the SMs busy; up to 256 k only where one block of rows per CTA is enough:
// with more the weights do not fit in the registers.  A CTA per SM and five blocks per CTA are one wave; a second one that is
// half empty costs more than the norm kernels and launches saved (step of 8 layers at batch 1, us, this kernel / separate norms:
// gate_up of 11264 rows 201 / 224, 13824 238 / 229, 16384 245 / 224, 17920 237 / 226, 22016 276 / 291).
bool fits(int M, int N, int K, int group) {
  const int ng = groups_per_warp(K / group);
  if (M < 1 || M > 2 || N < 1 || ng == 0 || ng * group > 256) return false;
  const int warps = K / (group * ng), rb = row_blocks(N);
  const long long wave = (long long)kMaxRB * sm_count(), blocks = ceil_div(N, 16), waves = (blocks + wave - 1) / wave;
  if (waves > 1 && blocks * 100 < waves * wave * 85) return false;
  return (rb == 1 || ng * group <= 128) && K / 8 <= 2 * warps * 32 && smem_bytes(warps, rb, M, K) <= 48 * 1024;
}

int run(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K, int group, cudaStream_t stream,
        const gemv::Fusion& given) {
  gemv::Fusion fu = given;
  fu.early = given.early || constants_are_old();
  const int ng = groups_per_warp(K / group), rb = row_blocks(N);
#define KFB_NORM(G, NG, RB) \
  if (group == G && ng == NG && rb == RB) return launch<G, NG, RB>(x, packed, scales, y, M, N, K, stream, fu)
#define KFB_NORM_RB(G, NG) KFB_NORM(G, NG, 1); KFB_NORM(G, NG, 3); KFB_NORM(G, NG, 4); KFB_NORM(G, NG, 5)
  KFB_NORM_RB(128, 1);
  KFB_NORM(128, 2, 1);
  KFB_NORM_RB(64, 1);
  KFB_NORM_RB(64, 2);
  KFB_NORM(64, 3, 1);
  KFB_NORM(64, 4, 1);
#undef KFB_NORM_RB
#undef KFB_NORM
  return fail(KFB_ERR_UNSUPPORTED, "no RMSNorm + INT4 kernel for N=%d K=%d group=%d", N, K, group);
}

}  // namespace normed
}  // namespace kfb
