// INT4 weight-only GEMM for sm_100a:  y[M, N] = x[M, K] @ W_hat[N, K]^T, any M, any N.
//
// Replaces dequant_gemm_tc_kernel + splitk_reduce of the reference
// (csrc/gemm/dequant_gemm_tc_kernel.cuh:55-162: mma.sync, 64x64 tiles, cp.async, N % 64 == 0).
//
// The product is computed transposed, y^T = W_hat x^T: weight rows are the M of tcgen05.mma, the batch is its N.  A
// persistent kernel of CTA pairs (clusters of two, cta_group::2): a pair owns 256 weight rows x `mt` batch rows
// (32 .. 256, chosen per call) of one K range.  Each CTA
//   * brings its own 128 rows of packed words (TMA, two K blocks of 128 per copy) and HALF of the batch rows of the
//     activation tile (TMA, 128-byte swizzle); the tensor cores of both read both halves;
//   * dequantises its weight rows from registers straight into TENSOR MEMORY, the A operand of the MMA: one thread per
//     row, exact q, one fp16 multiply by the group scale = the reference's fp16(q*s)
//     (dequant_gemm_tc_kernel.cuh:100-112).  TMEM holds a ring of 4 K blocks (256 columns) next to the accumulator;
//   * keeps 128 rows of the accumulator in its own TMEM and writes them: TMEM -> registers (which frees the accumulator
//     for the next tile) -> pairs of neighbouring features exchanged between lanes -> rows of y.
// What bounds it: the tensor pipe at large M (4 mt clocks per K block of 128), the dequantisation when mt is small.  Why pairs and TMEM operands: with one CTA per 128 x 256 tile and the dequantised
// tile in shared memory, every 64 k moved 36 KB from L2 and wrote and re-read 16 KB of weights in shared memory; L2 ->
// SM traffic was the limit at ~45 % of the tensor peak.  Here it is 20 KB per 64 k, and no dequantised weight
// touches shared memory.
//
// Warps of a CTA: 0-7 dequantise, 8-15 epilogue, 16 TMA producer, 17 MMA issuer (leader CTA only).
// Split-K partial sums are reduced in split order by a second kernel (deterministic).
// Rows past N and batch rows past M are zero-filled by TMA and never stored.
#include "common.cuh"
#include "int4_gemm.cuh"
#include "sm100.cuh"

namespace kfb {
namespace gemm {
namespace {

using namespace sm100;

constexpr int kPairRows = 256;   // weight rows of a pair's tile (MMA M); 128 per CTA
constexpr int kRows = 128;
constexpr int kBlockK = 128;     // k per pipeline stage: two 64-wide (128-byte) swizzled activation tiles
constexpr int kMaxTile = 256;    // most batch rows of a tile (MMA N)
constexpr int kStages = 4;       // K blocks of dequantised weights in TMEM
constexpr int kMaxXStages = 16;  // K blocks of activations in shared memory: as many as fit (4 at 256 batch rows per tile)
constexpr int kMaxSplits = 16;   // of K
constexpr int kWordStages = 4;   // copies of packed words in flight, two K blocks each
constexpr int kDequantGroups = 2;  // warpgroups; they take the K blocks in turn
constexpr int kDequantWarps = 4 * kDequantGroups, kEpilogueWarps = 8;
constexpr int kProducerWarp = kDequantWarps + kEpilogueWarps;
constexpr int kMmaWarp = kProducerWarp + 1;
constexpr int kThreads = (kProducerWarp + 4) * 32;   // whole warpgroups: registers move between them
// Registers per thread: 640 x 96 at launch; the epilogue keeps a row of the accumulator, rounded, in registers.
constexpr int kRegsLaunch = 96, kRegsDequant = 88, kRegsEpilogue = 128, kRegsMisc = 40;
static_assert(kDequantWarps * kRegsDequant + kEpilogueWarps * kRegsEpilogue + 4 * kRegsMisc <= kThreads / 32 * kRegsLaunch,
              "setmaxnreg.inc only takes what the block was launched with");
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColA = 256;  // 4 stages x 64 columns; the accumulator (or two of <= 128 columns) lies below

// shared memory
constexpr int kWordBytes = kRows * 128;                       // 128 rows x 32 words
constexpr int kXRing = 128 * 1024;                            // the activation ring; a K block takes mt / 2 rows x 256 bytes
constexpr int kOffX = kWordStages * kWordBytes;
constexpr int kOffBars = kOffX + kXRing;
constexpr int kNumBars = 2 * kWordStages + 2 * kMaxXStages + 2 * kStages + 4;
constexpr int kOffMisc = kOffBars + kNumBars * 8;
constexpr int kSmem = kOffMisc + 16 + 1024;                   // + alignment of the tiles to 1024 bytes
static_assert(kSmem <= 227 * 1024, "must fit in shared memory");

enum WaitCode : uint32_t { kWaitFree = 0x301, kWaitWords, kWaitX, kWaitAReady, kWaitAcc, kWaitAccFree, kWaitWordsFree, kWaitAFree };

// Where the 16-bit result goes.  Plain call: one buffer [M, N].  Output-feature-sharded call (fused
// all-gather): `count` buffers [M, ld], one per GPU of the group (peer-mapped device pointers, this
// GPU's own buffer included); this rank's N columns are stored at column `col0` of EVERY buffer with
// plain peer stores from the epilogue, so the gather overlaps the computation tile by tile and no
// separate collective kernel runs.  (Stores only: no load ever targets a peer's memory.)
constexpr int kMaxPeers = 8;
struct OutSpec {
  __half* y[kMaxPeers];
  int count;
  int ld;    // row stride of every buffer, in elements
  int col0;  // first column this rank writes
  int bf16;  // the buffers hold bf16 instead of fp16 (the 16-bit stores are the same)
  const uint16_t* bias;  // [N] of the output type or nullptr: added to the rounded product, rounded again (as `y + bias`)
  int silu;  // fp16: features 2j, 2j + 1 are gate and up of one; the buffers hold [M, N / 2] = fp16(fp16(silu(gate)) * up)
};

__device__ __forceinline__ uint16_t silu_pair(uint32_t gate_up) {
  const __half2 h = *reinterpret_cast<const __half2*>(&gate_up);
  const float g = __low2float(h);
  const __half a = __hmul(__float2half_rn(g / (1.0f + __expf(-g))), __high2half(h));
  return *reinterpret_cast<const uint16_t*>(&a);
}


struct Shape {
  int M, N, K, group;
  int mt;                          // batch rows per tile: a multiple of 32, <= 256
  int m_tiles, n_tiles, splits;
  int kblocks_per_split;           // a multiple of 2 (whole copies of packed words)
};

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// 8 packed weights -> 4 half2 of fp16(q * s) in k order
__device__ __forceinline__ uint4 dequant8(uint32_t w, __half2 s2) {
  constexpr uint32_t kMagic = 0x64006400u;
  const __half2 k1032 = u32_as_h2(0x64086408u);
  const __half2 kSixteenth = u32_as_h2(0x2C002C00u);
  const __half2 kMinus72 = u32_as_h2(0xD480D480u);
  const uint32_t h = w >> 8;
  uint4 r;
  r.x = h2_as_u32(__hmul2(__hsub2(u32_as_h2((w & 0x000F000Fu) | kMagic), k1032), s2));
  r.y = h2_as_u32(__hmul2(__hfma2(u32_as_h2((w & 0x00F000F0u) | kMagic), kSixteenth, kMinus72), s2));
  r.z = h2_as_u32(__hmul2(__hsub2(u32_as_h2((h & 0x000F000Fu) | kMagic), k1032), s2));
  r.w = h2_as_u32(__hmul2(__hfma2(u32_as_h2((h & 0x00F000F0u) | kMagic), kSixteenth, kMinus72), s2));
  return r;
}

// The same for bf16 activations: q is exact in fp16, the product q * s is formed in FP32 and rounded once to bf16.
__device__ __forceinline__ uint32_t bf2_mul(uint32_t q2, float s) {
  const float2 f = __half22float2(u32_as_h2(q2));
  const __nv_bfloat162 v = __floats2bfloat162_rn(f.x * s, f.y * s);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint4 dequant8_bf16(uint32_t w, float s) {
  constexpr uint32_t kMagic = 0x64006400u;
  const __half2 k1032 = u32_as_h2(0x64086408u);
  const __half2 kSixteenth = u32_as_h2(0x2C002C00u);
  const __half2 kMinus72 = u32_as_h2(0xD480D480u);
  const uint32_t h = w >> 8;
  uint4 r;
  r.x = bf2_mul(h2_as_u32(__hsub2(u32_as_h2((w & 0x000F000Fu) | kMagic), k1032)), s);
  r.y = bf2_mul(h2_as_u32(__hfma2(u32_as_h2((w & 0x00F000F0u) | kMagic), kSixteenth, kMinus72)), s);
  r.z = bf2_mul(h2_as_u32(__hsub2(u32_as_h2((h & 0x000F000Fu) | kMagic), k1032)), s);
  r.w = bf2_mul(h2_as_u32(__hfma2(u32_as_h2((h & 0x00F000F0u) | kMagic), kSixteenth, kMinus72)), s);
  return r;
}

__device__ __forceinline__ uint16_t round16(float v, bool bf16) {
  if (bf16) {
    const __nv_bfloat16 b = __float2bfloat16_rn(v);
    return *reinterpret_cast<const uint16_t*>(&b);
  }
  const __half h = __float2half_rn(v);
  return *reinterpret_cast<const uint16_t*>(&h);
}

// round16(v), then + bias as a 16-bit addition: the two roundings of `y = product; y + bias`
__device__ __forceinline__ uint16_t round16_bias(float v, uint16_t bias, bool bf16) {
  const uint16_t r = round16(v, bf16);
  if (bf16) {
    const __nv_bfloat16 a = *reinterpret_cast<const __nv_bfloat16*>(&r), b = *reinterpret_cast<const __nv_bfloat16*>(&bias);
    return round16(__bfloat162float(a) + __bfloat162float(b), true);
  }
  const __half a = *reinterpret_cast<const __half*>(&r), b = *reinterpret_cast<const __half*>(&bias);
  return round16(__half2float(a) + __half2float(b), false);
}

// Pairs: one packed conversion (a single cvt.rn.f16.f32 runs at a quarter of the packed one's rate: draining an
// accumulator took 3300 clocks with it), one packed addition.
template <bool kBf16>
__device__ __forceinline__ uint32_t round16x2(float lo, float hi) {
  if constexpr (kBf16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <bool kBf16>
__device__ __forceinline__ uint32_t add16x2(uint32_t a, uint32_t b) {
  if constexpr (kBf16) {
    const __nv_bfloat162 v = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __half2 v = __hadd2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&v);
}

// out: 16-bit y [M, N] when splits == 1, else FP32 partial [splits][M][N]
template <bool kBf16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
int4_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                 const __half* __restrict__ scales, const __grid_constant__ OutSpec out, float* __restrict__ partial,
                 const __grid_constant__ Shape sh,
                 unsigned int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + kOffBars);   // packed words landed
  uint64_t* w_free = w_full + kWordStages;                           // ... and have been read
  uint64_t* x_full = w_free + kWordStages;                           // activation tile landed
  uint64_t* x_free = x_full + kMaxXStages;                           // the MMAs that read it have completed
  uint64_t* a_ready = x_free + kMaxXStages;                             // leader: both CTAs' weights are in TMEM (and both x tiles landed)
  uint64_t* a_free = a_ready + kStages;                              // the MMAs that read them have completed
  uint64_t* acc_full = a_free + kStages;                         // [2] accumulator complete
  uint64_t* acc_free = acc_full + 2;                                 // [2] leader: accumulator read by both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffMisc);
  volatile uint32_t* abort_word = tmem_slot + 1;
  const AbortCtx ctx{abort_word, status};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int items = sh.m_tiles * sh.n_tiles * sh.splits;
  const int total_kb = (sh.K + kBlockK - 1) / kBlockK;   // a last half block: x is zero-filled past K
  const bool two_acc = sh.mt <= 128;
  const uint32_t x_half = (uint32_t)(sh.mt / 2) * 128u, x_bytes = 2 * x_half;   // this CTA's half of the batch rows x 64 / 128 k
  const uint32_t x_stages = min((uint32_t)kMaxXStages, (uint32_t)kXRing / x_bytes);

  struct Item {
    int m0, n0, kb_begin, n_kb, split;
  };
  auto item_at = [&](int it) {   // batch tiles fastest: the pairs running together share weight rows
    Item w;
    const int mt_i = it % sh.m_tiles, rest = it / sh.m_tiles;
    w.split = rest / sh.n_tiles;
    w.m0 = mt_i * sh.mt;
    w.n0 = (rest - w.split * sh.n_tiles) * kPairRows + (int)rank * kRows;   // this CTA's weight rows
    w.kb_begin = w.split * sh.kblocks_per_split;
    w.n_kb = min(total_kb - w.kb_begin, sh.kblocks_per_split);
    return w;
  };

  // One pipeline step of the TMA producer: the words of K blocks i, i + 1 (even i) and the activations of K block i.
  struct Ring {
    uint32_t slot = 0, parity = 0;
    __device__ void next(uint32_t stages) {
      if (++slot == stages) { slot = 0; parity ^= 1u; }
    }
  };
  Ring p_words, p_x;
  auto load = [&](const Item& w, int i) -> bool {
    if ((i & 1) == 0) {
      if (!mbar_wait(&w_free[p_words.slot], p_words.parity ^ 1u, ctx, kWaitWordsFree)) return false;
      mbar_arrive_expect_tx(&w_full[p_words.slot], kWordBytes);
      tma_load_2d(smem + p_words.slot * kWordBytes, &tm_w, &w_full[p_words.slot], (w.kb_begin + i) * (kBlockK / 8), w.n0);
      p_words.next(kWordStages);
    }
    if (!mbar_wait(&x_free[p_x.slot], p_x.parity ^ 1u, ctx, kWaitFree)) return false;
    mbar_arrive_expect_tx(&x_full[p_x.slot], x_bytes);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      tma_load_4d(smem + kOffX + p_x.slot * x_bytes + h * x_half, &tm_x, &x_full[p_x.slot], (w.kb_begin + i) * kBlockK + h * 64,
                  w.m0 + (int)rank * (sh.mt / 2), 0, 0);
    p_x.next(x_stages);
    return true;
  };
  if (warp == kProducerWarp) {
    if (lane == 0) {
      tma_prefetch_desc(&tm_w);
      tma_prefetch_desc(&tm_x);
      for (int s = 0; s < kWordStages; ++s) {
        mbar_init(&w_full[s], 1);
        mbar_init(&w_free[s], 8);   // the two groups that read a copy of words
      }
      for (int s = 0; s < kMaxXStages; ++s) {
        mbar_init(&x_full[s], 1);
        mbar_init(&x_free[s], 1);
      }
      for (int s = 0; s < kStages; ++s) {
        mbar_init(&a_ready[s], 8);   // the four warps of a group, in both CTAs
        mbar_init(&a_free[s], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&acc_full[i], 1);
        mbar_init(&acc_free[i], 2 * kEpilogueWarps);
      }
      *abort_word = 0;
      fence_mbar_init();
    }
    __syncwarp();
  }
  if (warp == kMmaWarp) {
    tmem_alloc_pair(tmem_slot, kTmemCols);
    tmem_relinquish_pair();
    tc_fence_before_sync();
  }
  // The producer only announces its part of the set-up and goes on to its first loads, which touch this CTA's barriers
  // only; everybody else waits for this CTA here and for the other one (whose barriers it will arrive on, whose TMEM the
  // MMAs will write) where it first needs it.
  if (warp == kProducerWarp) {
    asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
  } else {
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
  }
  cluster_arrive();
  tc_fence_after_sync();
  pdl_wait(scales);   // every role: from here on memory of the kernel in front is read (and what it reads may be overwritten)
  pdl_launch_dependents();
  const uint32_t tmem_base = *tmem_slot;   // (not used by the producer, which has not waited for it)

  if (warp >= kProducerWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsMisc));
    if (warp == kProducerWarp) {
    // ---------------------------------------------------------------- TMA
    if (lane == 0) {
      bool ok = true;
      for (int it = pair; ok && it < items; it += pairs) {
        const Item w = item_at(it);
        for (int i = 0; ok && i < w.n_kb; ++i) ok = load(w, i);
      }
    }
    __syncwarp();
    cluster_wait();
    } else if (warp == kMmaWarp) {
    // ---------------------------------------------------------------- tcgen05.mma of the pair
    // The whole warp walks the loop and one elected lane issues: addresses and descriptors then stay in uniform
    // registers (inside `if (lane == 0)` every MMA costs ~95 clocks of moves into them, more than a small MMA takes).
    cluster_wait();
    if (rank == 0) {
      const uint32_t idesc = idesc_f16(kPairRows, sh.mt, kBf16 ? 1 : 0, 0, 0);
      const uint64_t desc0 = smem_desc_sw128(smem_u32(smem + kOffX), 16, 1024);
      uint32_t kc = 0, ic = 0;
      Ring x;
      bool ok = true;
      for (int it = pair; ok && it < items; it += pairs, ++ic) {
        const int n_kb = item_at(it).n_kb;
        const uint32_t buf = two_acc ? (ic & 1u) : 0u, use = two_acc ? (ic >> 1) : ic;
        ok = __all_sync(0xffffffffu, mbar_wait(&acc_free[buf], (use & 1u) ^ 1u, ctx, kWaitAccFree));
        if (!ok) break;
        const uint32_t acc = tmem_base + buf * 128u;
        for (int i = 0; i < n_kb; ++i, ++kc) {
          const uint32_t s = kc % kStages;
          ok = __all_sync(0xffffffffu, mbar_wait(&a_ready[s], (kc / kStages) & 1u, ctx, kWaitAReady));
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t a = tmem_base + kColA + s * 64u;
          const uint64_t b = desc0 + (uint64_t)(x.slot * (x_bytes >> 4));
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kBlockK / 16; ++kk)
              mma_ts_pair(acc, a + kk * 8, b + (uint64_t)((kk / 4) * (x_half >> 4) + (kk % 4) * 2), idesc, (i > 0 || kk > 0) ? 1u : 0u);
            tc_commit_pair(&a_free[s]);
            tc_commit_pair(&x_free[x.slot]);
            if (i + 1 == n_kb) tc_commit_pair(&acc_full[buf]);
          }
          __syncwarp();
          x.next(x_stages);
        }
      }
    }
    } else {
      cluster_wait();   // the two warps that only fill the warpgroup: every arrive has its wait before the next one
    }
  } else if (warp < kDequantWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsDequant));
    // ---------------------------------------------------------------- dequantise (thread = weight row)
    // Two groups of four warps take the K blocks in turn: the mbarrier and TMEM round trips of one group pass while the
    // other unpacks.  (All eight warps on every block, half a row each: 1200 clocks per block of 128; this: ~800.  Four
    // groups are no faster: they saturate the issue slots, and the one warp that feeds the tensor cores suffers.)
    const int r = (warp & 3) * 32 + lane;   // row inside the CTA's 128 = TMEM lane
    const int turn = warp >> 2;             // which of the two K blocks of every copy of words
    const int groups = sh.K / sh.group, gshift = sh.group == 128 ? 7 : 6;
    const uint32_t a_base = tmem_base + kColA + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t kc0 = 0, wc = 0;   // K blocks and copies of words before this item
    bool ok = true, peer_ready = false;
    for (int it = pair; ok && it < items; it += pairs) {
      const Item w = item_at(it);
      const __half* srow = scales + (size_t)min(w.n0 + r, sh.N - 1) * groups;
      const int k_first = w.kb_begin * kBlockK;
      auto scale_at = [&](int i, int half) { return srow[min((k_first + i * kBlockK + half * 64) >> gshift, groups - 1)]; };
      __half nx[2] = {scale_at(turn, 0), scale_at(turn, 1)};   // scales of the two 64-wide halves, requested one block ahead
      const int copies = (w.n_kb + 1) / 2;
      uint32_t x_slot = (kc0 + turn) % x_stages, x_parity = ((kc0 + turn) / x_stages) & 1u;   // this group's K blocks in the x ring
      for (int c = turn >> 1; c < copies; c += kDequantGroups / 2) {
        const int i = 2 * c + (turn & 1);   // K block of this item
        const __half sc[2] = {nx[0], nx[1]};
        nx[0] = scale_at(i + kDequantGroups, 0);
        nx[1] = scale_at(i + kDequantGroups, 1);
        const uint32_t ws = (wc + c) % kWordStages;
        ok = __all_sync(0xffffffffu, mbar_wait(&w_full[ws], ((wc + c) / kWordStages) & 1u, ctx, kWaitWords));
        if (!ok) break;
        const uint8_t* words = smem + ws * kWordBytes + r * 128;
        const bool mine = i < w.n_kb;   // (not in the last copy of an odd number of blocks)
        const uint32_t kc = kc0 + i, s = kc % kStages, ph = (kc / kStages) & 1u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t pw[8];
#pragma unroll
          for (int e = 0; e < 2; ++e)
            *reinterpret_cast<uint4*>(&pw[4 * e]) = *reinterpret_cast<const uint4*>(words + (((4 * (turn & 1) + 2 * h + e) ^ (r & 7)) << 4));
          if (h == 1) {
            fence_proxy_async_smem();   // these reads are over before the next copy of words may land
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_free[ws]);
          }
          uint32_t a[32];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            uint4 q;
            if constexpr (kBf16) q = dequant8_bf16(pw[e], __half2float(sc[h]));
            else q = dequant8(pw[e], __half2half2(sc[h]));
            a[4 * e] = q.x; a[4 * e + 1] = q.y; a[4 * e + 2] = q.z; a[4 * e + 3] = q.w;
          }
          if (h == 0 && mine) {
            ok = __all_sync(0xffffffffu, mbar_wait(&a_free[s], ph ^ 1u, ctx, kWaitAFree));
            tc_fence_after_sync();
          }
          if (ok && mine) tmem_st_x32(a_base + s * 64u + h * 32u, a);
        }
        if (!ok || !mine) break;
        ok = __all_sync(0xffffffffu, mbar_wait(&x_full[x_slot], x_parity, ctx, kWaitX));
        if (!ok) break;
        x_slot += kDequantGroups;
        if (x_slot >= x_stages) { x_slot -= x_stages; x_parity ^= 1u; }   // x_stages >= kDequantGroups
        if (!peer_ready) cluster_wait();
        peer_ready = true;
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_at(&a_ready[s], 0);
      }
      kc0 += w.n_kb;
      wc += copies;
    }
    if (!peer_ready) cluster_wait();
  } else {
    // ---------------------------------------------------------------- epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
    // TMEM lane = weight row n, column = batch row m, but y is [M, N]: each of the two warpgroups (which own alternate
    // 32-column chunks) rounds its chunks into registers and frees the accumulator.  Lanes 2j and 2j + 1 then exchange
    // halves, so that each holds two neighbouring features of one batch row: 4-byte stores, 64 contiguous bytes of a
    // row per half warp.  (A transpose through shared memory into 16-byte stores took 1700-2200 clocks per chunk.)
    const int wg = (warp - kDequantWarps) >> 2, r = (warp & 3) * 32 + lane;
    const uint32_t lane_bits = (uint32_t)((warp & 3) * 32) << 16;
    const int chunks = sh.mt / 32;
    // A wait expired earlier on this device: nothing is written (the read's latency passes during the products), but the
    // accumulators are still given back: without that the MMA warp's wait for one would run out too, 2 s in every call.
    const bool muted = __any_sync(0xffffffffu, *reinterpret_cast<volatile unsigned int*>(status) != 0);
    bool ok = true;
    cluster_wait();
    uint32_t ic = 0;
    for (int it = pair; ok && it < items; it += pairs, ++ic) {
      const Item w = item_at(it);
      const uint32_t buf = two_acc ? (ic & 1u) : 0u, use = two_acc ? (ic >> 1) : ic;
      const int row = w.n0 + r;
      const bool with_bias = sh.splits == 1 && out.bias != nullptr;
      const uint32_t bias2 = with_bias ? out.bias[min(row, sh.N - 1)] * 0x10001u : 0u;
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], use & 1u, ctx, kWaitAcc));
      if (!ok) break;
      tc_fence_after_sync();
      if (muted) {
        if (lane == 0 && it + (two_acc ? 2 : 1) * pairs < items) mbar_arrive_at(&acc_free[buf], 0);
        continue;
      }
      const uint32_t acc = tmem_base + buf * 128u + lane_bits;
      if (sh.splits > 1) {   // FP32 partials: a warp's 32 rows are 128 contiguous bytes of every batch row
        float* dst = partial + ((size_t)w.split * sh.M + w.m0) * sh.N + row;
#pragma unroll 1
        for (int ch = wg; ch < chunks; ch += 2) {
          uint32_t v[32];
          tmem_ld_x32(acc + ch * 32, v);
          tmem_wait_ld_regs(v);
          if (row < sh.N) {
#pragma unroll
            for (int c = 0; c < 32; ++c)
              if (w.m0 + ch * 32 + c < sh.M) dst[(size_t)(ch * 32 + c) * sh.N] = __uint_as_float(v[c]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0 && it + (two_acc ? 2 : 1) * pairs < items) mbar_arrive_at(&acc_free[buf], 0);
        continue;
      }
      uint32_t p[4][16];   // two batch rows per register
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        const int ch = wg + 2 * cc;
        if (ch < chunks) {
          uint32_t v[32];
          tmem_ld_x32(acc + ch * 32, v);
          tmem_wait_ld_regs(v);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            p[cc][i] = round16x2<kBf16>(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            if (with_bias) p[cc][i] = add16x2<kBf16>(p[cc][i], bias2);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      // the next tile may accumulate (the last arrivals would have nobody waiting: none is in flight when a CTA leaves)
      if (lane == 0 && it + (two_acc ? 2 : 1) * pairs < items) mbar_arrive_at(&acc_free[buf], 0);
      const int pair_n = (row & ~1) - w.n0;               // the two features this lane stores: n0 + pair_n, + 1
      const int left = sh.N - (row & ~1);                 // how many of them (and beyond) exist
      const bool vec = ((out.ld | out.col0) & 1) == 0;    // pairs are 4-byte aligned
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        const int ch = wg + 2 * cc;
        if (ch < chunks) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {   // this lane's batch row of the pair 2i, 2i + 1: the even one for even lanes
            const uint32_t other = __shfl_xor_sync(0xffffffffu, p[cc][i], 1);
            p[cc][i] = lane & 1 ? __byte_perm(p[cc][i], other, 0x3276) : __byte_perm(p[cc][i], other, 0x5410);
          }
          const int m_first = w.m0 + ch * 32 + (lane & 1);
          const bool whole = vec && w.n0 + kRows <= sh.N && w.m0 + ch * 32 + 32 <= sh.M;   // uniform: no checks per store
          if (out.silu) {   // (N is even: both features of a pair exist or neither does)
            uint16_t* at = reinterpret_cast<uint16_t*>(out.y[0]) + (size_t)m_first * out.ld + ((w.n0 + pair_n) >> 1);
#pragma unroll
            for (int i = 0; i < 16; ++i, at += 2 * (size_t)out.ld)
              if (left > 0 && m_first + 2 * i < sh.M) *at = silu_pair(p[cc][i]);
            continue;
          }
          for (int o = 0; o < out.count; ++o) {
            uint16_t* at = reinterpret_cast<uint16_t*>(out.y[o]) + (size_t)m_first * out.ld + out.col0 + w.n0 + pair_n;
            const size_t two_rows = 2 * (size_t)out.ld;
            if (whole) {
#pragma unroll
              for (int i = 0; i < 16; ++i, at += two_rows) *reinterpret_cast<uint32_t*>(at) = p[cc][i];
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i, at += two_rows) {
                const bool row_ok = m_first + 2 * i < sh.M;
                if (row_ok && vec && left > 1) {
                  *reinterpret_cast<uint32_t*>(at) = p[cc][i];
                } else if (row_ok) {
                  if (left > 0) at[0] = (uint16_t)p[cc][i];
                  if (left > 1) at[1] = (uint16_t)(p[cc][i] >> 16);
                }
              }
            }
          }
        }
      }
    }
  }

  // teardown: every role of both CTAs falls through to here, also after an expired wait
  if (*abort_word != 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);  // let copies in flight land
  }
  tc_fence_before_sync();
  __syncthreads();
  // Neither CTA leaves (or frees TMEM) while the other may still read its memory or arrive on its barriers.  Relaxed: the
  // order of the output stores is not the barrier's business, and a release would wait for them (~1000 clocks).
  cluster_arrive_relaxed();
  cluster_wait();
  if (warp == kMmaWarp) {
    __syncwarp();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// y[m, col0 + n] = 16-bit(sum over splits, in split order, of partial[s][m][n]) (+ bias), in every output buffer.  V: columns
// per thread (4 where rows allow 16-byte loads).  S: all pieces of an element are requested before the first one is added (in
// split order): a kernel of few elements is bound by the round trips to L2.  With 5 to 16 pieces, four at a time and the rest one
// by one before: 512 x 12288, M = 48 11.3 us the whole call, now 9.7; 1536 x 8960, M = 33 12.1 and 10.5.  S = 0, up to four
// pieces or one column per thread: a plain loop; with registers for 16 pieces 2048 x 5632, M = 512 takes 23.5 instead of 20.9,
// 1001 x 2048, M = 33 8.3 instead of 7.8.
template <int V, int S>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ partial, const __grid_constant__ OutSpec out,
                                                            int M, int N, int splits) {
  pdl_wait(partial);
  pdl_launch_dependents();
  const long long elems = (long long)M * N, vecs = elems / V;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < vecs; i += (long long)gridDim.x * blockDim.x) {
    float acc[V];
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = 0.f;
    const float* p = partial + i * V;
    if constexpr (S > 0) {
      alignas(16) float v[S][V];
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (s < splits) {
          if constexpr (V == 4) *reinterpret_cast<float4*>(v[s]) = *reinterpret_cast<const float4*>(p + (size_t)s * elems);
          else v[s][0] = p[(size_t)s * elems];
        }
#pragma unroll
      for (int s = 0; s < S; ++s)
        if (s < splits) {
#pragma unroll
          for (int e = 0; e < V; ++e) acc[e] += v[s][e];
        }
    } else {
#pragma unroll 4
      for (int s = 0; s < splits; ++s) {
        if constexpr (V == 4) {
          const float4 v = *reinterpret_cast<const float4*>(p + (size_t)s * elems);
          acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w;
        } else {
          acc[0] += p[(size_t)s * elems];
        }
      }
    }
    const long long m = i * V / N;
    const int n = (int)(i * V - m * N);
    uint16_t r[V];
#pragma unroll
    for (int e = 0; e < V; ++e) r[e] = out.bias ? round16_bias(acc[e], out.bias[n + e], out.bf16 != 0) : round16(acc[e], out.bf16 != 0);
    if constexpr (V == 4) {
      if (out.silu) {
        *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(out.y[0]) + m * out.ld + n / 2) =
            silu_pair(r[0] | ((uint32_t)r[1] << 16)) | ((uint32_t)silu_pair(r[2] | ((uint32_t)r[3] << 16)) << 16);
        continue;
      }
    }
    for (int o = 0; o < out.count; ++o) {
      uint16_t* dst = reinterpret_cast<uint16_t*>(out.y[o]) + m * out.ld + out.col0 + n;
      if constexpr (V == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(r[0] | ((uint32_t)r[1] << 16), r[2] | ((uint32_t)r[3] << 16));
      else dst[0] = r[0];
    }
  }
}

// Batch rows per tile and K splits, by a cost model fitted to measurements on B200 (us, graph of L2-cold calls, deviation
// about 7 %): a K block of 128 takes 0.45 to dequantise (bf16: 0.55) and 2.3 per 1000 batch rows to multiply, whichever is
// longer; a tile 0.6 plus 1.0 per 100 batch rows to drain (the last one also to store); 5.5 for launch, set-up and the
// first block; a split plan 1.8 for the second kernel and its traffic at 5 TB/s.
Shape make_plan(int M, int N, int K, int group, bool bf16) {
  Shape best = {};
  double best_cost = 1e30;
  const int kblocks = ceil_div(K, kBlockK), n_tiles = ceil_div(N, kPairRows), pairs = sm_count() / 2;
  for (int mt = 32; mt <= kMaxTile; mt += 32) {
    const int m_tiles = ceil_div(M, mt);
    if (mt > 32 && m_tiles == ceil_div(M, mt - 32)) continue;   // the same tiles, more padding
    for (int sp = 1; sp <= kMaxSplits; ++sp) {
      const int per = ceil_div(ceil_div(kblocks, sp), 2) * 2;
      const int splits = ceil_div(kblocks, per);
      if (splits != sp) continue;
      const long long items = (long long)m_tiles * n_tiles * splits;
      const double waves = (double)((items + pairs - 1) / pairs);
      const double unpack = bf16 ? 0.55 : 0.45, multiply = 0.0023 * mt;
      double cost = 5.5 + waves * ((per < kblocks ? per : kblocks) * (multiply > unpack ? multiply : unpack) + 0.6) + 0.01 * mt;
      if (splits > 1) cost += 1.8 + (double)splits * M * N * 8.0 / 5.0e6;
      if (cost < best_cost) {
        best_cost = cost;
        best.mt = mt; best.m_tiles = m_tiles; best.n_tiles = n_tiles; best.splits = splits; best.kblocks_per_split = per;
      }
    }
  }
  best.M = M; best.N = N; best.K = K; best.group = group;
  return best;
}

template <bool kBf16>
int launch(const Shape& p, const CUtensorMap& tw, const CUtensorMap& tx, const void* scales, const OutSpec& out, float* partial,
           unsigned int* status, cudaStream_t stream) {
  auto kernel = int4_gemm_kernel<kBf16>;
  static bool configured[64] = {false};
  int dev = 0;
  KFB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    KFB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    configured[dev] = true;
  }
  const long long items = (long long)p.m_tiles * p.n_tiles * p.splits;
  const long long pairs = items < sm_count() / 2 ? items : sm_count() / 2;
  if (int rc = launch_kernel("int4_gemm_kernel", kernel, dim3((unsigned)(2 * pairs)), dim3(kThreads), kSmem, stream, tw, tx, (const __half*)scales,
                             out, partial, p, status))
    return rc;
  if (p.splits > 1) {
    const bool vec = ((p.N | out.col0) & 3) == 0 && (out.silu ? (out.ld & 1) == 0 : (out.ld & 3) == 0);
    const long long work = (long long)p.M * p.N / (vec ? 4 : 1);
    long long blocks = (work + 255) / 256;
    const long long cap = (long long)sm_count() * 8;
    if (blocks > cap) blocks = cap;
    auto reduce = !vec ? splitk_reduce_kernel<1, 0> : p.splits <= 4 ? splitk_reduce_kernel<4, 0> : splitk_reduce_kernel<4, kMaxSplits>;
    return launch_kernel("splitk_reduce_kernel", reduce, dim3((unsigned)blocks), dim3(256), 0, stream, (const float*)partial, out, p.M, p.N, p.splits);
  }
  return KFB_OK;
}

}  // namespace
}  // namespace gemm
}  // namespace kfb

using namespace kfb;

size_t kfb::gemm::ws_bytes(int M, int N, int K, int group, bool bf16) {
  if (M < 1 || N < 1 || K < 64 || (group != 64 && group != 128) || K % group) return 0;
  const Shape p = make_plan(M, N, K, group, bf16);
  return p.splits > 1 ? (size_t)p.splits * M * N * sizeof(float) : 0;
}

// (fp16 and bf16 plans may split K differently: enough for both)
extern "C" size_t kfb_int4_gemm_ws_bytes(int M, int N, int K, int group) {
  const size_t a = gemm::ws_bytes(M, N, K, group, false), b = gemm::ws_bytes(M, N, K, group, true);
  return a > b ? a : b;
}

namespace {

int gemm_common(const void* x, const void* packed, const void* scales, const gemm::OutSpec& out, int M, int N, int K,
                int group, void* ws, size_t ws_bytes, void* stream) {
  if (int rc = require_sm100()) return rc;
  if (M < 1) return fail(KFB_ERR_INVALID, "int4_gemm needs M >= 1, got M=%d", M);
  if (group != 64 && group != 128) return fail(KFB_ERR_INVALID, "group_size must be one of (64, 128), got %d", group);
  if (N < 1 || K < group || K % group) return fail(KFB_ERR_INVALID, "K=%d is not a multiple of group_size=%d", K, group);
  if (!x || !packed || !scales) return fail(KFB_ERR_INVALID, "null pointer");
  for (int i = 0; i < out.count; ++i)
    if (!out.y[i] || !aligned16(out.y[i])) return fail(KFB_ERR_ALIGNMENT, "output buffers must be non-null and 16-byte aligned");
  if (!aligned16(x) || !aligned16(packed)) return fail(KFB_ERR_ALIGNMENT, "x and packed must be 16-byte aligned");
  const gemm::Shape p = gemm::make_plan(M, N, K, group, out.bf16 != 0);
  if ((long long)p.m_tiles * p.n_tiles * p.splits > 0x7fffffffLL) return fail(KFB_ERR_INVALID, "too many tiles for one launch");
  const size_t need = p.splits > 1 ? (size_t)p.splits * M * N * sizeof(float) : 0;
  if (need > 0 && (!ws || ws_bytes < need))
    return fail(KFB_ERR_WORKSPACE, "int4_gemm needs a %zu-byte workspace for %d K splits, got %zu", need, p.splits, ws_bytes);
  if (need > 0 && !aligned16(ws)) return fail(KFB_ERR_ALIGNMENT, "workspace must be 16-byte aligned");
  unsigned int* status = device_status_word();
  if (!status) return fail(KFB_ERR_CUDA, "cannot resolve the device status word");

  CUtensorMap tw, tx;
  // packed int32 [N, K/8] as 32-bit elements, box 32 words (two K blocks) x 128 rows, 128-byte swizzle
  if (int rc = make_tmap_2d_plain(&tw, packed, /*elem_bytes=*/4, (uint64_t)K / 8, (uint64_t)N, (uint64_t)K / 2, 32, gemm::kRows, true)) return rc;
  // x [M, K], box 64 k x half a tile of rows, 128-byte swizzle (the 4-D helper with unit outer dims)
  const uint64_t xd[4] = {(uint64_t)K, (uint64_t)M, 1, 1};
  const uint64_t xs[3] = {(uint64_t)K * 2, (uint64_t)M * K * 2, (uint64_t)M * K * 2};
  const uint32_t xb[4] = {64, (uint32_t)(p.mt / 2), 1, 1};
  if (int rc = make_tmap_4d_sw128(&tx, x, out.bf16 ? KFB_BF16 : KFB_F16, xd, xs, xb)) return rc;

  cudaStream_t s = (cudaStream_t)stream;
  float* partial = static_cast<float*>(ws);
  return out.bf16 ? gemm::launch<true>(p, tw, tx, scales, out, partial, status, s) : gemm::launch<false>(p, tw, tx, scales, out, partial, status, s);
}

}  // namespace

int kfb::gemm::run(const void* x, const void* packed, const void* scales, const void* bias, void* y, int M, int N, int K, int group,
                   bool bf16, bool silu, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if (silu && (bf16 || N % 4)) return fail(KFB_ERR_UNSUPPORTED, "the SiLU-pair epilogue is fp16 and needs N %% 4 == 0, got N=%d", N);
  OutSpec out = {};
  out.y[0] = static_cast<__half*>(y);
  out.count = 1;
  out.ld = silu ? N / 2 : N;
  out.bf16 = bf16;
  out.bias = static_cast<const uint16_t*>(bias);
  out.silu = silu;
  return gemm_common(x, packed, scales, out, M, N, K, group, ws, ws_bytes, stream);
}

extern "C" int kfb_int4_gemm(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K,
                             int group, void* ws, size_t ws_bytes, void* stream) {
  if (!y) return fail(KFB_ERR_INVALID, "null pointer");
  return gemm::run(x, packed, scales, nullptr, y, M, N, K, group, false, false, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int kfb_int4_gemm_bf16(const void* x, const void* packed, const void* scales, void* y, int M, int N, int K,
                                  int group, void* ws, size_t ws_bytes, void* stream) {
  if (!y) return fail(KFB_ERR_INVALID, "null pointer");
  return gemm::run(x, packed, scales, nullptr, y, M, N, K, group, true, false, ws, ws_bytes, (cudaStream_t)stream);
}

extern "C" int kfb_int4_gemm_allgather(const void* x, const void* packed, const void* scales, void* const* y_all,
                                       int n_buffers, int M, int N_local, int K, int group, int ld, int col0, void* ws,
                                       size_t ws_bytes, void* stream) {
  if (n_buffers < 1 || n_buffers > gemm::kMaxPeers)
    return fail(KFB_ERR_INVALID, "n_buffers must be in [1, %d], got %d", gemm::kMaxPeers, n_buffers);
  if (!y_all) return fail(KFB_ERR_INVALID, "null pointer");
  if (col0 < 0 || ld < col0 + N_local)
    return fail(KFB_ERR_INVALID, "columns [%d, %d) do not fit in a row of %d", col0, col0 + N_local, ld);
  gemm::OutSpec out = {};
  for (int i = 0; i < n_buffers; ++i) out.y[i] = static_cast<__half*>(y_all[i]);
  out.count = n_buffers;
  out.ld = ld;
  out.col0 = col0;
  return gemm_common(x, packed, scales, out, M, N_local, K, group, ws, ws_bytes, stream);
}
