// Decode attention (q_len = 1) for sm_100a: split-KV, HBM-bound.
//
// The reference serves decode with its prefill kernel: one CTA per (batch, query head) walks all
// Nk keys serially with 127 of 128 tile rows padding, and K/V are re-read once per query head of a
// group (csrc/attention/attn_v4_kernel.cuh:43-214, grid (1, B*H)).  Here:
//   * grid = (splits, Hk * head-chunks, B): the key range of one (batch, kv head) is split across
//     CTAs so that even B = 1, Hk = 4 fills the 148 SMs;
//   * the G = H / Hk query heads of a KV head are the M rows of the MMA (chunks of 16), so every K/V
//     byte is read from HBM ONCE per group instead of once per query head;
//   * a producer warp streams 64-key K and V tiles with TMA (128-byte swizzle) through an mbarrier
//     ring; each consumer warp takes whole tiles in turn: S = Q K^T and O += P V on mma.sync.m16n8k16
//     (FP32 accumulate) -- the kernel is bandwidth-bound (8 FLOP per K/V byte at G = 8), tensor cores
//     only keep the ALU cost below the HBM time.  (Four warps sharing every tile, 16 keys each, walked
//     through as many dependent softmax steps as there are tiles; a warp per tile has a quarter or a
//     sixth of them, each with four times the independent work.)
//   * the key range of a split is cut on the device from the valid length, so the splits of a short
//     sequence in a long cache are as even as those of a full one;
//   * per-warp online softmax (base 2, FP32), warps merged in shared memory in fixed order.  Up to
//     eight splits form a thread-block cluster and are merged through distributed shared memory, in
//     split order, every CTA a share of the output: one launch, nothing goes through global memory.
//     Each CTA sends its sums to the CTA that needs them, so one cluster barrier is enough and no load
//     crosses the cluster (reading them from one another took two barriers and a round trip: 4 sequences
//     of 800..1100 keys 5.7 us, now 4.8; 8 of 1000..4096 8.4 and 7.9).
//     More splits write one partial (O, m, l) each to the caller's workspace, combined in split order
//     by a second small kernel.  Both are deterministic; with one split the result is written directly.
#include "attn.cuh"
#include "sm100.cuh"

namespace kfb {
namespace attn {
namespace {

using namespace sm100;

constexpr int kTileKeys = 64;
// Depth of the K/V tile ring and consumer warps.  A grid larger than the GPU runs several CTAs per SM with a shallow ring
// each: three of 4 tiles at D = 64, two of 3 tiles at D = 128.  A grid of at most one CTA per SM (decode at batch 1-8:
// B * Hk * splits CTAs) is bound by the bytes ONE SM keeps in flight, so there the ring takes (nearly) the whole shared
// memory and every tile of a short cache is requested at once.
template <int D> constexpr int shallow_stages() { return D == 64 ? 4 : 3; }
template <int D> constexpr int deep_stages() { return D == 64 ? 12 : 6; }
template <int D, int kStages> constexpr int consumer_warps() { return kStages == shallow_stages<D>() ? kStages : 6; }
constexpr int kRows = 16;  // query heads per CTA (MMA M)
constexpr int kMaxCluster = 8;

enum WaitCode : uint32_t { kWaitFull = 0x201, kWaitEmpty };

template <int D, int kStages>
struct Layout {
  static constexpr int kWarps = consumer_warps<D, kStages>();
  static constexpr int kThreads = (kWarps + 1) * 32;
  // a stage always holds tiles of the same warp: with another warp's tile in between, a wait for the round after next could
  // be taken for the round before (copies may complete out of order)
  static_assert(kStages % kWarps == 0, "");
  static constexpr int kHalf = kTileKeys * 128;       // 64 keys x 64 columns
  static constexpr int kTile = kTileKeys * D * 2;     // one K or V tile
  static constexpr int kStage = 2 * kTile;            // K then V
  static constexpr int kBars = kStages * kStage;
  static constexpr int kMisc = kBars + 2 * kStages * 8;
  // what the CTAs of a cluster send this one, outside the ring, which may still be in use then: its share of the output from each
  // (shares are multiples of four elements), then m[16] and l[16] of each
  static constexpr int kSent = kMisc + 16;
  static constexpr int kSentStats = kRows * D + 4 * kMaxCluster;   // floats before the first m
  static constexpr int kBytes = kSent + (kSentStats + kMaxCluster * 2 * kRows) * 4;
  static constexpr int kAlloc = kBytes + 1024, kAllocSingle = kSent + 1024;   // in a cluster, and not
  // the cross-warp merge reuses the tile ring: per warp O[16][D] + m[16] + l[16] floats
  static constexpr int kMergeBytes = kWarps * kRows * (D + 2) * 4;
  static_assert(kMergeBytes <= kBars, "merge scratch must fit in the tile ring");
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}

template <bool kBf16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}
template <bool kBf16>
__device__ __forceinline__ uint16_t pack1(float x) {
  if constexpr (kBf16) {
    __nv_bfloat16 v = __float2bfloat16_rn(x);
    return *reinterpret_cast<uint16_t*>(&v);
  } else {
    __half v = __float2half_rn(x);
    return *reinterpret_cast<uint16_t*>(&v);
  }
}

// To the same place in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ void st_cluster(const float* at, uint32_t rank, float v) {
  asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, %1;\n\tst.shared::cluster.f32 [ra], %2;\n\t}" ::"r"(smem_u32(at)),
               "r"(rank), "f"(v) : "memory");
}

// byte offset of (key row r, 16-byte chunk c of the 128-byte row) inside a 128B-swizzled 64-key half tile
__device__ __forceinline__ uint32_t swz(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// A warp whose wait has expired (or been called off) spends 200 us here before it goes on to the CTA's barrier, so that copies in
// flight land before the ring becomes the scratch of the merge or is freed.  Called in the loops, where only an expired wait comes
// by: a look at the abort word in front of the barrier instead cost every call (8 sequences of 1000..4096 keys 8.45 us against
// 8.38; a step of the 22-layer model at 512 keys 518.6 against 516.5).
__device__ __noinline__ void let_copies_land() {
  const unsigned long long t0 = globaltimer_ns();
  while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
}

// Partial results, per (batch, kv head * chunks + chunk, split): O[16][D], m[16], l[16] floats.
template <int D>
__host__ __device__ constexpr int partial_floats() { return kRows * (D + 2); }

// kOldRows: kv_len and all valid rows but the last are older than the kernel in front (kfb_flash_attn_decode_step): the tiles are on
// their way while that kernel ends (step of the 22-layer model at batch 1, 512 keys, with the merge above: 513 us -> 481; batch 32
// 996 -> 964).  kClustered and kOldRows are variants and not arguments: with them as arguments calls without either got slower (22
// sequences of 6000..7000 keys 27.6 us -> 29.5; 42 of 700..2600 12.0 -> 12.7 even where only kClustered was one).
template <int D, bool kBf16, int kStages, bool kClustered, bool kOldRows>
__global__ void __launch_bounds__((consumer_warps<D, kStages>() + 1) * 32)
attn_decode_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const uint16_t* __restrict__ q, uint16_t* __restrict__ o, float* __restrict__ partial, int H, int Hk,
                   int Nk, float scale_log2, unsigned int* status, const int* __restrict__ kv_len,
                   int force_partial) {
  using L = Layout<D, kStages>;
  constexpr int kConsumerWarps = L::kWarps, kThreads = L::kThreads;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* empty = full + kStages;
  volatile uint32_t* abort_word = reinterpret_cast<uint32_t*>(smem + L::kMisc);
  const AbortCtx ctx{abort_word, status};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = H / Hk;
  const int chunks = (G + kRows - 1) / kRows;
  const int split = blockIdx.x, splits = gridDim.x;
  const int hk = blockIdx.y / chunks, chunk = blockIdx.y % chunks;
  const int b = blockIdx.z;
  const int h0 = hk * G + chunk * kRows;               // first query head of this CTA
  const int rows = min(kRows, G - chunk * kRows);      // real query heads
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    *abort_word = *reinterpret_cast<volatile unsigned int*>(status);  // non-zero: an earlier wait expired
    fence_mbar_init();
  }
  if constexpr (kClustered) cluster_arrive_relaxed();   // (its counterpart: before this CTA writes to the others)
  __syncthreads();
  // q, the cache rows and kv_len may be the output of the kernel in front.  kOldRows: only q and the last valid row, so that every
  // tile in front of that row's is requested before the wait.
  if constexpr (!kOldRows) {
    pdl_wait(q, kv_len);
    pdl_launch_dependents();
  }
  // a static KV cache holds Nk rows of which only kv_len[b] are valid (read on the device, so the
  // same launch can be replayed from a CUDA graph while the cache fills up)
  const int valid = kv_len ? min(Nk, max(kv_len[b], 0)) : Nk;
  const int tiles_valid = (valid + kTileKeys - 1) / kTileKeys, per_split = (tiles_valid + splits - 1) / splits;
  const int key_begin = split * per_split * kTileKeys;
  const int key_end = min(valid, key_begin + per_split * kTileKeys);
  const int n_tiles = key_end > key_begin ? (key_end - key_begin + kTileKeys - 1) / kTileKeys : 0;
  const bool aborted = *abort_word != 0;   // uniform: written before the barrier, nothing has been issued yet
  if (kOldRows && aborted) pdl_wait();     // (whoever waits for this kernel relies on its having waited)
  if (aborted && !kClustered) return;

  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float oacc[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) oacc[i][e] = 0.f;

  if (aborted) {
    // a cluster's CTAs leave together
  } else if (warp == kConsumerWarps) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      const int first_new = min(kStages, (valid - 1 - key_begin) / kTileKeys);
      for (int t = 0; t < n_tiles; ++t) {
        const int s = t % kStages;
        if (kOldRows && t == first_new) pdl_wait();
        if (!mbar_wait(&empty[s], ((uint32_t)(t / kStages) & 1u) ^ 1u, ctx, kWaitEmpty)) {
          let_copies_land();
          break;
        }
        mbar_arrive_expect_tx(&full[s], L::kStage);
        uint8_t* dst = smem + s * L::kStage;
        const int key0 = key_begin + t * kTileKeys;
#pragma unroll
        for (int half = 0; half < D / 64; ++half) {
          tma_load_4d(dst + half * L::kHalf, &tm_k, &full[s], half * 64, key0, hk, b);
          tma_load_4d(dst + L::kTile + half * L::kHalf, &tm_v, &full[s], half * 64, key0, hk, b);
        }
      }
    }
    if constexpr (kOldRows) {
      pdl_wait();
      pdl_launch_dependents();
    }
  } else {
    // ------------------------------------------------------------------ consumers
    const int g = lane >> 2, t4 = lane & 3;
    if constexpr (kOldRows) {
      pdl_wait(q);
      pdl_launch_dependents();
    }
    // Q fragments (A operand, 16 heads x D), rows >= `rows` are zero
    uint32_t qa[D / 16][4];
    {
      const uint16_t* q0 = q + ((size_t)b * H + h0 + g) * D;        // row g      (Nq == 1)
      const uint16_t* q1 = q + ((size_t)b * H + h0 + g + 8) * D;    // row g + 8
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const int c = kk * 16 + 2 * t4;
        qa[kk][0] = g < rows ? *reinterpret_cast<const uint32_t*>(q0 + c) : 0u;
        qa[kk][1] = g + 8 < rows ? *reinterpret_cast<const uint32_t*>(q1 + c) : 0u;
        qa[kk][2] = g < rows ? *reinterpret_cast<const uint32_t*>(q0 + c + 8) : 0u;
        qa[kk][3] = g + 8 < rows ? *reinterpret_cast<const uint32_t*>(q1 + c + 8) : 0u;
      }
    }
    const int mat = lane >> 3, mrow = lane & 7;
    for (int t = warp; t < n_tiles; t += kConsumerWarps) {
      const int s = t % kStages;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (uint32_t)(t / kStages) & 1u, ctx, kWaitFull));
      if (!ok) {
        let_copies_land();
        break;
      }
      const uint32_t k_base = smem_u32(smem + s * L::kStage);
      const uint32_t v_base = k_base + L::kTile;
      constexpr int kBlocks = kTileKeys / 16;   // blocks of 16 keys

      // S[16 heads x 64 keys]: eight n-tiles of 8 keys
      float sacc[2 * kBlocks][4];
#pragma unroll
      for (int i = 0; i < 2 * kBlocks; ++i) sacc[i][0] = sacc[i][1] = sacc[i][2] = sacc[i][3] = 0.f;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
        for (int kb = 0; kb < kBlocks; ++kb) {
          // matrices: (keys 0-7, d 0-7) (keys 0-7, d 8-15) (keys 8-15, d 0-7) (keys 8-15, d 8-15)
          const int key = kb * 16 + (mat >> 1) * 8 + mrow;
          const int dchunk = kk * 2 + (mat & 1);
          uint32_t r0, r1, r2, r3;
          ldmatrix_x4(k_base + (dchunk >> 3) * L::kHalf + swz(key, dchunk & 7), r0, r1, r2, r3);
          mma16816<kBf16>(sacc[2 * kb], qa[kk], r0, r1);
          mma16816<kBf16>(sacc[2 * kb + 1], qa[kk], r2, r3);
        }
      // mask keys past this split's range (TMA zero-fills past Nk; keys of the next split are real data)
      const int left = key_end - (key_begin + t * kTileKeys);   // keys of this tile that count
      if (left < kTileKeys) {
#pragma unroll
        for (int nt = 0; nt < 2 * kBlocks; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (nt * 8 + 2 * t4 + (e & 1) >= left) sacc[nt][e] = -INFINITY;
      }

      // online softmax for rows g (e = 0,1) and g + 8 (e = 2,3)
      uint32_t pa[kBlocks][4];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float mx = sacc[0][2 * r];
#pragma unroll
        for (int nt = 0; nt < 2 * kBlocks; ++nt) mx = fmaxf(mx, fmaxf(sacc[nt][2 * r], sacc[nt][2 * r + 1]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(m_run[r], mx * scale_log2);
        const float base = (m_new == -INFINITY) ? 0.f : m_new;
        const float alpha = ex2(m_run[r] - base);
        float sum = 0.f;   // lane-local part of the row sum
#pragma unroll
        for (int kb = 0; kb < kBlocks; ++kb) {
          const float p00 = ex2(fmaf(sacc[2 * kb][2 * r], scale_log2, -base));
          const float p01 = ex2(fmaf(sacc[2 * kb][2 * r + 1], scale_log2, -base));
          const float p10 = ex2(fmaf(sacc[2 * kb + 1][2 * r], scale_log2, -base));
          const float p11 = ex2(fmaf(sacc[2 * kb + 1][2 * r + 1], scale_log2, -base));
          sum += (p00 + p01) + (p10 + p11);
          pa[kb][r] = pack2<kBf16>(p00, p01);       // a0a1 (row g) / a2a3 (row g+8): keys 2t, 2t+1
          pa[kb][2 + r] = pack2<kBf16>(p10, p11);   // a4a5 / a6a7: keys 2t+8, 2t+9
        }
        l_run[r] = fmaf(l_run[r], alpha, sum);
        m_run[r] = m_new;
#pragma unroll
        for (int i = 0; i < D / 8; ++i) {
          oacc[i][2 * r] *= alpha;
          oacc[i][2 * r + 1] *= alpha;
        }
      }
      // Rows of V past key_end get p = 0, but 0 * NaN = NaN: with a device-side length those rows are
      // whatever the cache buffer holds, so this warp zeroes them in its tile first.
      if (left < kTileKeys) {
        for (int i = lane; i < (kTileKeys - left) * 8 * (D / 64); i += 32) {
          const int row = left + i / (8 * (D / 64)), rem = i % (8 * (D / 64));
          *reinterpret_cast<uint4*>(smem + s * L::kStage + L::kTile + (rem >> 3) * L::kHalf + row * 128 + (rem & 7) * 16) =
              make_uint4(0u, 0u, 0u, 0u);
        }
        __syncwarp();
      }
      // O[16 x D] += P[16 x 64 keys] V[64 keys x D]
#pragma unroll
      for (int kb = 0; kb < kBlocks; ++kb)
#pragma unroll
        for (int dn = 0; dn < D / 16; ++dn) {
          // matrices: (keys 0-7, d c0) (keys 8-15, d c0) (keys 0-7, d c1) (keys 8-15, d c1), transposed on load
          const int key = kb * 16 + (mat & 1) * 8 + mrow;
          const int dchunk = dn * 2 + (mat >> 1);
          uint32_t r0, r1, r2, r3;
          ldmatrix_x4_trans(v_base + (dchunk >> 3) * L::kHalf + swz(key, dchunk & 7), r0, r1, r2, r3);
          mma16816<kBf16>(oacc[2 * dn], pa[kb], r0, r1);
          mma16816<kBf16>(oacc[2 * dn + 1], pa[kb], r2, r3);
        }
      // The stage is refilled through the async proxy: this warp's reads of it have to be over before it is given back.
      // (An earlier form of this kernel, four warps on every tile, released it without the fence: 8 of 100 calls at B = 8, Hk = 4,
      // 1152..4608 keys and 5 of 100 at B = 64, 1024..4096 were off by up to 0.03 from one another.  The fence alone, nothing else
      // changed, made all of them equal and right, although there too an mma.sync had taken every loaded word before the arrive:
      // that the words have been used does not order the reads before the copy.)
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    // finish the row sums across the quad
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
      l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    }
  }

  // ------------------------------------------------------------------ merge the warps
  __syncthreads();  // every tile has been consumed (or the CTA is aborting): the ring is free
  float* scratch = reinterpret_cast<float*>(smem);
  constexpr int kPerWarp = kRows * (D + 2);
  if (warp < kConsumerWarps) {
    float* mine = scratch + warp * kPerWarp;
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const int d = i * 8 + 2 * t4;
      mine[g * D + d] = oacc[i][0];
      mine[g * D + d + 1] = oacc[i][1];
      mine[(g + 8) * D + d] = oacc[i][2];
      mine[(g + 8) * D + d + 1] = oacc[i][3];
    }
    if (t4 == 0) {
      mine[kRows * D + g] = m_run[0];
      mine[kRows * D + g + 8] = m_run[1];
      mine[kRows * D + kRows + g] = l_run[0];
      mine[kRows * D + kRows + g + 8] = l_run[1];
    }
  }
  __syncthreads();
  float m_all = -INFINITY, acc = 0.f, l_all = 0.f;
  auto merge_warps = [&](int r, int d) {
    m_all = -INFINITY;
#pragma unroll
    for (int w = 0; w < kConsumerWarps; ++w) m_all = fmaxf(m_all, scratch[w * kPerWarp + kRows * D + r]);
    const float base = (m_all == -INFINITY) ? 0.f : m_all;
    acc = l_all = 0.f;
#pragma unroll
    for (int w = 0; w < kConsumerWarps; ++w) {  // fixed order
      const float f = ex2(scratch[w * kPerWarp + kRows * D + r] - base);
      acc = fmaf(f, scratch[w * kPerWarp + r * D + d], acc);
      l_all = fmaf(f, scratch[w * kPerWarp + kRows * D + kRows + r], l_all);
    }
  };
  if constexpr (!kClustered) {
    const bool direct = splits == 1 && !force_partial;   // otherwise (O, m, l) goes to `partial`
    float* out_partial = partial + (((size_t)b * gridDim.y + blockIdx.y) * splits + split) * kPerWarp;
    for (int idx = threadIdx.x; idx < rows * D; idx += kThreads) {
      const int r = idx / D, d = idx - r * D;
      merge_warps(r, d);
      if (direct) {
        o[((size_t)b * H + h0 + r) * D + d] = pack1<kBf16>(l_all == 0.f ? 0.f : acc / l_all);  // no valid key: zeros; a score that is NaN or +infinity: NaN
      } else {
        out_partial[r * D + d] = acc;
        if (d == 0) {
          out_partial[kRows * D + r] = m_all;
          out_partial[kRows * D + kRows + r] = l_all;
        }
      }
    }
  } else {
    float* sent = reinterpret_cast<float*>(smem + L::kSent);
    float* sent_stats = sent + L::kSentStats;
    const int share = ((rows * D + splits - 1) / splits + 3) & ~3;   // elements of the output that a CTA of the cluster puts together
    cluster_wait();   // every CTA has started: its shared memory may be written
#pragma unroll 1
    for (int idx = threadIdx.x; idx < rows * D; idx += kThreads) {
      const int r = idx / D, d = idx - r * D, owner = idx / share;
      merge_warps(r, d);
      st_cluster(sent + split * share + idx - owner * share, owner, acc);
      if (d < splits) {   // m and l to CTA d
        st_cluster(sent_stats + split * 2 * kRows + r, d, m_all);
        st_cluster(sent_stats + split * 2 * kRows + kRows + r, d, l_all);
      }
    }
    // After this barrier nobody touches another CTA's memory: no second one before the end.
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll 1
    for (int i = threadIdx.x; i < share && split * share + i < rows * D; i += kThreads) {
      const int idx = split * share + i, r = idx / D, d = idx - r * D;
      float m[kMaxCluster], l[kMaxCluster], a[kMaxCluster];
#pragma unroll
      for (int c = 0; c < kMaxCluster; ++c) {
        const bool there = c < splits;
        m[c] = there ? sent_stats[c * 2 * kRows + r] : -INFINITY;
        l[c] = there ? sent_stats[c * 2 * kRows + kRows + r] : 0.f;
        a[c] = there ? sent[c * share + i] : 0.f;
      }
      m_all = m[0];
#pragma unroll
      for (int c = 1; c < kMaxCluster; ++c) m_all = fmaxf(m_all, m[c]);
      const float base = (m_all == -INFINITY) ? 0.f : m_all;
      acc = l_all = 0.f;
#pragma unroll
      for (int c = 0; c < kMaxCluster; ++c) {
        const float f = ex2(m[c] - base);
        acc = fmaf(f, a[c], acc);
        l_all = fmaf(f, l[c], l_all);
      }
      if (!aborted) o[((size_t)b * H + h0 + r) * D + d] = pack1<kBf16>(l_all == 0.f ? 0.f : acc / l_all);
    }
  }
}

// Combines the per-split partials of one (batch, query head).  `sets` > 1: several partial buffers of the same layout,
// `set_stride` floats apart (one per rank of a cache sharded along the sequence).  The block is D x kMergeLanes threads:
// lane j of a column folds partials j, j + kMergeLanes, ... (sets outer, splits inner) into a running (m, acc, l), four
// independent loads in flight, and the kMergeLanes (8, or 1) running triples are merged in lane order through shared memory -- a
// fixed order, so the result does not depend on timing.  (One thread per column walking 100+ splits in two serial
// passes was the whole cost of long-context decode at small batch: 31 us at Nk = 16384, batch 1.)
// A handful of splits (large batches) is folded by one lane per column: the wide block only costs there.
template <int D, bool kBf16, int kMergeLanes>
__global__ void __launch_bounds__(D * kMergeLanes)
attn_decode_merge_kernel(const float* __restrict__ partial, uint16_t* __restrict__ o, int H, int Hk, int splits, int sets,
                         long long set_stride) {
  constexpr int kPer = kRows * (D + 2);
  __shared__ float sm_m[kMergeLanes][D], sm_a[kMergeLanes][D], sm_l[kMergeLanes][D];
  const int h = blockIdx.x, b = blockIdx.y, d = threadIdx.x % D, j = threadIdx.x / D;
  pdl_wait(partial);
  pdl_launch_dependents();
  const int G = H / Hk;
  const int chunks = (G + kRows - 1) / kRows;
  const int hk = h / G, within = h % G;
  const int slot = hk * chunks + within / kRows, r = within % kRows;
  const float* base_ptr = partial + ((size_t)b * (Hk * chunks) + slot) * splits * kPer;
  float m_run = -INFINITY, acc = 0.f, l_run = 0.f;
  const int total = sets * splits;
#pragma unroll 4
  for (int i = j; i < total; i += kMergeLanes) {
    const int t = i / splits, sp = i - t * splits;
    const float* ps = base_ptr + (size_t)t * set_stride + (size_t)sp * kPer;
    const float m_s = ps[kRows * D + r], l_s = ps[kRows * D + kRows + r], o_s = ps[r * D + d];
    const float m_new = fmaxf(m_run, m_s), base = m_new == -INFINITY ? 0.f : m_new;
    const float keep = ex2(m_run - base), f = ex2(m_s - base);   // ex2(-inf) = 0; a sum that is NaN stays in any case
    acc = fmaf(f, o_s, acc * keep);
    l_run = fmaf(f, l_s, l_run * keep);
    m_run = m_new;
  }
  sm_m[j][d] = m_run; sm_a[j][d] = acc; sm_l[j][d] = l_run;
  __syncthreads();
  if (j == 0) {
    float m_all = -INFINITY;
#pragma unroll
    for (int k = 0; k < kMergeLanes; ++k) m_all = fmaxf(m_all, sm_m[k][d]);
    const float base = m_all == -INFINITY ? 0.f : m_all;
    float a = 0.f, l = 0.f;
#pragma unroll
    for (int k = 0; k < kMergeLanes; ++k) {
      const float f = ex2(sm_m[k][d] - base);
      a = fmaf(f, sm_a[k][d], a);
      l = fmaf(f, sm_l[k][d], l);
    }
    o[((size_t)b * H + h) * D + d] = pack1<kBf16>(l == 0.f ? 0.f : a / l);  // no valid key: zeros; a score that is NaN or +infinity: NaN
  }
}

struct SplitPlan {
  int chunks, splits;
  bool clustered;
};

// How many CTAs share the keys of one (batch, kv head, chunk) group.  Only the capacity of the cache is known here, not the
// valid lengths.  Measured in a graph over 24..256 groups of 300..16384 keys, all lengths equal to the capacity / to half of it /
// spread from a quarter to the whole (us), best of unsplit / clusters of 2..8 / 3..48 splits with a merge kernel:
//   * as many as fit the GPU at once, one per SM, as a cluster of at most eight (8 x 4 groups of 1000..4096: 7.9; three splits
//     and a merge kernel 11.1).  A CTA may have as little as one tile, at D = 64 two from nine tiles on (sum of the three length
//     patterns; 8 groups of 6 tiles: unsplit 12.3, six CTAs 11.6, D = 128 16.4 and 15.2; of 9 tiles: four CTAs 12.4, five 11.7,
//     eight 11.8; D = 128 four 16.4, five 15.6, eight 15.1); of four tiles a group is as quick alone.  Two or three CTAs need
//     longer caches to pay for the merge: 44 groups of 6 tiles 12.9 alone, 13.3 in threes, of 8 tiles 14.0 and 13.5; 64 groups of
//     12 tiles 16.0 alone, 16.2 in pairs, of 16 tiles 17.8 and 17.4.
//   * more groups than clusters of two (74: the SMs come in pairs; 68 groups of 8192: pairs 26.1 / 12.5 / 18.7, unsplit 30.4 /
//     17.0 / 29.9): one CTA each; a second wave of CTAs or half-empty rings cost more than an uneven tail, except (D = 64,
//     three shallow CTAs per SM) where caches are so long that the longest sequence's CTA is on its own for most of the time:
//     80 groups of 16384: clusters of four 53.6 / 30.2 / 40.6, unsplit 59.3 / 31.0 / 55.5; 160 of 8192: pairs 53.8 / 30.8 /
//     40.9, unsplit 62.6 / 34.0 / 55.7.
//   * 45 to 51 groups of very long caches: pairs would leave a third of the SMs idle, six shallow CTAs each do not
//     (48 groups of 16384: 36.1 / 18.8 / 27.4, pairs 35.2 / 19.1 / 32.2).
//   * a handful of groups with long caches (the only plans that write partials, at most one per SM): eight CTAs each leave most
//     of the chip idle, and from 16 tiles of D = 64 per CTA on that costs more than the merge kernel, whose own cost grows with
//     the splits (4 groups of 16384 keys: eight in a cluster 11.4, 16 to 32 and a merge 9.7; 4096 keys: 6.7 and 6.8; one group
//     of 131072: 48 splits 16.3, 148 19.6).
// Where every split writes a partial (`partials`: one shard of a cache split along the sequence) there is no cluster to merge them:
// the partials go through an all-gather and a kernel that reads all ranks', so a CTA keeps two tiles and two or three CTAs need longer
// caches (partials + merge of 1 / of 4 ranks, us, with the lines of clusters and with these: 8 groups of 8 tiles D=128 6.6 / 7.3 and 6.1 /
// 6.9; 24 of 6 7.6 / 10.4 and 7.3 / 7.3; 40 of 8 7.7 / 11.1 and 7.9 / 8.0; 64 of 16 10.9 / 13.8 and 10.2 / 10.7; 24 of 8 D=64 6.0 / 7.3 and
// 5.3 / 6.6; but 8 groups of 7 tiles D=128 7.1 / 7.3 and 7.7 / 7.5).
SplitPlan plan_splits(int B, int H, int Hk, int Nk, int D, bool partials = false) {
  // Clusters of 1..8 CTAs, one per SM, that fit at once: cudaOccupancyMaxActiveClusters gives 148, 74, 45, 33, 26, 22, 15, 15;
  // from three on a little less here, since which SMs a chip has differs.  (With one cluster too many, 16 of eight, 3072 keys
  // took 13 us instead of 9.6.)
  constexpr int kFit[9] = {0, 148, 74, 44, 32, 24, 20, 14, 14};
  // tiles of the capacity, for so many CTAs: as a cluster, and with partials
  constexpr int kLeast[2][9] = {{0, 6, 16, 8, 6, 6, 6, 6, 6}, {0, 8, 24, 12, 8, 10, 12, 14, 16}};
  const int(&kLeastTiles)[9] = kLeast[partials];
  SplitPlan p;
  p.chunks = ceil_div(H / Hk, kRows);
  p.splits = 1;
  p.clustered = false;
  const long long groups = (long long)B * Hk * p.chunks;
  const int tiles = ceil_div(Nk, kTileKeys);
  if (tiles < kLeastTiles[1]) return p;
  int cluster = 1;
  if (D == 64 && groups > kFit[3] && groups <= 51 && tiles >= 256) cluster = 6;
  else if (D == 64 && groups > kFit[2] && groups <= 88 && tiles >= 128) cluster = 4;
  else if (D == 64 && groups > kFit[1] && groups <= 192 && tiles >= 64) cluster = 2;
  else if (groups <= kFit[2]) {
    const int wanted = partials ? tiles / 2 : D == 64 && tiles > 8 ? ceil_div(tiles, 2) : tiles;
    cluster = wanted < kMaxCluster ? wanted : kMaxCluster;
    while (cluster > 1 && groups > kFit[cluster]) --cluster;
    if (tiles < kLeastTiles[cluster]) return p;
  }
  p.splits = cluster;
  p.clustered = cluster > 1;
  const int at_once = sm_count() / (int)groups;
  if (at_once >= 2 * cluster && ceil_div(tiles, cluster) * (D / 64) > 16) {
    const int wanted = ceil_div(tiles, 10) < 48 ? ceil_div(tiles, 10) : 48;
    p.splits = wanted < at_once ? wanted : at_once;
    p.clustered = false;
  }
  return p;
}

template <int D, bool kBf16, int kStages, bool kClustered, bool kOldRows>
int launch_stages(const Problem& p, const SplitPlan& plan, const CUtensorMap& tk, const CUtensorMap& tv, float* partial,
                  unsigned int* status, cudaStream_t stream, bool partial_only);

template <int D, bool kBf16>
int launch_merge_lanes(const float* partial, uint16_t* o, int B, int H, int Hk, int splits, int sets, long long set_stride,
                       cudaStream_t stream) {
  const dim3 grid(H, B);
  if ((long long)splits * sets >= 8)
    return launch_kernel("attn_decode_merge_kernel", attn_decode_merge_kernel<D, kBf16, 8>, grid, dim3(D * 8), 0, stream, partial, o, H, Hk, splits, sets, set_stride);
  return launch_kernel("attn_decode_merge_kernel", attn_decode_merge_kernel<D, kBf16, 1>, grid, dim3(D), 0, stream, partial, o, H, Hk, splits, sets, set_stride);
}

template <int D, bool kBf16>
int launch(const Problem& p, const SplitPlan& plan, const CUtensorMap& tk, const CUtensorMap& tv, float* partial,
           unsigned int* status, cudaStream_t stream, bool partial_only = false) {
  const dim3 grid_probe(plan.splits, p.Hk * plan.chunks, p.B);
  const long long ctas = (long long)grid_probe.x * grid_probe.y * grid_probe.z;
  const bool deep = ctas <= sm_count() && ceil_div(ceil_div(p.Nk, kTileKeys), plan.splits) > shallow_stages<D>();
  constexpr int kDeep = deep_stages<D>(), kShallow = shallow_stages<D>();
  int (*run)(const Problem&, const SplitPlan&, const CUtensorMap&, const CUtensorMap&, float*, unsigned int*, cudaStream_t, bool);
  if (plan.clustered && !partial_only)
    run = p.old_rows ? (deep ? launch_stages<D, kBf16, kDeep, true, true> : launch_stages<D, kBf16, kShallow, true, true>)
                     : (deep ? launch_stages<D, kBf16, kDeep, true, false> : launch_stages<D, kBf16, kShallow, true, false>);
  else
    run = p.old_rows ? (deep ? launch_stages<D, kBf16, kDeep, false, true> : launch_stages<D, kBf16, kShallow, false, true>)
                     : (deep ? launch_stages<D, kBf16, kDeep, false, false> : launch_stages<D, kBf16, kShallow, false, false>);
  return run(p, plan, tk, tv, partial, status, stream, partial_only);
}

template <int D, bool kBf16, int kStages, bool kClustered, bool kOldRows>
int launch_stages(const Problem& p, const SplitPlan& plan, const CUtensorMap& tk, const CUtensorMap& tv, float* partial,
                  unsigned int* status, cudaStream_t stream, bool partial_only) {
  using L = Layout<D, kStages>;
  auto kernel = attn_decode_kernel<D, kBf16, kStages, kClustered, kOldRows>;
  constexpr int kSmem = kClustered ? L::kAlloc : L::kAllocSingle;
  static bool configured[64] = {false};
  int dev = 0;
  KFB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    KFB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(plan.splits, p.Hk * plan.chunks, p.B);
  cfg.blockDim = dim3(L::kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = plan.splits;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = kClustered ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tk, tv, (const uint16_t*)p.q, (uint16_t*)p.o, partial, p.H, p.Hk, p.Nk,
                                     p.scale * 1.4426950408889634f, status, p.kv_len_dev, partial_only ? 1 : 0);
  if (e != cudaSuccess) return fail(KFB_ERR_CUDA, "launch of attn_decode_kernel failed: %s", cudaGetErrorString(e));
  if (kClustered) return KFB_OK;
  if (plan.splits > 1 && !partial_only)
    return launch_merge_lanes<D, kBf16>((const float*)partial, (uint16_t*)p.o, p.B, p.H, p.Hk, plan.splits, 1, 0LL, stream);
  return KFB_OK;
}

}  // namespace

// (the splits of a cluster are merged through shared memory)
size_t decode_ws_bytes(int B, int H, int Hk, int Nk, int D) {
  const SplitPlan plan = plan_splits(B, H, Hk, Nk, D);
  if (plan.splits <= 1 || plan.clustered) return 0;
  return (size_t)B * Hk * plan.chunks * plan.splits * kRows * (D + 2) * sizeof(float);
}

size_t decode_partial_bytes(int B, int H, int Hk, int Nk, int D, int* splits_out) {
  const SplitPlan plan = plan_splits(B, H, Hk, Nk, D, true);
  if (splits_out) *splits_out = plan.splits;
  return (size_t)B * Hk * plan.chunks * plan.splits * kRows * (D + 2) * sizeof(float);
}

int launch_merge(const float* partial, void* o, int dtype, int B, int H, int Hk, int D, int splits, int sets, long long set_stride,
                 cudaStream_t stream) {
  if (H > 65535 || B > 65535) return fail(KFB_ERR_INVALID, "B and H must each be <= 65535");
  const bool bf16 = dtype == KFB_BF16;
  if (D == 64)
    return bf16 ? launch_merge_lanes<64, true>(partial, (uint16_t*)o, B, H, Hk, splits, sets, set_stride, stream)
                : launch_merge_lanes<64, false>(partial, (uint16_t*)o, B, H, Hk, splits, sets, set_stride, stream);
  return bf16 ? launch_merge_lanes<128, true>(partial, (uint16_t*)o, B, H, Hk, splits, sets, set_stride, stream)
              : launch_merge_lanes<128, false>(partial, (uint16_t*)o, B, H, Hk, splits, sets, set_stride, stream);
}

int launch_decode(const Problem& p, void* ws, size_t ws_bytes, cudaStream_t stream, bool partial_only) {
  if (p.Hk * ceil_div(p.H / p.Hk, kRows) > 65535 || p.B > 65535 || p.H > 65535)
    return fail(KFB_ERR_INVALID, "B, H and Hk * ceil(H/Hk/16) must each be <= 65535");
  const SplitPlan plan = plan_splits(p.B, p.H, p.Hk, p.Nk, p.D, partial_only);
  const size_t need = partial_only ? decode_partial_bytes(p.B, p.H, p.Hk, p.Nk, p.D, nullptr) : decode_ws_bytes(p.B, p.H, p.Hk, p.Nk, p.D);
  if (need > 0 && (!ws || ws_bytes < need))
    return fail(KFB_ERR_WORKSPACE, "decode attention needs a %zu-byte workspace, got %zu", need, ws_bytes);
  if (need > 0 && !aligned16(ws)) return fail(KFB_ERR_ALIGNMENT, "workspace must be 16-byte aligned");
  unsigned int* status = device_status_word();
  if (!status) return fail(KFB_ERR_CUDA, "cannot resolve the device status word");
  CUtensorMap tk, tv;
  const uint64_t D = p.D;
  const uint64_t kd[4] = {D, (uint64_t)p.Nk, (uint64_t)p.Hk, (uint64_t)p.B};
  const uint64_t ks[3] = {(uint64_t)p.kv_stride_n * 2, (uint64_t)p.kv_stride_h * 2, (uint64_t)p.kv_stride_b * 2};
  const uint32_t box[4] = {64, kTileKeys, 1, 1};
  if (int rc = make_tmap_4d_sw128(&tk, p.k, p.dtype, kd, ks, box)) return rc;
  if (int rc = make_tmap_4d_sw128(&tv, p.v, p.dtype, kd, ks, box)) return rc;
  const bool bf16 = p.dtype == KFB_BF16;
  float* partial = static_cast<float*>(ws);
  if (p.D == 64)
    return bf16 ? launch<64, true>(p, plan, tk, tv, partial, status, stream, partial_only)
                : launch<64, false>(p, plan, tk, tv, partial, status, stream, partial_only);
  return bf16 ? launch<128, true>(p, plan, tk, tv, partial, status, stream, partial_only)
              : launch<128, false>(p, plan, tk, tv, partial, status, stream, partial_only);
}

}  // namespace attn
}  // namespace kfb

// ------------------------------------------------------------------------------------------------
// Decode attention for callers that must not allocate device memory.
//
// The split-KV kernel above hands its per-split partial results (O, m, l) from the first kernel to
// the merge kernel through a workspace that the caller normally allocates.  Some callers cannot do
// that: a serving loop that has already handed all device memory to its KV-cache pool, code running
// inside a CUDA-graph capture (cudaMalloc is illegal there), or a host runtime that simply has no
// allocator of its own.  For them the partials live in the fixed array below, which is part of the
// library image: every GPU that loads the library holds these kMaxScratchBytes until the process
// exits, whether or not the entry point is ever called.
//
// In host code the NAME of a __device__ array is only a host-side stand-in, not a device address,
// so the address is resolved once per device with cudaGetSymbolAddress (that device being current)
// and that pointer is what the kernels receive.
// ------------------------------------------------------------------------------------------------
#include <mutex>

namespace kfb {
namespace attn {
namespace {

// A plan that is not a cluster's has at most one partial per SM (plan_splits): 1.2 MB on 148 SMs at D = 128.  2 MiB hold 252.
constexpr size_t kMaxScratchBytes = 2u << 20;
static __device__ __align__(256) unsigned char g_decode_scratch[kMaxScratchBytes];

std::mutex g_scratch_mutex;
void* g_scratch_ptr[64] = {nullptr};

// Device address of g_decode_scratch on the current device (resolved on the first call per device).
int static_scratch(void** out) {
  int dev = 0;
  KFB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(KFB_ERR_INVALID, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_decode_scratch);
    if (e != cudaSuccess || !p)
      return fail(KFB_ERR_CUDA, "cudaGetSymbolAddress(decode scratch) failed: %s", cudaGetErrorString(e));
    g_scratch_ptr[dev] = p;
  }
  *out = g_scratch_ptr[dev];
  return KFB_OK;
}

}  // namespace
}  // namespace attn
}  // namespace kfb

extern "C" int kfb_flash_attn_decode_noalloc(const void* q, const void* k, const void* v, void* o, int dtype, int B,
                                             int H, int Hk, int Nk, int D, float scale, const int64_t* kv_strides,
                                             void* stream) {
  using namespace kfb;
  if (int rc = require_sm100()) return rc;
  if (dtype != KFB_F16 && dtype != KFB_BF16) return fail(KFB_ERR_INVALID, "attention takes fp16 or bf16 tensors");
  if (B < 1 || H < 1 || Hk < 1 || Nk < 1) return fail(KFB_ERR_INVALID, "B, H, Hk, Nk must be >= 1");
  if (D != 64 && D != 128) return fail(KFB_ERR_INVALID, "head dim must be one of (64, 128), got %d", D);
  if (H % Hk) return fail(KFB_ERR_INVALID, "query heads (%d) must be a multiple of key/value heads (%d)", H, Hk);
  if (!(scale > 0.0f)) return fail(KFB_ERR_INVALID, "scale must be positive, got %g", (double)scale);
  if (!q || !k || !v || !o) return fail(KFB_ERR_INVALID, "null pointer");
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o))
    return fail(KFB_ERR_ALIGNMENT, "q, k, v, o must be 16-byte aligned");
  const size_t need = attn::decode_ws_bytes(B, H, Hk, Nk, D);
  if (need > attn::kMaxScratchBytes)
    return fail(KFB_ERR_WORKSPACE,
                "this problem needs %zu bytes of split-KV scratch but the built-in array holds %zu; "
                "use kfb_flash_attn_fwd with a caller-provided workspace",
                need, attn::kMaxScratchBytes);
  attn::Problem p;
  p.q = q; p.k = k; p.v = v; p.o = o;
  p.dtype = dtype; p.B = B; p.H = H; p.Hk = Hk; p.Nq = 1; p.Nk = Nk; p.D = D;
  p.causal = 0;  // a single query at the last position sees every key
  p.scale = scale;
  if (kv_strides) {
    p.kv_stride_b = kv_strides[0]; p.kv_stride_h = kv_strides[1]; p.kv_stride_n = kv_strides[2];
    if (p.kv_stride_n < D || p.kv_stride_h < 1 || p.kv_stride_b < 1 || (p.kv_stride_b % 8) || (p.kv_stride_h % 8) ||
        (p.kv_stride_n % 8))
      return fail(KFB_ERR_ALIGNMENT, "kv strides must be positive multiples of 8 elements with a row stride >= D");
  } else {
    p.kv_stride_n = D; p.kv_stride_h = (long long)Nk * D; p.kv_stride_b = (long long)Hk * Nk * D;
  }
  void* scratch = nullptr;
  if (int rc = attn::static_scratch(&scratch)) return rc;
  // Every partial the merge kernel reads is written by the split kernel of the same call, so
  // nothing left in the array by an earlier call is ever consumed and nothing needs clearing.
  return attn::launch_decode(p, scratch, attn::kMaxScratchBytes, (cudaStream_t)stream);
}
