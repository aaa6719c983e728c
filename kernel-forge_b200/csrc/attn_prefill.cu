// Fused attention forward for sm_100a, general path (any Nq, Nk; GQA; bottom-right causal mask).
//
// Replaces attn_v4_kernel of the reference (csrc/attention/attn_v4_kernel.cuh:43-214), which is an
// mma.sync / ldmatrix / cp.async kernel.  One kernel built on the Blackwell execution model (TMA into
// 128-byte-swizzled shared-memory tiles, tcgen05.mma issued by one thread, accumulators in TMEM), with two
// tiles of 128 query rows per CTA or one, and a merge kernel for key splits.
//
// Thread r of a softmax warpgroup owns query row r = TMEM lane r, so row maximum and
// row sum need no shuffles; lazy rescale (the running base of a row only moves when the new maximum
// exceeds it by more than 8 in log2 units -- a factor 256, far inside fp32 range -- and only then is
// O in TMEM rescaled; O and l always share one base, so O / l is unaffected); causal: key steps above
// the diagonal are never loaded or multiplied (loop bound), masking only on the diagonal / ragged
// steps, query tiles are scheduled heaviest-first (query tile is the slowest-varying grid index,
// reversed); GQA: kv head = h / (H / Hk); TMA zero-fills rows past Nq / Nk, those keys are masked.
//
// Numerics (as the reference, attn_v4_kernel.cuh:133-213): scores accumulate in FP32; x = s *
// (scale * log2 e); masked = -inf; p = 2^(x - base); the row sum adds the unrounded p, the PV
// product uses p rounded to fp16/bf16; O / l rounded once.  2^x is ex2.approx.ftz.f32 or a
// polynomial of the same accuracy.
#include "attn.cuh"
#include "sm100.cuh"

#include <algorithm>

namespace kfb {
namespace attn {
namespace {

using namespace sm100;

constexpr int kBlockM = 128;
constexpr int kBlockN = 128;   // keys per TMA tile and per step
constexpr int kHalfBytes = kBlockN * 128;  // one 64-column half of a tile: 128 rows x 128 bytes
constexpr float kRescaleThreshold = 8.0f;  // log2 units

enum WaitCode : uint32_t {
  kWaitQ = 0x101, kWaitKEmpty, kWaitKFull, kWaitVEmpty, kWaitVFull, kWaitSFull, kWaitPReady, kWaitPvDone, kWaitIssuer, kWaitTurn
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// three-input maximum (one instruction on sm_100); NaN if any of the three is
__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
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

// Launch order of the 1-D grid.  (batch, head) pairs are taken in groups of `heads_per_group` whose K/V fit in L2
// together; inside a group the query tile (or tile pair) index is the slower one and runs from the last tile to the
// first, so that under a causal mask every long tile of the group starts before any short one, while the CTAs
// resident at one time still share the K/V of few heads.  (Heaviest-first over ALL heads at once made the resident
// CTAs stream the K/V of every head at the same time: at N = 8192, D = 128 that is 134 MB, more than L2.)
struct TileOrder {
  int q_index, bh;
};
struct Strides {   // of the output, in elements; the D axis is dense
  long long b, h, n;
};
__device__ __forceinline__ TileOrder decode_tile_order(unsigned int block, int n_q, int bh_total, int heads_per_group) {
  const unsigned int per_group = (unsigned int)n_q * (unsigned int)heads_per_group;
  const int group = (int)(block / per_group);
  const int base = group * heads_per_group;
  const int size = min(heads_per_group, bh_total - base);
  const int r = (int)(block - (unsigned int)group * per_group);
  return TileOrder{n_q - 1 - r / size, base + r % size};
}

// ------------------------------------------------------------------------------------------------
// NT = 2: one CTA per SM owns two tiles (A and B) of 128 query rows that attend to one KV head, steps of 128 keys.  384
// threads (three warpgroups; warp 11 only takes part in barriers):
//   warps 0-3  softmax of tile A, warps 4-7 softmax of tile B (warp w touches TMEM lanes 32 (w % 4)..);
//   warp 8     TMA producer: both Q tiles once, then K and V tiles of 128 keys through mbarrier rings;
//   warps 9,10 issue the tcgen05.mma of tile A / tile B.  The warp stays uniform and one elected lane issues: addresses and
//              descriptors are then uniform registers (inside `if (lane == 0)` every MMA costs ~95 clocks of moves into
//              them); it sleeps in blocking waits, because polling takes issue slots from two of the softmax warps.
// NT = 1: one tile, 192 threads (warps 0-3, 4, 5), half of the TMEM columns, two CTAs per SM: smaller pieces, for grids
// that would leave SMs idle (plan_prefill).  kDouble (head dim 128): one tile with the SM to itself and two buffers of scores.
// TMEM: S_X [128 X, +128), then head dim 64: O_X [128 NT + 64 X, +64), P_X [192 NT + 64 X, +64);  head dim 128: P_X on the first
// 64 columns of S_X, O_X [128 NT + 128 X, +128);  kDouble: S(j) [128 (j % 2), +128), P(j) on its first 64 columns, O [256, +128)
// Both tiles read the same K/V tiles, so each is brought into shared memory once for 256 query rows.
//
// What a tile's rows are.  Two or more query tiles per head: 128 consecutive queries of one head, tiles A and B neighbours.
// At most 128 queries per head and grouped heads: `heads_per_tile` heads of a group x all Nq queries, so that a tile is as
// full as it gets and K/V is read once for the group (16 queries of 8 heads are one tile, not eight).
//
// What bounds it: the exponentials (a 128 x 128 tile costs 1024 clocks of the SM's exponential units) and, at head dim
// 128, equally the tensor pipe (1024 clocks per tile and step).  Either is reached only if a softmax warp never waits, so
// its own chain -- scores, maximum, exponentials, P, PV, next QK -- is what counts:
//   * exponentials do not wait for the maximum of their step: they are taken with the base of the steps before, while the
//     maxima of the row run under them, and in a step whose maximum outgrows the base they are taken again (the results are those
//     of looking first).  One row of a warp's 32 is enough for that, so with scores of a standard deviation of 6 (natural units)
//     every second step is such a step.  The first of four chunks is taken ahead, two in head dim 128 CTAs of two tiles, where the
//     baton makes one chunk too short, and of two score buffers, where one costs short calls more than it gives (us, scores of
//     deviation 1 / 3 / 6, looking first - two chunks ahead - one: 2 x 16 x 2048 D=64 56.9 / 58.5 / 61.6 - 53.1 / 58.6 / 72.8 - 52.9 /
//     55.8 / 64.0; 4 heads x 5806 causal D=64 45.2 / 45.7 / 47.8 - 44.0 / 48.8 / 63.7 - 44.4 / 45.4 / 52.3; 1 x 16 x 2048 causal D=128
//     33.3 / 33.8 / 35.4 - 27.0 / 28.5 / 33.0 - 27.0 / 28.1 / 31.7; 2 x 16 x 314 causal D=128 8.8 / 8.9 / 9.2 - 7.8 / 8.3 / 9.1 - 8.0 / 8.2 /
//     8.8; 2 x 16 x 2048 D=128 73.9 / 75.4 / 80.1 - 68.0 / 75.7 / 96.5 - 73.6 / 79.1 / 95.8).  Going back to looking first after two grown steps in a row helps
//     there (92.5 at 6, 85 at 30 instead of 98) but costs every call (8192 causal 550 us -> 556).  Only the first step looks first;
//   * the scores are loaded in chunks of 32, one ahead.  Head dim 64 releases the S buffer after the last, and QK(j+1) runs
//     under step j; P has columns of its own;
//   * head dim 128: P(j) overwrites half of S(j), so QK(j+1) can only follow PV(j).  P is handed over in two halves, and
//     PV starts on the first 64 keys while the exponentials of the others run.  With two buffers (kDouble) QK(j+1) is
//     complete before step j ends and the softmax warps never wait for a product;
//   * two tiles of a CTA take turns on the exponential units (a "baton"): one tile's exponentials run under the other's score
//     load, P store and products.  Left alone the tiles fall into step and compete for the same unit;
//   * head dim 64 computes some exponentials on the FMA pipe (exp_pair_fma), which is idle otherwise.
// What is left (clocks of one step of 128 keys, stamps of the clock in a copy of the kernel, two tiles at head dim 128): 3200 for
// the pair of tiles, each 1200 from its last P to its next scores and 1640 of exponentials (1024 at the unit's rate; a single
// warp per scheduler reaches 86 % of it), which overlap with the other tile's.
// Measured (us in a graph, before -> after the exponentials stopped waiting, one-tile CTAs with an SM to themselves got two
// buffers and head dim 64 one-tile CTAs wherever keys are not split): B=2 H=16 N=2048 D=64 58.0 -> 53.9 (back to back, at the power limit,
// 58.7 -> 57.8), N=8192 701 -> 651; 32 x 32 heads
// x 200 tokens D=64 causal 50.6 -> 45.3; N=2048 D=128 75.4 -> 69.8; N=8192 D=128 causal 495 -> 471 (577 -> 549 back to back at the
// power limit's clock); 1 x 16 x 2048 D=128 causal 34.0 -> 29.5; 509 queries on 4093 keys, 12 heads over 2, D=128 26.5 -> 23.5.
// Also measured: D=64, N=2048, two tiles per CTA 56.8, without baton 58.1; two pairs of 16 by polynomial 56.7, four 57.2; the last
// chunk of scores read twice, to save registers, 55.3; the first step on the path that takes exponentials again (registers spill) 73.  D=128, N=2048 (70.0): no baton 86.7, baton after two chunks 83.7, after
// four 75.1; one polynomial pair in 16 73.7; P handed over in three pieces 70.6.  Registers: head dim 64 spills 12 bytes (two tiles 16),
// head dim 128 28 in CTAs of two tiles, none in the others.
//
// Split over keys: a problem with few tiles (short chunks against a long cache) is cut along the keys too; a CTA then
// writes its unnormalised O and (m, l) per row and attn_prefill_merge_kernel puts the pieces together in order.
// ------------------------------------------------------------------------------------------------
namespace tiles {

constexpr int kPolyPairs = 3;       // head dim 64: of 16 pairs of scores, this many take exp_pair_fma

template <int D, int NT, bool kDouble>
struct TileLayout {
  static constexpr int kProducerWarp = 4 * NT, kMmaWarp = 4 * NT + 1;   // (then one issuer warp per tile)
  static constexpr int kThreads = NT == 2 ? 384 : 192;
  static constexpr uint32_t kTmemCols = kDouble ? 512u : 256u * NT;
  static constexpr bool kAliasP = D == 128;
  static constexpr int kHalves = kAliasP ? 2 : 1;     // pieces in which P is handed to the tensor cores
  static constexpr int kScores = kDouble ? 2 : 1;     // buffers of scores
  static constexpr int kStages = kDouble ? 2 : D == 64 ? 2 * NT : NT;
  static constexpr int kTile = kBlockN * D * 2;       // bytes of one 128-row tile (Q, K or V)
  static constexpr int kQ = 0;                        // Q_A, Q_B
  static constexpr int kK = NT * kTile;
  static constexpr int kV = kK + kStages * kTile;
  static constexpr int kBars = kV + kStages * kTile;
  static constexpr int kNumBars = 1 + 4 * kStages + 12;
  static constexpr int kMisc = kBars + kNumBars * 8;
  static constexpr int kBytes = kMisc + 16;
  static constexpr int kAlloc = kBytes + 1024;        // room to align the tiles to 1024 bytes
  static constexpr int kAllocAlone = kDouble ? kAlloc : 116 * 1024;   // more than half of what an SM has
  static_assert(!kDouble || (NT == 1 && kAliasP), "for a tile whose P lies on its scores; two tiles leave no room in TMEM");
  static_assert((NT == 1 && !kDouble ? 2 : 1) * kAlloc <= 227 * 1024, "two one-tile CTAs, or a two-tile CTA, must fit on an SM");
  static_assert((NT == 1 && !kDouble) || 2 * kAlloc > 228 * 1024, "one CTA per SM where it allocates all 512 TMEM columns");
  static constexpr uint32_t kColS = 0;                              // + 128 X (+ 128 for the second buffer)
  static constexpr uint32_t kColO = 128 * NT * kScores;             // + D X
  static constexpr uint32_t kColP = kAliasP ? 0u : 192u * NT;       // + (kAliasP ? 128 : 64) X
  static constexpr uint32_t kStrideP = kAliasP ? 128u : 64u;
};

struct Params {
  int B, H, Hk, Nq, Nk, causal;
  float scale_log2;
  int heads_per_tile;    // 0: a tile is 128 queries of one head; else that many heads x all Nq queries
  int tiles;             // tiles of a unit: a (batch, head), or a (batch, KV head) with heads_per_tile
  int units_per_group;   // launch order, see decode_tile_order
  int splits;            // pieces of the key range
  float* partial;        // splits > 1: [split][B H Nq][D] floats, then [split][B H Nq][2] (m in log2 units, l)
};

// Columns c0 .. c0 + 31 past `limit` (causal diagonal / ragged end) become -inf.
__device__ __forceinline__ void mask32(uint32_t (&v)[32], int c0, int limit) {
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (c0 + i > limit) v[i] = 0xFF800000u;
}

// Running maxima of 32 scores: four independent chains of three-input maxima.
__device__ __forceinline__ void max32(const uint32_t (&v)[32], float (&mx)[4]) {
#pragma unroll
  for (int i = 0; i < 32; i += 2) mx[(i >> 1) & 3] = max3(mx[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
}
__device__ __forceinline__ float max_of(const float (&mx)[4]) { return max3(max3(mx[0], mx[1], mx[2]), mx[3], mx[3]); }

// Two scores, p = 2^(x * scale - base), rounded to the I/O type into one register; the unrounded p are added to `sum`.
// Scale-and-subtract and the sums use the two-wide FP32 instructions of sm_100 (results per element are those of the scalar
// forms).
template <bool kBf16>
__device__ __forceinline__ uint32_t exp_pair(uint32_t v0, uint32_t v1, float2 sc2, float2 nb2, float2& sum) {
  const float2 x = __ffma2_rn(make_float2(__uint_as_float(v0), __uint_as_float(v1)), sc2, nb2);
  const float2 e = make_float2(ex2(x.x), ex2(x.y));
  sum = __fadd2_rn(sum, e);
  return pack2<kBf16>(e.x, e.y);
}

constexpr float kExp2C1 = 0.693146944f, kExp2C2 = 0.240221202f, kExp2C3 = 0.0555071346f, kExp2C4 = 0.00967554096f,
                kExp2C5 = 0.00132764538f;

// The same on the FMA pipe instead of the exponential unit: 2^x = 2^r 2^f with r = rint(x), f in [-1/2, 1/2] (Cody and
// Waite's reduction), 2^f by a degree-5 polynomial fitted for least relative error there (2^-22, like ex2.approx), r added
// to the exponent.  x below -125 counts as -125: far below the last bit of any sum it enters.  So does NaN: rows with a
// score that is NaN or +infinity are told by their maximum instead (see l_run).
template <bool kBf16>
__device__ __forceinline__ uint32_t exp_pair_fma(uint32_t v0, uint32_t v1, float2 sc2, float2 nb2, float2& sum) {
  float2 x = __ffma2_rn(make_float2(__uint_as_float(v0), __uint_as_float(v1)), sc2, nb2);
  x.x = fmaxf(x.x, -125.0f);
  x.y = fmaxf(x.y, -125.0f);
  auto both = [](float c) { return make_float2(c, c); };
  const float2 t = __fadd2_rn(x, both(12582912.0f));   // 1.5 * 2^23: the low bits are rint(x)
  const float2 f = __ffma2_rn(__fadd2_rn(t, both(-12582912.0f)), both(-1.0f), x);
  float2 y = __ffma2_rn(both(kExp2C5), f, both(kExp2C4));
  y = __ffma2_rn(y, f, both(kExp2C3));
  y = __ffma2_rn(y, f, both(kExp2C2));
  y = __ffma2_rn(y, f, both(kExp2C1));
  y = __ffma2_rn(y, f, both(1.0f));
  y.x = __uint_as_float(__float_as_uint(y.x) + (__float_as_uint(t.x) << 23));
  y.y = __uint_as_float(__float_as_uint(y.y) + (__float_as_uint(t.y) << 23));
  sum = __fadd2_rn(sum, y);
  return pack2<kBf16>(y.x, y.y);
}

template <int D, bool kBf16, int NT, bool kDouble>
__global__ void __launch_bounds__(TileLayout<D, NT, kDouble>::kThreads, NT == 2 || kDouble ? 1 : 2)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                         const __grid_constant__ CUtensorMap tm_v, void* __restrict__ o_ptr, const Strides o_st,
                         const __grid_constant__ Params pr, unsigned int* status) {
  using L = TileLayout<D, NT, kDouble>;
  constexpr int S = L::kStages, kHalves = L::kHalves;
  constexpr bool kAliasP = L::kAliasP;
  constexpr bool kBaton = NT == 2;               // the two tiles take turns
  constexpr int kGuess = D == 128 && (NT == 2 || kDouble) ? 2 : 1;   // chunks whose exponentials do not wait for the step's maximum
  constexpr int kOrder = D == 64 && NT == 1 ? 7 : 5;    // pairs of a chunk are taken in the order e * kOrder (see chunk)
  constexpr int kBatonAfter = kAliasP ? 2 : 1;   // the chunk after which the other tile may start
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = k_full + S;
  uint64_t* v_full = k_empty + S;
  uint64_t* v_empty = v_full + S;
  uint64_t* s_full = v_empty + S;    // [X]: S_X written by QK
  uint64_t* s_free = s_full + 2;     // [X]: all 128 threads of tile X hold their scores in registers
  uint64_t* p_ready = s_free + 2;    // [X][half]: P_X stored by all 128 threads
  uint64_t* pv_done = p_ready + 4;   // [X]: the PV product that read P_X has completed (O_X updated)
  uint64_t* turn = pv_done + 2;      // [X]: the baton: X may start its exponentials
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kMisc);
  volatile uint32_t* abort_word = tmem_slot + 1;
  const AbortCtx ctx{abort_word, status};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int H = pr.H, Hk = pr.Hk, Nq = pr.Nq, Nk = pr.Nk, causal = pr.causal, hpt = pr.heads_per_tile;
  const int per_batch = hpt ? Hk : H;   // units of a batch item
  const TileOrder ord = decode_tile_order(blockIdx.x, (pr.tiles + NT - 1) / NT, pr.B * per_batch, pr.units_per_group);
  const int tile0 = NT * ord.q_index;
  const int b = ord.bh / per_batch, within = ord.bh - b * per_batch;
  const int hk = hpt ? within : within / (H / Hk);
  const int causal_off = Nk - Nq;
  const bool has_b = NT == 2 && tile0 + 1 < pr.tiles;
  // first head and first query of tile X
  auto head_of = [&](int X) { return hpt ? hk * (H / Hk) + (tile0 + X) * hpt : within; };
  auto query_of = [&](int X) { return hpt ? 0 : (tile0 + X) * kBlockM; };
  int n_steps[2];
#pragma unroll
  for (int X = 0; X < 2; ++X) {
    int kv_end = Nk;
    if (causal && !hpt) kv_end = min(Nk, min(query_of(X) + kBlockM, Nq) + causal_off);
    n_steps[X] = X == 0 || has_b ? (kv_end + kBlockN - 1) / kBlockN : 0;
  }
  // this CTA's steps [j0, j0 + n_max) of the key range; tile X takes part in the first n_of(X) of them
  int j0 = 0, n_max = max(n_steps[0], n_steps[1]);
  if (pr.splits > 1) {
    const int per = (n_max + pr.splits - 1) / pr.splits;
    j0 = blockIdx.y * per;
    n_max = max(0, min(n_max - j0, per));
  }
  auto n_of = [&](int X) { return max(0, min(n_steps[X] - j0, n_max)); };

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < S; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], NT);   // one arrival per issuer
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], NT);
    }
    for (int X = 0; X < 2; ++X) {
      mbar_init(&s_full[X], 1);
      mbar_init(&s_free[X], 128);
      mbar_init(&p_ready[2 * X], 128);
      mbar_init(&p_ready[2 * X + 1], 128);
      mbar_init(&pv_done[X], 1);
      mbar_init(&turn[X], 128);
    }
    *abort_word = *reinterpret_cast<volatile unsigned int*>(status);  // a wait expired earlier on this device:
    fence_mbar_init();                                                // do no work, return at once
  }
  if (warp == L::kMmaWarp) {   // the first issuer warp also owns the TMEM allocation
    tmem_alloc(tmem_slot, L::kTmemCols);
    tmem_relinquish();
  }
  if (warp == L::kProducerWarp && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_wait();   // every role: from here on memory of the kernel in front is read (and what it reads may be overwritten)
  pdl_launch_dependents();
  const uint32_t tmem_base = *tmem_slot;
  const bool dead_on_arrival = *abort_word != 0;

  // Two tiles: registers move from the warpgroup of the three single-warp roles to the softmax warpgroups, which keep
  // the 128 scores of a row in registers (2 x 128 x 208 + 128 x 88 = 64512 of 65536).  Each role branch
  // starts with its setmaxnreg, executed by all four warps of its warpgroup.
  if (dead_on_arrival) {
    // fall through to the teardown
  } else if (warp >= L::kProducerWarp) {
    if constexpr (NT == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == L::kProducerWarp) {
      // ---------------------------------------------------------------- TMA producer
      if (lane == 0 && n_max > 0) {
        const int tiles = has_b ? 2 : 1;
        const int q_rows = hpt ? hpt * Nq : kBlockM;   // rows a Q copy brings (hpt: the box is hpt heads x Nq queries)
        mbar_arrive_expect_tx(q_full, (uint32_t)(tiles * q_rows * D * 2));
        for (int X = 0; X < tiles; ++X)
#pragma unroll
          for (int half = 0; half < D / 64; ++half)
            tma_load_4d(smem + L::kQ + X * L::kTile + half * kHalfBytes, &tm_q, q_full, half * 64, query_of(X), head_of(X), b);
        for (int i = 0; i < n_max; ++i) {
          const int s = i % S, key0 = (j0 + i) * kBlockN;
          const uint32_t ph = (uint32_t)(i / S) & 1u;
          if (!mbar_wait(&k_empty[s], ph ^ 1u, ctx, kWaitKEmpty)) break;
          mbar_arrive_expect_tx(&k_full[s], L::kTile);
#pragma unroll
          for (int half = 0; half < D / 64; ++half)
            tma_load_4d(smem + L::kK + s * L::kTile + half * kHalfBytes, &tm_k, &k_full[s], half * 64, key0, hk, b);
          if (!mbar_wait(&v_empty[s], ph ^ 1u, ctx, kWaitVEmpty)) break;
          mbar_arrive_expect_tx(&v_full[s], L::kTile);
#pragma unroll
          for (int half = 0; half < D / 64; ++half)
            tma_load_4d(smem + L::kV + s * L::kTile + half * kHalfBytes, &tm_v, &v_full[s], half * 64, key0, hk, b);
        }
      }
    } else if (warp < L::kMmaWarp + NT) {
      // ---------------------------------------------------------------- tcgen05.mma issuers (one warp per tile)
      // The two warps never touch each other's TMEM columns.  A K / V stage goes back to the producer when BOTH have
      // arrived on its `empty` barrier (count 2): a tile that does not need a key tile (no tile B, or one step less under
      // a causal mask) still arrives for it once it has been loaded.
      const int X = warp - L::kMmaWarp;
      constexpr uint32_t idesc_qk = idesc_f16(kBlockM, kBlockN, kBf16 ? 1 : 0, 0, 0);
      constexpr uint32_t idesc_pv = idesc_f16(kBlockM, D, kBf16 ? 1 : 0, 0, 1);
      const uint64_t q_desc = smem_desc_sw128(smem_u32(smem + L::kQ) + (uint32_t)X * L::kTile, 16, 1024);
      const uint64_t k_desc = smem_desc_sw128(smem_u32(smem + L::kK), 16, 1024);
      const uint64_t v_desc = smem_desc_sw128(smem_u32(smem + L::kV), kHalfBytes, 1024);
      const uint32_t s_col = tmem_base + L::kColS + 128u * X, o_col = tmem_base + L::kColO + (uint32_t)D * X;
      const uint32_t p_col = tmem_base + L::kColP + L::kStrideP * X;
      const int n = n_of(X);
      constexpr int kAhead = kDouble ? 2 : 1;   // steps by which the scores of an aliased P are ahead of its products
      bool ok = true;
      auto wait_for = [&](uint64_t* bar, uint32_t parity, uint32_t code) {
        ok = ok && __all_sync(0xffffffffu, mbar_wait(bar, parity, ctx, code));
        return ok;
      };
      // S(j) = Q K(j)^T
      auto await_k = [&](int j) { return wait_for(&k_full[j % S], (uint32_t)(j / S) & 1u, kWaitKFull); };
      auto qk = [&](int j) {   // K(j) has been awaited
        const int s = j % S, buf = kDouble ? j & 1 : 0;
        tc_fence_after_sync();
        const uint64_t kd = k_desc + (uint64_t)(s * (L::kTile >> 4));
        if (ok && elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint64_t off = (uint64_t)(((kk / 4) * kHalfBytes + (kk % 4) * 32) >> 4);
            mma_ss(s_col + 128u * buf, q_desc + off, kd + off, idesc_qk, kk > 0 ? 1u : 0u);
          }
          tc_commit(&s_full[kDouble ? buf : X]);
        }
        __syncwarp();
      };
      // O += P(j) V(j), in kHalves pieces of the 128 keys
      auto pv = [&](int j) {
        const int s = j % S;
        const uint32_t p_at = p_col + (kDouble ? 128u * (j & 1) : 0u);
        constexpr int kPer = kBlockN / 16 / kHalves;
        if (!wait_for(&v_full[s], (uint32_t)(j / S) & 1u, kWaitVFull)) return;
        const uint64_t vd = v_desc + (uint64_t)(s * (L::kTile >> 4));
#pragma unroll
        for (int half = 0; half < kHalves; ++half) {
          // (the next product follows at once: its keys are awaited before the last piece of P)
          if (half + 1 == kHalves && kAliasP && j + kAhead < n && !await_k(j + kAhead)) return;
          if (!wait_for(&p_ready[2 * (kDouble ? j & 1 : X) + half], (uint32_t)(kDouble ? j >> 1 : j) & 1u, kWaitPReady)) return;
          tc_fence_after_sync();
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kPer; ++kk) {
              // 16 keys per MMA: 16 rows of 128 bytes; the second 64-column block of V is kHalfBytes away
              const int k = half * kPer + kk;
              mma_ts(o_col, p_at + (uint32_t)k * 8u, vd + (uint64_t)(k * (2048 >> 4)), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
            }
            // (aliased P, one buffer: S(j + 1) complete implies PV(j) complete, so only the last step needs a commit of its own)
            if (half + 1 == kHalves && (!kAliasP || kDouble || j + 1 == n)) tc_commit(&pv_done[X]);
          }
          __syncwarp();
        }
      };
      auto release = [&](uint64_t* bar) {
        if (ok && elect_one()) tc_commit(bar);
        __syncwarp();
      };
      // A commit keeps the issuing thread for some 50-130 clocks, so the ones that only return a stage come last.
      if (n > 0) {
        wait_for(q_full, 0, kWaitQ);
        for (int j = 0; j < kAhead && j < n; ++j) {
          if (await_k(j)) qk(j);
          release(&k_empty[j % S]);
        }
        for (int j = 0; ok && j < n; ++j) {
          const int next = j + kAhead;
          if (!kAliasP && next < n) {   // S(j + 1) as soon as the scores of step j are in registers
            await_k(next);
            wait_for(&s_free[X], (uint32_t)j & 1u, kWaitSFull);
            qk(next);
          }
          pv(j);
          if (kAliasP && next < n) qk(next);   // tcgen05.mma instructions of one thread execute in issue order
          release(&v_empty[j % S]);
          if (next < n) release(&k_empty[next % S]);
        }
      }
      for (int j = n; ok && j < n_max; ++j) {   // steps that only the other tile has: hand the stages on once filled
        const int s = j % S;
        const uint32_t ph = (uint32_t)(j / S) & 1u;
        if (wait_for(&k_full[s], ph, kWaitKFull) && elect_one()) mbar_arrive(&k_empty[s]);
        __syncwarp();
        if (wait_for(&v_full[s], ph, kWaitVFull) && elect_one()) mbar_arrive(&v_empty[s]);
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (warps 0-7)
    if constexpr (NT == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int X = warp >> 2;                      // which tile
    const int row = threadIdx.x & 127;            // query row inside the tile == TMEM lane
    const int head = head_of(X) + (hpt ? row / Nq : 0);
    const int query = hpt ? row % Nq : query_of(X) + row;
    const bool real = (X == 0 || has_b) && (hpt ? row < hpt * Nq : query < Nq);
    const int n = n_of(X);
    const uint32_t lane_bits = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_tmem = tmem_base + L::kColS + 128u * X + lane_bits;
    const uint32_t p_tmem = tmem_base + L::kColP + L::kStrideP * X + lane_bits;
    const uint32_t o_tmem = tmem_base + L::kColO + (uint32_t)D * X + lane_bits;
    const int row_limit = causal ? min(Nk - 1, query + causal_off) : Nk - 1;   // last visible key of this row
    const int tile_limit = causal ? min(Nk - 1, query_of(X) + causal_off) : Nk - 1;   // ... of the tile's first row
    const float2 sc2 = make_float2(pr.scale_log2, pr.scale_log2);
    float m_base = -INFINITY;  // the base O and l are currently expressed in (log2 units)
    float l_run = 0.f;
    bool ok = true;
    auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t code) {   // every lane polls: faster than one and a shuffle
      ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, ctx, code));
      return ok;
    };
    auto wait_turn = [&](int i) { return wait_all(&turn[X], (X == 1 ? (uint32_t)i : (uint32_t)i + 1u) & 1u, kWaitTurn); };
    // With two buffers of scores those of the next step are there before this one ends: their first chunk of 32 is requested
    // then.  (Head dim 64, whose next product has only been started in the middle of the step, two tiles: 62.0 us with that, 57.0
    // without.)
    constexpr bool kPrefetch = kDouble;
    uint32_t v[4][32];         // the 128 scores of this row
    auto await_scores = [&](int i) {
      if (!wait_all(&s_full[kDouble ? i & 1 : X], (uint32_t)(kDouble ? i >> 1 : i) & 1u, kWaitSFull)) return false;
      tc_fence_after_sync();
      return true;
    };
    auto fetch = [&](int i, int c) { tmem_ld_x32(s_tmem + (kDouble ? 128u * (i & 1) : 0u) + c * 32, v[c]); };
    if (kPrefetch && n > 0 && await_scores(0)) fetch(0, 0);
    for (int i = 0; ok && i < n; ++i) {
      const uint32_t ph = (uint32_t)i & 1u;
      const uint32_t p_at = p_tmem + (kDouble ? 128u * (i & 1) : 0u);
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      const int k0 = (j0 + i) * kBlockN;
      const bool masked = k0 + kBlockN - 1 > tile_limit;
      auto mask = [&](int c) {
        if (masked) mask32(v[c], c * 32, row_limit - k0);
      };
      if (!kPrefetch) {
        if (!await_scores(i)) break;
        fetch(i, 0);
      }
      tmem_wait_ld_regs(v[0]);
      fetch(i, 1);
      fetch(i, 2);
      fetch(i, 3);
      mask(0);
      if (i == 0) {   // the first step has no base to guess with
        tmem_wait_ld_regs(v[1]);
        tmem_wait_ld_regs(v[2]);
        tmem_wait_ld_regs(v[3]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c > 0) mask(c);
          max32(v[c], mx);
        }
        m_base = max_of(mx) * pr.scale_log2;
      }
      float base = (m_base == -INFINITY) ? 0.f : m_base;
      if (kBaton && (X == 1 || i > 0) && !wait_turn(i)) break;
      float2 nb2 = make_float2(-base, -base);
      float2 sum[2] = {{0.f, 0.f}, {0.f, 0.f}};
      uint32_t p[4][16];
      auto expo = [&](int c, int e) {
        if (!kAliasP && e < kPolyPairs) p[c][e] = exp_pair_fma<kBf16>(v[c][2 * e], v[c][2 * e + 1], sc2, nb2, sum[e & 1]);
        else p[c][e] = exp_pair<kBf16>(v[c][2 * e], v[c][2 * e + 1], sc2, nb2, sum[e & 1]);
      };
      auto seen = [&](int c, int e) { mx[e & 3] = max3(mx[e & 3], __uint_as_float(v[c][2 * e]), __uint_as_float(v[c][2 * e + 1])); };
      // The order spreads the polynomials among the others.  (7 instead of 5 in head dim 64 one-tile CTAs: 53.8 us -> 52.9 at 2 x 16 x
      // 2048, fewer registers spilled; in two-tile CTAs 5 is the better one, 44.5 and 45.6 at 4 heads x 5806 causal.)
      auto chunk = [&](int c) {
#pragma unroll
        for (int e = 0; e < 16; ++e) expo(c, (e * kOrder) & 15);
      };
      auto pass_baton = [&]() {   // (the operands keep the exponentials summed so far in front of it)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0]; // %1 %2" ::"r"(smem_u32(&turn[X ^ 1])), "f"(sum[0].x), "f"(sum[1].x) : "memory");
      };
      // The maxima run under the exponentials of the first kGuess chunks, which are taken with the base of the steps before: it
      // only moves when a maximum outgrows it by more than the threshold, and then they are taken again.
      auto land = [&]() {
        tmem_wait_ld_regs(v[1]);
        tmem_wait_ld_regs(v[2]);
        tmem_wait_ld_regs(v[3]);
        if (i > 0) {
          mask(1);
          mask(2);
          mask(3);
        }
      };
      if constexpr (kGuess == 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          expo(0, (e * kOrder) & 15);
          seen(0, e);
        }
        land();
#pragma unroll
        for (int e = 8; e < 16; ++e) {
          expo(0, (e * kOrder) & 15);
          seen(0, e);
#pragma unroll
          for (int x = 2 * e - 16; x < 2 * e - 14; ++x) {
            seen(1, x);
            seen(2, x);
            seen(3, x);
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          if (e == 16) land();
          expo(e / 16, (e * kOrder) & 15);
          if (e < 16) {
            seen(0, e);
          } else {
            seen(1, e - 16);
            seen(2, e - 16);
            seen(3, e - 16);
          }
        }
      }
      const float m_step = max_of(mx) * pr.scale_log2;
      // lazy rescale: move the base only when the maximum outgrew it by more than the threshold
      // (-inf + 8 = -inf: the first finite maximum counts.)  Rows of a tile that are no query's do not count: where heads share a tile
      // they hold what was in shared memory before (2 x 32 heads over 4, 2 queries on 422 keys, D=64 8.2 us and 6.9, D=128 9.1 and 7.9).
      const bool grow = real && m_step > m_base + kRescaleThreshold;
      float alpha = 1.0f;
      // PV(j-1) must have finished accumulating before O is rescaled, and reading before P is overwritten.  (One buffer with
      // aliased P: S(j) complete implies PV(j-1) complete.)
      bool pv_waited = (kAliasP && !kDouble) || i == 0;
      auto wait_pv = [&]() {
        if (!pv_waited) {
          if (!wait_all(&pv_done[X], ph ^ 1u, kWaitPvDone)) return false;
          pv_waited = true;
        }
        tc_fence_after_sync();
        return true;
      };
      if (__any_sync(0xffffffffu, grow)) {   // (not in the first step)
        // O is rescaled between PV(j-1) and PV(j), which cannot have started (it waits for this step's P).  Rare after the
        // first steps.
        if (grow) {
          alpha = ex2(m_base - m_step);  // 0 when m_base is still -inf
          m_base = m_step;
        }
        if (!wait_pv()) break;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld_x32(o_tmem + c * 32, o);
          tmem_wait_ld_regs(o);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
          tmem_st_x32(o_tmem + c * 32, o);
        }
        base = (m_base == -INFINITY) ? 0.f : m_base;
        nb2 = make_float2(-base, -base);
        sum[0] = sum[1] = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < kGuess; ++c) fetch(i, c);
#pragma unroll
        for (int c = 0; c < kGuess; ++c) {
          tmem_wait_ld_regs(v[c]);
          mask(c);
        }
#pragma unroll
        for (int c = 0; c < kGuess; ++c) chunk(c);
      }
      if (kGuess == 1) chunk(1);
      if constexpr (!kAliasP) {   // the S buffer can take the next product already
        tc_fence_before_sync();
        mbar_arrive(&s_free[X]);
      }
      // (two buffers of scores: only so that the wait after the last step is for one phase)
      if (kDouble && i + 1 == n && !wait_pv()) break;
      if constexpr (kAliasP) {
        tmem_st_x16(p_at, p[0]);
        tmem_st_x16(p_at + 16, p[1]);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(&p_ready[2 * (kDouble ? i & 1 : X)]);
      }
      if (kBaton && kBatonAfter == 1) pass_baton();
      chunk(2);
      if constexpr (kAliasP) tmem_st_x16(p_at + 32, p[2]);
      if (kBaton && kBatonAfter == 2) pass_baton();
      chunk(3);
      if constexpr (kAliasP) tmem_st_x16(p_at + 48, p[3]);
      const float2 t = __fadd2_rn(sum[0], sum[1]);
      // A score that is NaN or +infinity makes its row NaN, whichever way its exponential was taken.
      l_run = m_step < INFINITY ? fmaf(l_run, alpha, t.x + t.y) : __int_as_float(0x7FFFFFFF);
      if constexpr (!kAliasP) {   // (each chunk stored on its own, as above, is slower here: 61.5 us at 2 x 16 x 2048)
        if (!wait_pv()) break;
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_st_x16(p_at + 16 * c, p[c]);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(&p_ready[2 * (kDouble ? i & 1 : X) + kHalves - 1]);
      if (kPrefetch && i + 1 < n) {
        if (!await_scores(i + 1)) break;
        fetch(i + 1, 0);
      }
    }
    for (int i = n; kBaton && ok && i < n_max; ++i) {   // steps that only the other tile has: pass the baton on
      if ((X == 1 || i > 0) && !wait_turn(i)) break;
      mbar_arrive(&turn[X ^ 1]);
    }
    // PVs complete in issue order: the last one done means all are
    if (ok && n > 0) wait_all(&pv_done[X], kAliasP && !kDouble ? 0u : (uint32_t)(n - 1) & 1u, kWaitPvDone);
    if (ok) {
      tc_fence_after_sync();
      const long long grow_row = ((long long)b * H + head) * Nq + query;   // row of the dense [B H Nq] order of the partials
      const long long rows = (long long)pr.B * H * Nq;
      const bool part = pr.splits > 1;
      float* o32 = part ? pr.partial + ((long long)blockIdx.y * rows + grow_row) * D : nullptr;
      uint8_t* dst = static_cast<uint8_t*>(o_ptr) + (b * o_st.b + head * o_st.h + query * o_st.n) * 2;
      if (part && real)
        reinterpret_cast<float2*>(pr.partial + pr.splits * rows * D)[(long long)blockIdx.y * rows + grow_row] = make_float2(m_base, l_run);
      if (n > 0) {
        const float inv_l = 1.0f / l_run;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld_x32(o_tmem + c * 32, o);
          tmem_wait_ld_regs(o);
          if (real && part) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              reinterpret_cast<uint4*>(o32 + c * 32)[e] = make_uint4(o[4 * e], o[4 * e + 1], o[4 * e + 2], o[4 * e + 3]);
          } else if (real) {
            uint32_t packed[16];
#pragma unroll
            for (int e = 0; e < 16; ++e)
              packed[e] = pack2<kBf16>(__uint_as_float(o[2 * e]) * inv_l, __uint_as_float(o[2 * e + 1]) * inv_l);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              reinterpret_cast<uint4*>(dst + c * 64)[e] =
                  make_uint4(packed[4 * e], packed[4 * e + 1], packed[4 * e + 2], packed[4 * e + 3]);
          }
        }
      }
    }
  }

  // teardown: every role falls through to here, also after an expired wait
  if (!dead_on_arrival && *abort_word != 0) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);  // let copies in flight land
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == L::kMmaWarp) {
    __syncwarp();
    tmem_dealloc(tmem_base, L::kTmemCols);
  }
}

// o[row] = sum over splits of 2^(m_s - m) O_s[row] / sum of 2^(m_s - m) l_s, in split order.  A row per D / 4 threads.
template <int D, bool kBf16>
__global__ void __launch_bounds__(256) attn_prefill_merge_kernel(const float* __restrict__ partial, void* __restrict__ o_ptr, const Strides o_st,
                                                                 int H, int Nq, long long rows, int splits) {
  pdl_wait(partial);
  pdl_launch_dependents();
  constexpr int kPerRow = D / 4;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x, row = idx / kPerRow;
  const int c = (int)(idx % kPerRow) * 4;
  if (row >= rows) return;
  const float2* ml = reinterpret_cast<const float2*>(partial + splits * rows * D);
  float m = -INFINITY;
  for (int s = 0; s < splits; ++s) m = fmaxf(m, ml[s * rows + row].x);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float l = 0.f;
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float2 w = ml[s * rows + row];
    if (w.x == -INFINITY && !isnan(w.y)) continue;   // no step of this split reached the row (its O was not written)
    const float f = ex2(w.x - m);
    const float4 v = *reinterpret_cast<const float4*>(partial + (s * rows + row) * D + c);
    acc.x = fmaf(f, v.x, acc.x); acc.y = fmaf(f, v.y, acc.y); acc.z = fmaf(f, v.z, acc.z); acc.w = fmaf(f, v.w, acc.w);
    l = fmaf(f, w.y, l);
  }
  const float inv = 1.0f / l;
  const long long bh = row / Nq;
  uint8_t* dst = static_cast<uint8_t*>(o_ptr) + (bh / H * o_st.b + bh % H * o_st.h + (row - bh * Nq) * o_st.n + c) * 2;
  *reinterpret_cast<uint2*>(dst) = make_uint2(pack2<kBf16>(acc.x * inv, acc.y * inv), pack2<kBf16>(acc.z * inv, acc.w * inv));
}

}  // namespace tiles

// How a problem is cut (see the header of the kernel); max_splits = 1 where there is no workspace for the pieces.
struct PrefillPlan {
  int heads_per_tile, tiles, units, per_cta, splits;
  bool alone;   // a one-tile CTA that has its SM to itself
};

PrefillPlan plan_prefill(const Problem& p, int max_splits = 32) {
  PrefillPlan c;
  const int G = p.H / p.Hk, q_tiles = ceil_div(p.Nq, kBlockM), sms = sm_count();
  c.heads_per_tile = 0;
  c.tiles = q_tiles;
  c.units = p.B * p.H;
  if (q_tiles == 1 && G > 1) {
    c.heads_per_tile = 1;
    for (int d = 2; d <= G; ++d)
      if (G % d == 0 && d * p.Nq <= kBlockM) c.heads_per_tile = d;
    c.tiles = G / c.heads_per_tile;
    c.units = p.B * p.Hk;
  }
  // Tiles per CTA, CTAs per SM and key splits, by a cost model in us fitted to 700 shapes, 4713 measured plans in graphs on
  // B200 (mean deviation 4 % at head dim 64, 9 % at 128; the plan it picks is on average 0.5 % slower than the best one measured,
  // before the fit to these kernels 4 %): a CTA takes `step` per 128 keys and `fixed` for set-up and drain; the merge kernel
  // 2.4 or 3.2, 0.2 or 0.3 per split and its traffic at 5.1 TB/s.  So a grid smaller than the GPU takes one tile per CTA and may
  // split the keys (1 x 12 heads x 509 queries, 4093 keys, D = 128: three splits 23.5 us, two tiles per CTA in six 26.2), long
  // ones share K / V between two tiles (2 x 16 x 2048 D = 128: 70.6 against 75.6 for one in pairs, 101 for one apart).
  // One-tile CTAs fit in pairs on an SM, and the hardware does pair them while other SMs stay idle.  Where the grid has at
  // most one for each SM, and under a causal mask also for longer grids, where short CTAs even out what is left over, they are
  // kept apart: at D = 128 with the TMEM of the whole SM (1 x 16 x 2048 causal: in pairs 35.9, apart 29.5), at D = 64, where
  // that gains nothing, by the shared memory they ask for (1 x 4 heads x 7: in pairs 4.5, apart 4.1).
  struct Kind {
    int per_cta;
    bool alone;
    double step, fixed, wave, tail;   // wave: `fixed` where CTAs follow one another on an SM; tail: share of the longest CTA that
  };                                  // a causal grid of more CTAs than slots ends with
  const bool wide = p.D == 128;
  const Kind kinds[3] = {{1, false, wide ? 2.06 : 1.44, wide ? 4.5 : 3.8, wide ? 6.5 : 4.6, wide ? 0.24 : 0.17},
                         {1, true, wide ? 1.33 : 0.97, wide ? 3.7 : 3.6, wide ? 4.0 : 3.9, wide ? 0.24 : 0.33},
                         {2, false, wide ? 1.80 : 1.46, wide ? 3.9 : 3.3, wide ? 4.7 : 4.4, wide ? 0.39 : 0.20}};
  const int steps = ceil_div(p.Nk, kBlockN), hidden = ceil_div(p.Nk - p.Nq, kBlockN);   // hidden: steps that every causal tile has
  const bool uneven = p.causal && !c.heads_per_tile && p.Nq > p.Nk / 2;   // CTAs of all lengths, longest first
  const double merge_us = (double)p.B * p.H * p.Nq * p.D * 8.0 / 5.1e6 + (wide ? 0.30 : 0.22);
  double best = 1e30;
  c.per_cta = 1;
  c.splits = 1;
  c.alone = false;
  for (const Kind& k : kinds)
    for (int s = 1; s <= steps && s <= max_splits; ++s) {
      const int longest = ceil_div(steps, s);
      if (ceil_div(steps, longest) != s) continue;   // an empty split
      const int per_unit = ceil_div(c.tiles, k.per_cta);
      const long long ctas = (long long)c.units * per_unit * s;
      if (s > 1 && ctas > 2 * sms) break;
      if (k.per_cta == 1 && !k.alone && ctas <= sms) continue;
      if (k.alone && ctas > sms && (wide ? longest < 6 : s > 1 || longest < 8)) continue;
      // Two tiles per CTA: not for short CTAs (D = 128, 320 of at most four steps: 37.2 us, in pairs of one tile 34.1), and at D = 64
      // only where the keys are split (2 x 16 x 8192: 694 us, one tile 664; 4 heads x 5806 causal: two splits 45.0, one tile 50.6)
      if (k.per_cta == 2 && (longest < 5 || (!wide && s == 1))) continue;
      const long long slots = k.per_cta == 2 || k.alone ? sms : 2 * sms;
      const double one = longest * k.step + k.fixed;
      double cost = one;
      if (ctas > slots && uneven && per_unit > 1) {
        const double total = (double)c.units * (k.per_cta * (per_unit - 1.0) * per_unit / 2 + (per_unit - 1.0) * hidden + steps);
        const double shared = (total * k.step + ctas * k.wave) / slots + k.tail * longest * k.step;
        cost = one > shared ? one : shared;
      } else if (ctas > slots) {   // (the last wave of pairs: CTAs on their own where there is an SM for each)
        const long long last = ctas % slots;
        const Kind& left = slots > sms && last <= sms ? kinds[1] : k;
        cost = (double)(ctas / slots) * (longest * k.step + k.wave) + (last ? longest * left.step + left.wave : 0.0);
      }
      if (s > 1) {
        double merge = (wide ? 3.2 : 2.4) + s * merge_us;
        // Pieces of one step have a cheaper kernel, which counts where they are few and short of rows (4 steps, in one piece and in four:
        // 2 x 32 heads over 4 x 2 queries 7.9 and 7.5, 8 heads x 20 7.6 and 7.4, 32 heads x 4 7.85 and 7.77, but 8 heads x 100 8.4 and 9.0).
        if (wide && k.alone && longest == 1) merge = std::min(merge, 1.8 + s * (0.43 + 2.5 * (merge_us - 0.30)));
        cost += merge;
      }
      if (cost < best) { best = cost; c.per_cta = k.per_cta; c.splits = s; c.alone = k.alone; }
    }
  return c;
}

template <int D, bool kBf16, int NT, bool kDouble>
int launch_tiles(const Problem& p, const PrefillPlan& plan, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, float* partial,
                 unsigned int* status, cudaStream_t stream) {
  using L = tiles::TileLayout<D, NT, kDouble>;
  auto kernel = tiles::attn_prefill_kernel<D, kBf16, NT, kDouble>;
  static bool configured[64] = {false};
  int dev = 0;
  KFB_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    KFB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NT == 1 ? L::kAllocAlone : L::kAlloc));
    configured[dev] = true;
  }
  const Strides o_st{p.o_stride_b, p.o_stride_h, p.o_stride_n};
  // units whose K and V (one KV head each at worst) fit in ~48 MB of L2 together
  const long long kv_bytes_per_unit = 4LL * p.Nk * p.D;
  const int units_per_group = (int)std::min<long long>(plan.units, std::max<long long>(1, (48LL << 20) / kv_bytes_per_unit));
  const long long ctas = (long long)plan.units * ceil_div(plan.tiles, NT);
  if (ctas > 0x7fffffffLL) return fail(KFB_ERR_INVALID, "too many query tiles for one launch");
  tiles::Params pr = {p.B, p.H, p.Hk, p.Nq, p.Nk, p.causal, p.scale * 1.4426950408889634f, plan.heads_per_tile, plan.tiles, units_per_group,
                     plan.splits, partial};
  if (int rc = launch_kernel("attn_prefill_kernel", kernel, dim3((unsigned)ctas, plan.splits), dim3(L::kThreads), plan.alone ? L::kAllocAlone : L::kAlloc, stream, tq, tk, tv,
                             p.o, o_st, pr, status))
    return rc;
  if (plan.splits == 1) return KFB_OK;
  const long long rows = (long long)p.B * p.H * p.Nq, blocks = (rows * (D / 4) + 255) / 256;
  return launch_kernel("attn_prefill_merge_kernel", tiles::attn_prefill_merge_kernel<D, kBf16>, dim3((unsigned)blocks), dim3(256), 0, stream,
                       (const float*)partial, p.o, o_st, p.H, p.Nq, rows, plan.splits);
}

template <int D, bool kBf16>
int launch(const Problem& p, const PrefillPlan& plan, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, float* partial,
           unsigned int* status, cudaStream_t stream) {
  if (plan.per_cta == 2) return launch_tiles<D, kBf16, 2, false>(p, plan, tq, tk, tv, partial, status, stream);
  if constexpr (D == 128) {
    // A second buffer of scores has a use from two steps of keys on.  One step, us in a graph, two buffers and one: 88 heads of 3 tokens
    // 5.17 and 4.92, 128 heads of 60 5.54 and 5.34, 32 heads of 128 5.20 and 4.99; two steps, 16 heads of 200 tokens 6.13 and 6.22.
    const bool one_step = ceil_div(ceil_div(p.Nk, kBlockN), plan.splits) == 1;
    if (plan.alone && !one_step) return launch_tiles<D, kBf16, 1, true>(p, plan, tq, tk, tv, partial, status, stream);
  }
  return launch_tiles<D, kBf16, 1, false>(p, plan, tq, tk, tv, partial, status, stream);
}

size_t partial_bytes(const Problem& p, const PrefillPlan& plan) {
  return plan.splits > 1 ? (size_t)plan.splits * p.B * p.H * p.Nq * (p.D + 2) * sizeof(float) : 0;
}

}  // namespace

size_t prefill_ws_bytes(int B, int H, int Hk, int Nq, int Nk, int D) {
  Problem p = {};
  p.B = B; p.H = H; p.Hk = Hk; p.Nq = Nq; p.Nk = Nk; p.D = D;
  const size_t full = partial_bytes(p, plan_prefill(p));
  p.causal = 1;   // (its plan may have more splits)
  const size_t causal = partial_bytes(p, plan_prefill(p));
  return full > causal ? full : causal;
}

void prefill_plan(const Problem& p, size_t ws_bytes, int* tiles_per_cta, int* splits) {
  PrefillPlan plan = plan_prefill(p);
  if (ws_bytes < partial_bytes(p, plan)) plan = plan_prefill(p, 1);   // the workspace is optional
  *tiles_per_cta = plan.per_cta;
  *splits = plan.splits;
}

int launch_prefill(const Problem& given, void* ws, size_t ws_bytes, cudaStream_t stream) {
  Problem p = given;
  if (p.q_stride_n == 0) { p.q_stride_n = p.D; p.q_stride_h = (long long)p.Nq * p.D; p.q_stride_b = (long long)p.H * p.Nq * p.D; }
  if (p.o_stride_n == 0) { p.o_stride_n = p.D; p.o_stride_h = (long long)p.Nq * p.D; p.o_stride_b = (long long)p.H * p.Nq * p.D; }
  unsigned int* status = device_status_word();
  if (!status) return fail(KFB_ERR_CUDA, "cannot resolve the device status word");
  PrefillPlan plan = plan_prefill(p);
  if (!ws || !aligned16(ws) || ws_bytes < partial_bytes(p, plan)) plan = plan_prefill(p, 1);   // the workspace is optional
  CUtensorMap tq, tk, tv;
  const uint64_t D = p.D;
  const uint64_t qd[4] = {D, (uint64_t)p.Nq, (uint64_t)p.H, (uint64_t)p.B};
  const uint64_t qs[3] = {(uint64_t)p.q_stride_n * 2, (uint64_t)p.q_stride_h * 2, (uint64_t)p.q_stride_b * 2};
  const uint64_t kd[4] = {D, (uint64_t)p.Nk, (uint64_t)p.Hk, (uint64_t)p.B};
  const uint64_t ks[3] = {(uint64_t)p.kv_stride_n * 2, (uint64_t)p.kv_stride_h * 2, (uint64_t)p.kv_stride_b * 2};
  const uint32_t box[4] = {64, 128, 1, 1};
  const uint32_t qbox[4] = {64, plan.heads_per_tile ? (uint32_t)p.Nq : 128u, plan.heads_per_tile ? (uint32_t)plan.heads_per_tile : 1u, 1};
  if (int rc = make_tmap_4d_sw128(&tq, p.q, p.dtype, qd, qs, qbox)) return rc;
  if (int rc = make_tmap_4d_sw128(&tk, p.k, p.dtype, kd, ks, box)) return rc;
  if (int rc = make_tmap_4d_sw128(&tv, p.v, p.dtype, kd, ks, box)) return rc;
  const bool bf16 = p.dtype == KFB_BF16;
  float* partial = static_cast<float*>(ws);
  if (p.D == 64)
    return bf16 ? launch<64, true>(p, plan, tq, tk, tv, partial, status, stream) : launch<64, false>(p, plan, tq, tk, tv, partial, status, stream);
  return bf16 ? launch<128, true>(p, plan, tq, tk, tv, partial, status, stream) : launch<128, false>(p, plan, tq, tk, tv, partial, status, stream);
}

}  // namespace attn
}  // namespace kfb
