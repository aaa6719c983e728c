// Internal interface between the attention C-ABI entry point (flash_attn.cu) and the two kernels.
#pragma once

#include "common.cuh"

namespace kfb {
namespace attn {

struct Problem {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  int dtype;  // KFB_F16 / KFB_BF16
  int B, H, Hk, Nq, Nk, D;
  int causal;
  float scale;
  long long kv_stride_b, kv_stride_h, kv_stride_n;  // elements
  // prefill only: strides of q and o in elements (D axis dense); n = 0 means dense [B, H, Nq, D]
  long long q_stride_b = 0, q_stride_h = 0, q_stride_n = 0;
  long long o_stride_b = 0, o_stride_h = 0, o_stride_n = 0;
  // decode only: device array of B valid lengths (<= Nk, the capacity of the cache); nullptr = all Nk keys
  const int* kv_len_dev = nullptr;
  // decode only: kv_len_dev and all valid rows but the last are older than the kernel in front (kfb_flash_attn_decode_step)
  bool old_rows = false;
};

// Prefill / general path: tiles of 128 query rows, TMA + tcgen05 + TMEM (attn_prefill.cu).  The workspace is optional: a
// problem with few tiles is split along the keys when it has prefill_ws_bytes bytes (enough with and without the causal mask).
size_t prefill_ws_bytes(int B, int H, int Hk, int Nq, int Nk, int D);
// The plan that launch_prefill takes with a workspace of ws_bytes.
void prefill_plan(const Problem& p, size_t ws_bytes, int* tiles_per_cta, int* splits);
int launch_prefill(const Problem& p, void* ws, size_t ws_bytes, cudaStream_t stream);

// Decode path (Nq == 1): split-KV, one CTA per (batch, kv head, split) (attn_decode.cu).
size_t decode_ws_bytes(int B, int H, int Hk, int Nk, int D);
int launch_decode(const Problem& p, void* ws, size_t ws_bytes, cudaStream_t stream, bool partial_only = false);
// Partial results only (no merge, no output): bytes of the (O, m, l) buffer and the number of key splits per
// (batch, kv-head slot); and the merge of `sets` such buffers, `set_stride` floats apart, into the output.
size_t decode_partial_bytes(int B, int H, int Hk, int Nk, int D, int* splits_out);
int launch_merge(const float* partial, void* o, int dtype, int B, int H, int Hk, int D, int splits, int sets, long long set_stride,
                 cudaStream_t stream);

}  // namespace attn
}  // namespace kfb
