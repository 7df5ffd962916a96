// What the kernels of attention with one or two softmax maps per head share: their arguments, masks, the cap on scores, gates.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace sprout_maps {

// The first position that a query at `pos` sees: 0 (causal), pos - size + 1 (a window of `size` positions, itself
// included) or the start of its chunk of `size` positions counted from position 0.
// `keep` (a window only): the first `keep` positions stay visible to every later query, at their own positions.
enum MaskKind : int { MASK_CAUSAL = 0, MASK_WINDOW = 1, MASK_CHUNK = 2 };
// cap * tanh(s / cap) for the bfloat16 kernel: through one exponential, absolute error about cap * 2e-7
__device__ __forceinline__ float soft_cap_fast(float s, float cap, float inv_cap) {
  const float e = __expf(2.0f * s * inv_cap);
  return cap * (1.0f - __fdividef(2.0f, e + 1.0f));
}
__device__ __forceinline__ int first_visible(int kind, int size, int pos) {
  if (kind == MASK_WINDOW) return max(0, pos - size + 1);
  if (kind == MASK_CHUNK) return pos < 0 ? 0 : (pos / size) * size;
  return 0;
}

// Where the packed rows of a request begin whose first query of the step stands at `first`: at the 64-position boundary at or before
// the first position that any of its queries sees.
__device__ __forceinline__ int packed_base(int kind, int size, int first) { return first_visible(kind, size, first) & ~63; }

// Turns a head's output back by the query's position (values that were turned by theirs): tables float32
// [positions, vdim / 2]; null: no turn.  Pair m is (m, m + vdim / 2), or (2m, 2m + 1) when `interleaved`.
struct OutputTurn {
  const float* cos; const float* sin; int positions, interleaved;
};

struct MultiMapParams {
  const __nv_bfloat16* q; int q_stride;
  const __nv_bfloat16* k_cache; const __nv_bfloat16* v_cache;
  const int* block_table; int table_stride;
  const int* q_start; const int* positions;
  __nv_bfloat16* out; int out_stride;
  int requests, heads, kv_heads, page_tokens, num_pages;
  float scale, lambda, norm_eps, out_scale;
  int* status;
  // single-token steps may divide a request's tiles among `ksplit` CTAs (blockIdx.z); each then leaves its maxima, sums
  // and unnormalised accumulators in `partial` [requests, kv_heads, ksplit, 16 rows, maps, 2 + vdim] for the merge kernel
  int ksplit; float* partial;
  // what a query sees (MaskKind and its size), an optional term exp(sink[head]) in every softmax denominator, and an
  // optional gate: the head's output times sigmoid(gate[token * gate_stride + head])
  int mask_kind, mask_size; const float* sink; const __nv_bfloat16* gate; int gate_stride;
  // a window's kept first positions, and the cap on the scaled scores (0: none)
  int mask_keep; float softcap;
  // the gate row holds a number per element of the output instead of one per head; the turn back of the output
  int gate_elements; OutputTurn turn;
};

// A gate per element: sigmoid of the gate row's number for column `col` of the head's output.
__device__ __forceinline__ float element_gate(const MultiMapParams& p, int token, int head, int vdim, int col) {
  return 1.0f / (1.0f + __expf(-__bfloat162float(p.gate[(size_t)token * p.gate_stride + (size_t)head * vdim + col])));
}

// What the running maxima are multiplied by on their way into the exponentials: capped scores are already scaled.
__device__ __forceinline__ float score_scale(const MultiMapParams& p) { return p.softcap > 0.f ? 1.0f : p.scale; }

}  // namespace sprout_maps

// Prompt portions on tcgen05 (attention_maps_tcgen05.cu).
extern "C" int sprout_maps_attention_tc_supported(int maps, int dim, int vdim, int page_tokens, int out_stride);
int sprout_maps_attention_tc(const sprout_maps::MultiMapParams& m, int tokens, int maps, int dim, int vdim, float* scratch, int* counters,
                             cudaStream_t stream);
