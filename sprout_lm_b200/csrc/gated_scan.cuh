// What the gated scan's kernels share (gated_recurrence.cu walks token by token, gated_scan_mma.cu 16 tokens at a time on tensor cores).
#pragma once

#include "common.cuh"

namespace sprout_scan {

enum ScanDecay : int { DECAY_PER_CHANNEL = 0, DECAY_PER_HEAD = 1, DECAY_GIVEN = 2, DECAY_FLOOR = 3, DECAY_BONUS = 4 };
enum ScanPhase : int { SCAN_WHOLE = 0, SCAN_CHUNK_SUMS = 1, SCAN_CHUNK_OUT = 2 };

template <typename T>
struct ScanParams {
  const T* q; int q_stride;            // [tokens, groups * dim]
  const T* k; int k_stride;            // [tokens, groups * dim]
  const T* v; int v_stride;            // [tokens, heads * vdim]
  const void* z; int z_stride, z_f32;  // per channel: [tokens, heads * dim]; per head: [tokens, heads]; of T, or float when z_f32
  const float* bias;                   // added to z: [heads * dim] or [heads]
  const float* a_log;                  // per head (per-head decay only); with a floor: the floors [heads * dim]
  const float* skip;                   // per head, or null
  const float* bonus;                  // [heads * dim] (DECAY_BONUS only)
  float inv_tau, q_scale;
  int mode, heads, groups, dim, vdim;
  const int* q_start; const int* state_slots; float* state; int num_slots;
  float* out;                          // [tokens, heads * vdim]
  int* status;
  // portions cut into chunks (null / 0 when every request's tokens are walked by one block):
  const float* da;                     // decays made beforehand: [tokens, heads * dim] per channel, [tokens, heads] per head
  const float* dc;                     // per head: the factor on k, [tokens, heads]
  float* sums;                         // [max_chunks, heads, dim, vdim]: a chunk's own sums, then the state before the chunk
  float* prods;                        // [max_chunks, heads, dim]: the product of a chunk's decays
  int chunk, requests;
  int q_silu;                          // silu on the query rows (with a floor only)
  int v_cols, ones_col;                // columns the value rows really have (<= vdim); column v_cols of the state is fed 1
};

// The chunks of all requests are numbered in the requests' order, ceil(tokens / chunk) each.  Finds chunk `index`:
// its request, its place among the request's chunks and how many the request has; false beyond the last chunk.
__device__ __forceinline__ bool find_chunk(const int* q_start, int requests, int chunk, int index, int& r, int& c, int& n) {
  for (int i = 0; i < requests; i++) {
    n = (q_start[i + 1] - q_start[i] + chunk - 1) / chunk;
    if (index < n) { r = i; c = index; return true; }
    index -= n;
  }
  return false;
}

// gated_scan_mma.cu: whether it takes these sizes, forms and addresses, and its walks over the chunks (SCAN_CHUNK_SUMS or SCAN_CHUNK_OUT).
bool scan_mma_takes(const ScanParams<__nv_bfloat16>& p);
int launch_scan_mma(const ScanParams<__nv_bfloat16>& p, int phase, int max_chunks, cudaStream_t stream);

}  // namespace sprout_scan
