// The routed experts' activation, shared by their products' kernels.
#pragma once

#include "common.cuh"

namespace sprout_experts {

// What an expert does with its first products: the clamped gated unit, the exact gelu of one product (an expert without a
// gate), silu(g) u.
enum ExpertUnit : int { UNIT_CLAMPED = 0, UNIT_PLAIN = 1, UNIT_SILU = 2 };
__device__ __forceinline__ float glu(int unit, float g, float u, float limit, float alpha) {
  if (unit == UNIT_PLAIN) return 0.5f * g * (1.0f + erff(g * 0.7071067811865476f));
  if (unit == UNIT_SILU) return g / (1.0f + expf(-g)) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g * (1.0f / (1.0f + expf(-alpha * g))) * (u + 1.0f);
}

}  // namespace sprout_experts

// One of the experts' products on tcgen05 in CTA pairs (experts_tcgen05.cu): rows [entries, K] bfloat16 arranged by expert (`offsets`
// [experts + 1]), w [experts, matrix rows, K].  GLU or gelu units (`unit` >= 0): out bfloat16 [entries, N], the matrix has 2 N rows
// (gate rows, then up rows) or for UNIT_PLAIN N; `row_weights` (of entry order[row]) multiply the products before the activation.
// `unit` -1: out float32 [entries, N], the products as they are.  `offsets` null: one expert that has every row.
int sprout_experts_product_tc(const void* rows, int row_stride, const int* offsets, const int* order, const void* w, void* out, int entries, int experts, int N,
                              int K, int unit, const float* row_weights, float limit, float alpha, int* status, cudaStream_t stream);
