// Rows of bfloat16 in 16-byte pieces as float32, and the rotation of two pieces.
#pragma once

#include "attention_bf16.cuh"

namespace sprout_attn {

__device__ __forceinline__ void unpack8(uint4 raw, float (&v)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// a, b: the runs that turn together; angles `at` on (8 of them): pairs (a[i], b[i]), or with `interleaved` neighbours of a, then of b.
__device__ __forceinline__ void turn16(float (&a)[8], float (&b)[8], const float* cos_at, const float* sin_at, bool interleaved) {
  float c[8], s[8];
  load8(cos_at, c);
  load8(sin_at, s);
  if (interleaved) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float x = a[2 * i], y = a[2 * i + 1], z = b[2 * i], w = b[2 * i + 1];
      a[2 * i] = x * c[i] - y * s[i]; a[2 * i + 1] = y * c[i] + x * s[i];
      b[2 * i] = z * c[4 + i] - w * s[4 + i]; b[2 * i + 1] = w * c[4 + i] + z * s[4 + i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float x = a[i], y = b[i];
      a[i] = x * c[i] - y * s[i];
      b[i] = y * c[i] + x * s[i];
    }
  }
}

}  // namespace sprout_attn
