// out[m, n] = sum_k A[m, k] * W[n, k] (+ bias[n]) (+ residual[m, n]) on CUDA cores with
// float32 fused multiply-adds: the matrix product of the true 32-bit path (no tensor cores,
// no reduced-precision mode), and a plain reference for the tensor-core kernels.  Each output
// element is accumulated by one thread in ascending k, so its value does not depend on how
// many rows the call has, on where a row sits among them, or on the tile that a call's sizes pick.
//
// Bound by the fused multiply-adds and the shared-memory reads that feed them.  A thread holds TM x TN sums as pairs of
// neighbouring columns for the packed `fma.rn.f32x2` (two IEEE fused multiply-adds an instruction, A's value doubled in registers);
// both operands lie in shared memory as [k][row], the next k's values are read while one k is multiplied, and the next
// k-block's 16-byte loads are in flight meanwhile.  K cannot be split (the order of the additions is fixed), so what
// fills the device is the tile: see `launch_sizes`.
#include "common.cuh"

namespace {

__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ unsigned long long twice(float a) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
  return d;
}

// Four neighbouring elements of a row as float32.
__device__ __forceinline__ float4 load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 raw = *(const uint2*)p;
  return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                     __uint_as_float(raw.y & 0xffff0000u));
}

// Elements k .. k + 3 of a row of K elements, zeros beyond its end or for a row that does not exist.  VEC: the row starts on a
// boundary of four elements and K is a multiple of four.
template <bool VEC, typename T>
__device__ __forceinline__ float4 fetch(const T* row, bool exists, int k, int K) {
  if (!exists) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (VEC) return k < K ? load4(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(k < K ? to_float(row[k]) : 0.f, k + 1 < K ? to_float(row[k + 1]) : 0.f, k + 2 < K ? to_float(row[k + 2]) : 0.f,
                     k + 3 < K ? to_float(row[k + 3]) : 0.f);
}

template <int BM, int BN, int BK, int TM, int TN, bool VEC, typename TA, typename TW, typename TO>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simple_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias,
                   const float* residual, TO* out, int M, int N, int K, int lda, int ldo) {
  constexpr int THREADS = (BM / TM) * (BN / TN), COLS = BN / TN;
  constexpr int A_LOADS = (BM * BK / 4 + THREADS - 1) / THREADS, W_LOADS = (BN * BK / 4 + THREADS - 1) / THREADS;
  constexpr int A_STRIDE = BM + 4, W_STRIDE = BN + 4;              // floats of a k's row, padded against conflicts of the stores
  static_assert(TM == 2 || TM == 4 || TM == 8, "a thread's rows are neighbours");
  static_assert(TN == 4 || TN == 8, "a thread's columns are one or two groups of four");
  static_assert(COLS % 8 == 0 && (BM / TM) % 4 == 0, "a warp is 4 x 8 threads");
  extern __shared__ __align__(16) float smem[];
  float* As = smem;                                                // 2 x BK x A_STRIDE
  float* Ws = smem + 2 * BK * A_STRIDE;                            // 2 x BK x W_STRIDE
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ty = (warp / (COLS / 8)) * 4 + lane / 8, tx = (warp % (COLS / 8)) * 8 + lane % 8;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;
  float4 a_next[A_LOADS], w_next[W_LOADS];
  // load i of a thread: row (tid + i * THREADS) / (BK / 4), elements 4 * (that % (BK / 4)) on
  auto fetch_block = [&](int k0) {
#pragma unroll
    for (int i = 0; i < A_LOADS; i++) {
      const int idx = tid + i * THREADS, row = m0 + idx / (BK / 4);
      if (BM * BK / 4 % THREADS == 0 || idx < BM * BK / 4)
        a_next[i] = fetch<VEC>(A + (size_t)row * lda, row < M, k0 + 4 * (idx % (BK / 4)), K);
    }
  };
  auto fetch_weights = [&](int k0) {
#pragma unroll
    for (int i = 0; i < W_LOADS; i++) {
      const int idx = tid + i * THREADS, row = n0 + idx / (BK / 4);
      if (BN * BK / 4 % THREADS == 0 || idx < BN * BK / 4)
        w_next[i] = fetch<VEC>(W + (size_t)row * K, row < N, k0 + 4 * (idx % (BK / 4)), K);
    }
  };
  auto store_block = [&](int stage) {
    float* a_s = As + stage * BK * A_STRIDE;
    float* w_s = Ws + stage * BK * W_STRIDE;
#pragma unroll
    for (int i = 0; i < A_LOADS; i++) {
      const int idx = tid + i * THREADS, row = idx / (BK / 4), k = 4 * (idx % (BK / 4));
      if (BM * BK / 4 % THREADS == 0 || idx < BM * BK / 4) {
        const float v[4] = {a_next[i].x, a_next[i].y, a_next[i].z, a_next[i].w};
#pragma unroll
        for (int e = 0; e < 4; e++) a_s[(k + e) * A_STRIDE + row] = v[e];
      }
    }
#pragma unroll
    for (int i = 0; i < W_LOADS; i++) {
      const int idx = tid + i * THREADS, row = idx / (BK / 4), k = 4 * (idx % (BK / 4));
      if (BN * BK / 4 % THREADS == 0 || idx < BN * BK / 4) {
        const float v[4] = {w_next[i].x, w_next[i].y, w_next[i].z, w_next[i].w};
#pragma unroll
        for (int e = 0; e < 4; e++) w_s[(k + e) * W_STRIDE + row] = v[e];
      }
    }
  };

  fetch_weights(0);                                                // no earlier kernel writes weights
  pdl_wait();
  fetch_block(0);
  store_block(0);
  __syncthreads();
  const int blocks = (K + BK - 1) / BK;
  for (int block = 0; block < blocks; block++) {
    const int stage = block & 1;
    if (block + 1 < blocks) {
      fetch_block((block + 1) * BK);
      fetch_weights((block + 1) * BK);
    }
    const float* a_s = As + stage * BK * A_STRIDE + ty * TM;
    const float* w_s = Ws + stage * BK * W_STRIDE + tx * 4;
    float a[2][TM];
    unsigned long long w[2][TN / 2];
    auto read = [&](int k, int slot) {
      if (TM == 2) *(float2*)a[slot] = *(const float2*)&a_s[k * A_STRIDE];
#pragma unroll
      for (int i = 0; i < TM / 4; i++) *(float4*)&a[slot][4 * i] = *(const float4*)&a_s[k * A_STRIDE + 4 * i];
#pragma unroll
      for (int j = 0; j < TN / 4; j++) *(ulonglong2*)&w[slot][2 * j] = *(const ulonglong2*)&w_s[k * W_STRIDE + j * (BN / 2)];
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < BK; k++) {
      if (k + 1 < BK) read(k + 1, (k + 1) & 1);
#pragma unroll
      for (int i = 0; i < TM; i++) {
        const unsigned long long both = twice(a[k & 1][i]);
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = fma_pair(both, w[k & 1][j], acc[i][j]);
      }
    }
    if (block + 1 < blocks) store_block(stage ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const int gn = n0 + (j / 4) * (BN / 2) + tx * 4 + j % 4;
      if (gn >= N) continue;
      float v = __uint_as_float((unsigned)(j % 2 ? acc[i][j / 2] >> 32 : acc[i][j / 2]));
      if (bias) v += bias[gn];
      if (residual) v += residual[(size_t)gm * ldo + gn];
      out[(size_t)gm * ldo + gn] = from_float<TO>(v);
    }
  }
}

template <int BM, int BN, int BK, int TM, int TN, bool VEC, typename TA, typename TW, typename TO>
int launch_tile(const TA* A, const TW* W, const float* bias, const float* residual, TO* out, int M, int N, int K, int lda, int ldo,
                cudaStream_t stream) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr size_t smem = (size_t)2 * BK * (BM + 4 + BN + 4) * sizeof(float);
  auto* kernel = gemm_simple_kernel<BM, BN, BK, TM, TN, VEC, TA, TW, TO>;
  static_assert(smem <= 48 * 1024, "fits without asking for more");
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  sprout_launch(kernel, grid, dim3(THREADS), smem, stream, A, W, bias, residual, out, M, N, K, lda, ldo);
  return sprout_check_launch("gemm_simple");
}

// The tile for a call's sizes, measured in float32 (512 rows unless said).  Few rows are a stream of weights: rows of 128 bytes a
// k-block and no more sums than rows.  Between: 64 x 64, so that small matrices still put a CTA on most SMs (1,152 x 896: 144 CTAs,
// 43 us; 128 x 64 65 us, 128 x 128 101 us; 9,728 x 896: 226, 234, 265 us).  From eight CTAs an SM on, 128 x 64 with 8 x 8 sums a
// thread reads less shared memory a multiply-add (2,048 rows of 9,728 x 896: 745 us = 48 TFLOP/s; 64 x 64 802, 128 x 128 761 us).
template <bool VEC, typename TA, typename TW, typename TO>
int launch_sizes(const TA* A, const TW* W, const float* bias, const float* residual, TO* out, int M, int N, int K, int lda, int ldo,
                 cudaStream_t stream) {
  if (M <= 8) return launch_tile<8, 128, 32, 2, 4, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  if (M <= 16) return launch_tile<16, 128, 32, 4, 4, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  const long long tiles = (long long)((M + 127) / 128) * ((N + 63) / 64);
  if (tiles >= 8 * sprout_sm_count()) return launch_tile<128, 64, 16, 8, 8, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  return launch_tile<64, 64, 16, 8, 4, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
}

template <typename TA, typename TW, typename TO>
int launch(const void* A, const void* W, const float* bias, const float* residual, void* out, int M, int N,
           int K, int lda, int ldo, cudaStream_t stream) {
  const bool vec = K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % (4 * sizeof(TA)) == 0 && (uintptr_t)W % (4 * sizeof(TW)) == 0;
  return vec ? launch_sizes<true>((const TA*)A, (const TW*)W, bias, residual, (TO*)out, M, N, K, lda, ldo, stream)
             : launch_sizes<false>((const TA*)A, (const TW*)W, bias, residual, (TO*)out, M, N, K, lda, ldo, stream);
}

}  // namespace

// A is [M, K] with row stride lda, W is [N, K] contiguous, out (and residual) [M, N] with row
// stride ldo.  `residual` may be the same buffer as `out`.  a_dtype is also the weight's dtype.
SPROUT_API int sprout_gemm_simple(const void* A, const void* W, const float* bias, const float* residual,
                                  void* out, int a_dtype, int out_dtype, int M, int N, int K, int lda, int ldo,
                                  cudaStream_t stream) {
  SPROUT_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_simple: sizes must be positive (M=%d N=%d K=%d)", M, N, K);
  SPROUT_REQUIRE(A && W && out, "gemm_simple: null pointer");
  SPROUT_REQUIRE(lda >= K && ldo >= N, "gemm_simple: row strides smaller than the rows");
  SPROUT_REQUIRE(!residual || out_dtype == SPROUT_F32, "gemm_simple: a residual needs a float32 output");
  SPROUT_REQUIRE((M + 63) / 64 <= 65535, "gemm_simple: too many rows (%d)", M);
  if (a_dtype == SPROUT_F32 && out_dtype == SPROUT_F32)
    return launch<float, float, float>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  if (a_dtype == SPROUT_BF16 && out_dtype == SPROUT_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  if (a_dtype == SPROUT_BF16 && out_dtype == SPROUT_F32)
    return launch<__nv_bfloat16, __nv_bfloat16, float>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  return sprout_fail("gemm_simple: unsupported dtypes a=%d out=%d", a_dtype, out_dtype);
}
