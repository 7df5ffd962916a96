// out[m, n] = sum_k A[m, k] * W[n, k] (+ bias[n]) (+ residual[m, n]) on CUDA cores with
// float32 fused multiply-adds: the matrix product of the true 32-bit path (no tensor cores,
// no reduced-precision mode), and a plain reference for the tensor-core kernels.  Each output
// element is one sum in ascending k, or two to eight such sums over equal shares of K added in their order; how many follows from the
// matrix alone (`split_of`), so its value does not depend on how many rows the call has, on where a row sits among them, or on the
// tile that a call's sizes pick.
//
// Bound by the fused multiply-adds and the shared-memory reads that feed them.  A thread holds TM x TN sums as pairs of
// neighbouring rows for the packed `fma.rn.f32x2` (two IEEE fused multiply-adds an instruction, W's value doubled in registers);
// both operands lie in shared memory as [k][row], the next k's values are read while one k is multiplied, and the next
// k-block's 16-byte loads are in flight meanwhile.  What fills the device is the tile (`launch_sizes`) and the shares of K: the CTAs
// of a cluster take one each and add them up out of each other's shared memory.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int K_SHARE = 32;             // a share of K is a multiple of this: whole k-blocks of every tile, 16-byte loads

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

// Every thread of the cluster's CTAs meets here; their shared memory written before is visible after.
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Four floats at this CTA's shared-memory address `p`, in the cluster's CTA of rank `rank`.
__device__ __forceinline__ float4 load_shared_of(const float* p, int rank) {
  uint32_t at;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
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

// A k's row of an operand in shared memory.  A warp's stores go to several k at one row: whole banks of 32 are swizzled, row r of k at
// place r ^ (k / 4 << 3) (<< 2 with 32 k: groups of eight or four rows move), other rows are padded.  With 8 x 8 sums a thread the
// padded rows are the faster ones (2,048 x 9,728 x 896: 744 us, 768 swizzled); with fewer the swizzled (512 x 896 x 4,864: 160 padded, 153
// swizzled; 64 x 896 x 4,864: 58 and 54; 1 x 151,936 x 896: 180 and 136).
constexpr bool swizzled(int rows, int TN) { return TN == 4 && rows % 32 == 0; }
constexpr int row_floats(int rows, int TN) { return swizzled(rows, TN) ? rows : rows + 4; }

// Four neighbouring results of a row into `out`: bias and residual added, in one access where the row allows it.
template <typename TO>
__device__ __forceinline__ void put4(float4 sum, const float* bias, const float* residual, TO* out, size_t at, int gn, int N, bool wide) {
  float v[4] = {sum.x, sum.y, sum.z, sum.w};
  if (sizeof(TO) == 4 && wide && gn + 4 <= N) {
#pragma unroll
    for (int j = 0; j < 4; j++) if (bias) v[j] += bias[gn + j];
    if (residual) {
      const float4 r = *(const float4*)(residual + at);
      v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
    }
    *(float4*)(out + at) = make_float4(v[0], v[1], v[2], v[3]);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (gn + j >= N) break;
    if (bias) v[j] += bias[gn + j];
    if (residual) v[j] += residual[at + j];
    out[at + j] = from_float<TO>(v[j]);
  }
}

template <int BM, int BN, int BK, int TM, int TN, int SPLIT, bool VEC, typename TA, typename TW, typename TO>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_simple_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const float* __restrict__ bias,
                   const float* residual, TO* out, int M, int N, int whole_K, int k_share, int lda, int ldo, bool wide) {
  constexpr int THREADS = (BM / TM) * (BN / TN), COLS = BN / TN;
  constexpr int A_LOADS = (BM * BK / 4 + THREADS - 1) / THREADS, W_LOADS = (BN * BK / 4 + THREADS - 1) / THREADS;
  constexpr bool W_SWIZZLED = swizzled(BN, TN), A_SWIZZLED = swizzled(BM, TN);
  constexpr int A_STRIDE = row_floats(BM, TN), W_STRIDE = row_floats(BN, TN);
  // r's place in the row of k
  auto a_place = [](int k, int r) { return A_SWIZZLED ? r ^ ((k / 4) << (BK == 16 ? 3 : 2)) : r; };
  auto w_place = [](int k, int r) { return W_SWIZZLED ? r ^ ((k / 4) << (BK == 16 ? 3 : 2)) : r; };
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
  // this CTA's share of K: rank z of the cluster has [z * k_share, (z + 1) * k_share)
  const int k_begin = SPLIT > 1 ? (int)blockIdx.z * k_share : 0;
  const int K = SPLIT > 1 ? min(whole_K, k_begin + k_share) : whole_K;
  unsigned long long acc[TM / 2][TN];                              // rows 2 i and 2 i + 1 of a column
#pragma unroll
  for (int i = 0; i < TM / 2; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0ull;
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
        w_next[i] = fetch<VEC>(W + (size_t)row * whole_K, row < N, k0 + 4 * (idx % (BK / 4)), K);
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
        for (int e = 0; e < 4; e++) a_s[(k + e) * A_STRIDE + a_place(k, row)] = v[e];
      }
    }
#pragma unroll
    for (int i = 0; i < W_LOADS; i++) {
      const int idx = tid + i * THREADS, row = idx / (BK / 4), k = 4 * (idx % (BK / 4));
      if (BN * BK / 4 % THREADS == 0 || idx < BN * BK / 4) {
        const float v[4] = {w_next[i].x, w_next[i].y, w_next[i].z, w_next[i].w};
#pragma unroll
        for (int e = 0; e < 4; e++) w_s[(k + e) * W_STRIDE + w_place(k, row)] = v[e];
      }
    }
  };

  fetch_weights(k_begin);                                          // no earlier kernel writes weights
  pdl_wait();
  fetch_block(k_begin);
  store_block(0);
  __syncthreads();
  const int blocks = (K - k_begin + BK - 1) / BK;
  for (int block = 0; block < blocks; block++) {
    const int stage = block & 1;
    if (block + 1 < blocks) {
      fetch_block(k_begin + (block + 1) * BK);
      fetch_weights(k_begin + (block + 1) * BK);
    }
    const float* a_s = As + stage * BK * A_STRIDE;
    const float* w_s = Ws + stage * BK * W_STRIDE;
    unsigned long long a[2][TM / 2];
    float w[2][TN];
    auto read = [&](int k, int slot) {
      if (TM == 2) a[slot][0] = *(const unsigned long long*)&a_s[k * A_STRIDE + a_place(k, ty * TM)];
#pragma unroll
      for (int i = 0; i < TM / 4; i++) *(ulonglong2*)&a[slot][2 * i] = *(const ulonglong2*)&a_s[k * A_STRIDE + a_place(k, ty * TM + 4 * i)];
#pragma unroll
      for (int j = 0; j < TN / 4; j++) *(float4*)&w[slot][4 * j] = *(const float4*)&w_s[k * W_STRIDE + w_place(k, j * (BN / 2) + tx * 4)];
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < BK; k++) {
      if (k + 1 < BK) read(k + 1, (k + 1) & 1);
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const unsigned long long both = twice(w[k & 1][j]);
#pragma unroll
        for (int i = 0; i < TM / 2; i++) acc[i][j] = fma_pair(a[k & 1][i], both, acc[i][j]);
      }
    }
    if (block + 1 < blocks) store_block(stage ^ 1);
    __syncthreads();
  }
  auto sum4 = [&](int i, int j) {                                  // row i, columns 4 j .. 4 j + 3 of the thread's
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = __uint_as_float((unsigned)(i % 2 ? acc[i / 2][4 * j + e] >> 32 : acc[i / 2][4 * j + e]));
    return make_float4(v[0], v[1], v[2], v[3]);
  };
  if constexpr (SPLIT == 1) {
#pragma unroll
    for (int i = 0; i < TM; i++) {
      const int gm = m0 + ty * TM + i;
      if (gm >= M) continue;
#pragma unroll
      for (int j = 0; j < TN / 4; j++) {
        const int gn = n0 + j * (BN / 2) + tx * 4;
        if (gn < N) put4(sum4(i, j), bias, residual, out, (size_t)gm * ldo + gn, gn, N, wide);
      }
    }
  } else {
    // the shares' sums lie in their CTAs' shared memory (the operands have been read); every CTA adds up its part of the tile's
    // rows, share by share in the order of K
    constexpr int P_STRIDE = BN + 4;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN / 4; j++) *(float4*)&smem[(ty * TM + i) * P_STRIDE + j * (BN / 2) + tx * 4] = sum4(i, j);
    cluster_meet();
    constexpr int PART = BM * BN / 4 / SPLIT;
    static_assert(BM * BN / 4 % SPLIT == 0, "the tile divides among the cluster's CTAs");
    for (int idx = blockIdx.z * PART + tid; idx < ((int)blockIdx.z + 1) * PART; idx += THREADS) {
      const int row = idx / (BN / 4), col = 4 * (idx % (BN / 4)), gm = m0 + row, gn = n0 + col;
      if (gm >= M || gn >= N) continue;
      float4 part[SPLIT];
#pragma unroll
      for (int z = 0; z < SPLIT; z++) part[z] = load_shared_of(&smem[row * P_STRIDE + col], z);
#pragma unroll
      for (int z = 1; z < SPLIT; z++) {
        part[0].x += part[z].x; part[0].y += part[z].y; part[0].z += part[z].z; part[0].w += part[z].w;
      }
      put4(part[0], bias, residual, out, (size_t)gm * ldo + gn, gn, N, wide);
    }
    cluster_meet();                                                // nobody leaves while others read its sums
  }
}

template <int BM, int BN, int BK, int TM, int TN, int SPLIT, bool VEC, typename TA, typename TW, typename TO>
int launch_tile(const TA* A, const TW* W, const float* bias, const float* residual, TO* out, int M, int N, int K, int lda, int ldo,
                cudaStream_t stream) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  constexpr size_t operands = (size_t)2 * BK * (row_floats(BM, TN) + row_floats(BN, TN)) * sizeof(float), sums = SPLIT > 1 ? (size_t)BM * (BN + 4) * sizeof(float) : 0;
  constexpr size_t smem = operands > sums ? operands : sums;
  auto* kernel = gemm_simple_kernel<BM, BN, BK, TM, TN, SPLIT, VEC, TA, TW, TO>;
  static_assert(smem <= 48 * 1024, "fits without asking for more");
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((N + BN - 1) / BN, (M + BM - 1) / BM, SPLIT);
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  int count = 0;
  if (SPLIT > 1) {
    attributes[count].id = cudaLaunchAttributeClusterDimension;
    attributes[count].val.clusterDim.x = 1;
    attributes[count].val.clusterDim.y = 1;
    attributes[count++].val.clusterDim.z = SPLIT;
  }
  if (sprout_pdl_enabled()) {
    attributes[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[count++].val.programmaticStreamSerializationAllowed = 1;
  }
  config.attrs = attributes;
  config.numAttrs = count;
  const bool wide = sizeof(TO) == 4 && ldo % 4 == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)residual % 16 == 0;
  const int k_share = ((K + SPLIT - 1) / SPLIT + K_SHARE - 1) / K_SHARE * K_SHARE;
  cudaLaunchKernelEx(&config, kernel, A, W, bias, residual, out, M, N, K, k_share, lda, ldo, wide);
  return sprout_check_launch("gemm_simple");
}

// The tile for a call's sizes, measured in float32.  Few rows are a stream of weights: rows of 128 bytes a
// k-block and no more sums than rows.  Between: 64 x 64, so that small matrices still put a CTA on most SMs.  From eight CTAs an SM on
// (shares counted; from sixteen where there are eight shares), 128 x 64 with 8 x 8 sums a thread reads less shared memory a multiply-add (2,048 rows of 9,728 x 896: 745 us = 48
// TFLOP/s; 64 x 64 802, 128 x 128 761 us).
template <int SPLIT, bool VEC, typename TA, typename TW, typename TO>
int launch_sizes(const TA* A, const TW* W, const float* bias, const float* residual, TO* out, int M, int N, int K, int lda, int ldo,
                 cudaStream_t stream) {
  if (M <= 8) return launch_tile<8, 128, 32, 2, 4, SPLIT, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  if (M <= 16) return launch_tile<16, 128, 32, 4, 4, SPLIT, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  const long long tiles = (long long)((M + 127) / 128) * ((N + 63) / 64) * SPLIT;
  if (tiles >= (SPLIT > 4 ? 16 : 8) * sprout_sm_count()) return launch_tile<128, 64, 16, 8, 8, SPLIT, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
  return launch_tile<64, 64, 16, 8, 4, SPLIT, VEC>(A, W, bias, residual, out, M, N, K, lda, ldo, stream);
}

// How many CTAs (a cluster) share K: by the matrix alone, so that a row's bits do not depend on the rows beside it.  Small matrices
// have too few tiles for the device (M x 896 x 4,864 in one, two, four shares: 1 row 135, 73, 33 us; 64 rows 203, 113, 54; 512 rows 203,
// 152, 153; 2,048 rows 712, 468, 413; M x 1,152 x 896: 64 rows 39, 24, 13, 2,048 rows 138, 104, 106).  Wide ones fill it by their columns
// from some hundred rows on (M x 9,728 x 896: 64 rows 60, 46, 36; 512 rows 230, 211, 213; 2,048 rows 752, 745, 804), and a vocabulary's
// from one (1 x 151,936 x 896: 136, 160, 165).  Eight shares from a K of 4,096 on (M x 896 x 4,864, four and eight: 1 row
// 35, 19, 64 rows 55, 35, 512 rows 151, 119, 2,048 rows 415, 411; M x 2,048 x 2,048: 64 rows 33, 26, but 512 rows 114, 119).
int split_of(int N, int K) {
  if (K < 256 || N > 65536) return 1;
  return N > 4096 ? 2 : K < 4096 ? 4 : 8;
}

template <typename TA, typename TW, typename TO>
int launch(const void* A, const void* W, const float* bias, const float* residual, void* out, int M, int N,
           int K, int lda, int ldo, cudaStream_t stream) {
  const bool vec = K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % (4 * sizeof(TA)) == 0 && (uintptr_t)W % (4 * sizeof(TW)) == 0;
  const int split = split_of(N, K);
  auto sizes = [&](auto shares) {
    constexpr int SPLIT = decltype(shares)::value;
    return vec ? launch_sizes<SPLIT, true>((const TA*)A, (const TW*)W, bias, residual, (TO*)out, M, N, K, lda, ldo, stream)
               : launch_sizes<SPLIT, false>((const TA*)A, (const TW*)W, bias, residual, (TO*)out, M, N, K, lda, ldo, stream);
  };
  if (split == 8) return sizes(std::integral_constant<int, 8>());
  if (split == 4) return sizes(std::integral_constant<int, 4>());
  if (split == 2) return sizes(std::integral_constant<int, 2>());
  return sizes(std::integral_constant<int, 1>());
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
