// The routed experts' products on the 5th-generation tensor cores, the experts' matrices on the MMA's M axis:
//   D[feature, row] = sum_k W_e[feature, k] * rows[row, k]   for the rows offsets[e] .. offsets[e + 1] - 1 of every expert e.
//
// What bounds them: the stream of all experts' matrices from memory (in a prompt each is read once for some two hundred rows, in a
// decode batch for a handful), as long as nothing is done for padding.  So the weights fill the 256 rows of a CTA pair's tile, which
// an expert's matrix does without a remainder, and the rows are its columns, as many as there are in multiples of 16 (the MMA's N
// is a number in its descriptor): an expert's rows are cut into equal tiles of up to 256.  With the rows on M, as before, 32 experts
// of 227 rows each were computed as 256 or 512, and a decode batch's 7 rows were 256, whose copies took the place of weights.
//
// CTAs come in pairs (tcgen05.mma.cta_group::2): each copies its 128 rows of W and half of the tile's rows, the first issues the MMAs
// for both.  Operand tiles of 64 K-elements (128-byte swizzle) come by TMA through a ring of stages; rows in a box of 8 to 128.  A gated unit's tile has 64 gate rows a CTA and the 64 up rows that go with them, in
// blocks of 8 in turn (a dimension of the tensor map), so that lanes l and l ^ 8 of a warp hold both products of a feature.  Two
// accumulators alternate: a tile's epilogue runs under the next one's products.  Persistent: a pair walks the tiles with the stride of
// the grid, an expert's row tiles of the same features side by side, so that the second finds the weights in L2.
//
// 32 experts of 1,024 over 2,048 wide rows, top 4, the whole layer when the matrices moved to M: 2,048 tokens 303 -> 272 us, 64 tokens 156 ->
// 121 (with the router, the arrangement and the calls as they are now 246 and 117).  Both products and the gather 134 and 95 us (cold caches): for 2,048 tokens the gated one takes 70 us, reads 300 MB and keeps the tensor
// cores busy for half of that time; for 64 tokens 402 MB pass at 4.2 TB/s with the launches' ends.
//
// Waits are bounded as in the dense products.
#include <cuda.h>

#include "common.cuh"
#include "experts.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int BLOCK_M = 128, BLOCK_K = 64, MAX_N = 256, NUM_THREADS = 320;     // a CTA's weight rows, elements of K a stage, rows a tile
constexpr int MAX_EXPERTS = 2048;
constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2, B_BYTES = MAX_N / 2 * BLOCK_K * 2, STAGE_BYTES = A_BYTES + B_BYTES, STAGES = 6;
constexpr int TABLE_BYTES = (2 * (MAX_EXPERTS + 1) * 4 + 15) / 16 * 16;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + TABLE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
constexpr int ROW_MAPS = 5;                            // boxes of 8, 16, 32, 64 and 128 rows

// The unit is part of the kernel: as a question to every activation it kept them from running side by side.
enum Kind : int { KIND_CLAMPED = 0, KIND_SILU = 1, KIND_GELU = 2, KIND_DOWN = 3 };

// 1 / x and g / x for x of 1 to infinity (1 + exp), rounded as IEEE has it: from an approximate reciprocal r, r + r (1 - x r) and
// q + r (g - x q), each remainder in one fused multiply-add (Newton's iteration; its last rounding: P. W. Markstein, IBM J. Res. Develop. 34,
// 1990).  The operators are right for any operand and branch for that, and eight activations no longer run side by side: 2,048 tokens of
// 2,048 over 2,048, the clamped unit's product 49 us with them, 31 so.  Compared with the operators: 1 / x over every x up to 2^126, g / x
// over every bfloat16 g.  Above 2^126 (a sigmoid under 2^-126) 1 / x may be off by the last bit of its denormal.
__device__ __forceinline__ float scaled_reciprocal(float x, float& scaled, float& scale) {
  scale = x > 0x1p100f ? 0x1p-64f : 1.0f;                // keeps the reciprocal normal
  scaled = x * scale;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(scaled));
  r = fmaf(r, fmaf(-scaled, r, 1.0f), r);
  return x == INFINITY ? 0.f : r;
}
__device__ __forceinline__ float reciprocal_of(float x) {
  float scaled, scale;
  return scaled_reciprocal(x, scaled, scale) * scale;
}
__device__ __forceinline__ float quotient_of(float g, float x) {
  float scaled, scale;
  const float r = scaled_reciprocal(x, scaled, scale), q = g * r, rest = fmaf(-scaled, q, g);
  return (fabsf(rest) > 0.f ? fmaf(rest, r, q) : q) * scale;       // nothing left, or no number left (infinities): q as it is
}

// The gated units as the other kernels compute them (experts.cuh).
template <int KIND>
__device__ __forceinline__ float gated_unit(float g, float u, float limit, float alpha) {
  if (KIND == KIND_SILU) return quotient_of(g, 1.0f + expf(-g)) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g * reciprocal_of(1.0f + expf(-alpha * g)) * (u + 1.0f);
}

struct RowMaps { CUtensorMap box[ROW_MAPS]; };

struct ExpertsParams {
  void* out;                       // [entries, N]: bfloat16, or float32 for KIND_DOWN
  int N, K, experts, entries;
  const int* offsets; const int* order;        // null: one expert with all entries
  const float* row_weights;        // of entry order[row], or null: multiply the products before the activation
  float limit, alpha;
  int* status;
};

// tiles of an expert's rows, and the rows of each but perhaps the last
__device__ __forceinline__ int tiles_of(int rows) { return (rows + MAX_N - 1) / MAX_N; }

struct Tile { int expert, row0, rows, col; };        // `col`: the tile's place across the features

__device__ __forceinline__ void tma_load_pair_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_pair_5d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, int u, int v) {
  asm volatile("cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(u), "r"(v) : "memory");
}

template <int KIND>
__global__ void __launch_bounds__(NUM_THREADS, 1)
experts_tcgen05_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ RowMaps maps_x, const ExpertsParams p) {
  constexpr bool GATED = KIND == KIND_CLAMPED || KIND == KIND_SILU;
  constexpr int FEATURES = GATED ? BLOCK_M / 2 : BLOCK_M;         // output features of a CTA's tile
  const uint32_t rank = cluster_ctarank();                                   // 0 issues the MMAs
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  int* tile_prefix = (int*)(smem + STAGES * STAGE_BYTES);                    // row tiles before expert e, and its first row
  int* row_prefix = tile_prefix + p.experts + 1;
  uint64_t* full_bar = (uint64_t*)(smem + STAGES * STAGE_BYTES + TABLE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;             // [2] accumulator complete (MMA -> epilogue)
  uint64_t* acc_empty = acc_full + 2;                  // [2] accumulator read out (both CTAs' epilogues -> MMA)
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K, cols = (p.N + 2 * FEATURES - 1) / (2 * FEATURES);

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 16); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  pdl_wait();                                          // the offsets are an earlier kernel's
  if (warp == 0) {
    int before = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      const int begin = p.offsets && e < p.experts ? p.offsets[e] : 0, end = e >= p.experts ? 0 : p.offsets ? p.offsets[e + 1] : p.entries;
      const int own = tiles_of(end - begin);
      int sum = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int other = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += other;
      }
      if (e < p.experts) {
        tile_prefix[e] = before + sum - own;
        row_prefix[e] = begin;
        if (e == p.experts - 1) { tile_prefix[p.experts] = before + sum; row_prefix[p.experts] = end; }
      }
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // the pair's MMAs write both CTAs' tensor memory at one address: both have all of it, from column 0
  if (tmem_base != 0 && threadIdx.x == 0) { *abort_flag = 1; atomicOr(p.status, SPROUT_STATUS_BAD_LAYOUT); }
  cluster_barrier();                                   // nobody counts on the other CTA's barriers before they are initialised

  const int total_work = tile_prefix[p.experts] * cols;
  const int first_work = (int)blockIdx.x >> 1, work_stride = (int)gridDim.x >> 1;
  auto tile_at = [&](int w) {
    const int at = w / cols;
    int e = 0, hi = p.experts;                         // the last e with tile_prefix[e] <= at: it has rows
    while (hi - e > 1) {
      const int mid = (e + hi) / 2;
      if (tile_prefix[mid] <= at) e = mid; else hi = mid;
    }
    const int tiles = tile_prefix[e + 1] - tile_prefix[e], local = w - tile_prefix[e] * cols, rows = row_prefix[e + 1] - row_prefix[e];
    const int per = ((rows + tiles - 1) / tiles + 15) / 16 * 16, first = local % tiles * per;
    return Tile{e, row_prefix[e] + first, min(per, rows - first), local / tiles};
  };
  const uint32_t smem_base = smem_u32(smem), full_base = smem_u32(full_bar), empty_base = smem_u32(empty_bar);
  int issued = 0;
  if (warp == 0 && elect_one()) {
    // ---------------- copies: both CTAs' count on the first CTA's barriers
    const uint32_t count_base = cluster_map_shared(full_base, 0);
    uint32_t s = 0, parity = 1;
    bool ok = true;
    for (int w = first_work; w < total_work && ok; w += work_stride) {
      const Tile t = tile_at(w);
      const int half = (t.rows + 15) / 16 * 8, row = t.row0 + (int)rank * half;         // this CTA's rows of the tile
      int box = 0;                                     // the smallest box that holds them
      while ((8 << box) < half) box++;
      const CUtensorMap* map_x = &maps_x.box[box];
      const uint32_t bytes = 2 * (A_BYTES + (8 << box) * BLOCK_K * 2);
      const int feature = (t.col * 2 + (int)rank) * FEATURES;
      for (int i = 0; i < num_kb; i++) {
        if (!mbar_wait_addr(empty_base + 8 * s, parity, abort_flag)) { *abort_flag = 1; atomicOr(p.status, SPROUT_STATUS_WAIT_TIMEOUT); ok = false; break; }
        const uint32_t bar = count_base + 8 * s, a = smem_base + s * STAGE_BYTES;
        if (rank == 0) mbar_expect_tx_addr(full_base + 8 * s, bytes);
        if (GATED) tma_load_pair_5d(a, &map_w, bar, i * BLOCK_K, 0, 0, feature / 8, t.expert);
        else tma_load_pair_3d(a, &map_w, bar, i * BLOCK_K, feature, t.expert);
        tma_load_2d_pair(a + A_BYTES, map_x, bar, i * BLOCK_K, row);
        issued++;
        if (++s == STAGES) { s = 0; parity ^= 1; }
      }
    }
  } else if (warp == 1 && rank == 0 && elect_one()) {
    // ---------------- MMAs of the pair
    const uint64_t a_desc0 = umma_smem_desc(smem), b_desc0 = umma_smem_desc(smem + A_BYTES);
    constexpr uint64_t STAGE_STEP = STAGE_BYTES >> 4;
    uint64_t a_desc = a_desc0, b_desc = b_desc0;
    uint32_t s = 0, parity = 0;
    bool ok = true;
    int tiles_done = 0;
    for (int w = first_work; w < total_work && ok; w += work_stride, tiles_done++) {
      const Tile t = tile_at(w);
      const uint32_t idesc = umma_idesc(2 * BLOCK_M, (t.rows + 15) / 16 * 16);
      const int acc = tiles_done & 1;
      if (!mbar_wait_cluster(smem_u32(&acc_empty[acc]), ((tiles_done >> 1) & 1) ^ 1, abort_flag)) { *abort_flag = 1; atomicOr(p.status, SPROUT_STATUS_WAIT_TIMEOUT); break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * MAX_N;
      uint32_t accumulate = 0;
      for (int i = 0; i < num_kb; i++) {
        if (!mbar_wait_addr(full_base + 8 * s, parity, abort_flag)) { *abort_flag = 1; atomicOr(p.status, SPROUT_STATUS_WAIT_TIMEOUT); ok = false; break; }
        tc_fence_after();
        umma_bf16_pair(d_tmem, a_desc, b_desc, idesc, accumulate);
        umma_bf16_pair(d_tmem, a_desc + 2, b_desc + 2, idesc, 1);
        umma_bf16_pair(d_tmem, a_desc + 4, b_desc + 4, idesc, 1);
        umma_bf16_pair(d_tmem, a_desc + 6, b_desc + 6, idesc, 1);
        umma_commit_pair(empty_base + 8 * s, 3);
        accumulate = 1;
        if (++s == STAGES) { s = 0; parity ^= 1; a_desc = a_desc0; b_desc = b_desc0; } else { a_desc += STAGE_STEP; b_desc += STAGE_STEP; }
      }
      if (ok) umma_commit_pair(smem_u32(&acc_full[acc]), 3);
    }
  } else if (warp >= 2) {
    // ---------------- epilogue: lanes are features, columns rows; two warps per 32-lane quarter take 16 columns in turn
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    int tiles_done = 0;
    for (int w = first_work; w < total_work; w += work_stride, tiles_done++) {
      const Tile t = tile_at(w);
      const int acc = tiles_done & 1;
      bool ok = true;
      if (lane == 0) {
        ok = mbar_wait(&acc_full[acc], (tiles_done >> 1) & 1, abort_flag);
        if (!ok) { *abort_flag = 1; atomicOr(p.status, SPROUT_STATUS_WAIT_TIMEOUT); }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * MAX_N;
      const int feature0 = (t.col * 2 + (int)rank) * FEATURES;
#pragma unroll 1
      for (int c = part * 16; c < t.rows; c += 32) {
        uint32_t raw[16];
        tmem_load16(taddr + c, raw);
        if constexpr (GATED) {
          // lanes l and l ^ 8 hold a gate and its up product: of two neighbouring rows each finishes one.  All eight are computed side
          // by side (rows that are padding too): two warps a scheduler hide no latency of one after the other.
          const int upper = (lane >> 3) & 1, feature = feature0 + quarter * 16 + (lane >> 4) * 8 + (lane & 7);
          float weight[8], v[8];
#pragma unroll
          for (int j = 0; j < 8; j++) weight[j] = p.row_weights ? p.row_weights[p.order[t.row0 + min(c + 2 * j + upper, t.rows - 1)]] : 1.0f;
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const float mine = __uint_as_float(upper ? raw[2 * j + 1] : raw[2 * j]);
            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(upper ? raw[2 * j] : raw[2 * j + 1]), 8);
            // rounded to bfloat16 before the activation, as separate products would leave them
            const float g = __bfloat162float(__float2bfloat16_rn((upper ? other : mine) * weight[j]));
            const float u = __bfloat162float(__float2bfloat16_rn((upper ? mine : other) * weight[j]));
            v[j] = gated_unit<KIND>(g, u, p.limit, p.alpha);
          }
          __nv_bfloat16* out = (__nv_bfloat16*)p.out + (size_t)(t.row0 + c + upper) * p.N + feature;
          const int left = feature < p.N ? t.rows - c - upper : 0;
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (2 * j < left) out[(size_t)(2 * j) * p.N] = __float2bfloat16_rn(v[j]);
        } else {
          const int feature = feature0 + quarter * 32 + lane;
          const int left = feature < p.N ? t.rows - c : 0;
          const size_t at = (size_t)(t.row0 + c) * p.N + feature;
          if (KIND == KIND_DOWN) {
#pragma unroll
            for (int j = 0; j < 16; j++)
              if (j < left) ((float*)p.out)[at + (size_t)j * p.N] = __uint_as_float(raw[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; j++) {
              const float weight = p.row_weights ? p.row_weights[p.order[t.row0 + min(c + j, t.rows - 1)]] : 1.0f;
              const float g = __bfloat162float(__float2bfloat16_rn(__uint_as_float(raw[j]) * weight));
              const float v = sprout_experts::glu(sprout_experts::UNIT_PLAIN, g, 0.f, 0.f, 0.f);
              if (j < left) ((__nv_bfloat16*)p.out)[at + (size_t)j * p.N] = __float2bfloat16_rn(v);
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (rank == 1) mbar_arrive_cluster(cluster_map_shared(smem_u32(&acc_empty[acc]), 0));
        else mbar_arrive(&acc_empty[acc]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) issued = __reduce_max_sync(0xffffffffu, issued);      // the copy thread's count
  if (*abort_flag && rank == 0 && warp == 0 && lane == 0) {
    // copies already issued still write shared memory: wait for them (bounded) before leaving; the first CTA's barriers count both CTAs'
    for (int i = max(0, issued - STAGES); i < issued; i++) mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1);
  }
  __syncthreads();
  cluster_barrier();                                   // neither CTA leaves while the other may still count on its barriers
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// ------------------------------------------------------------------ host side
// The map of the experts' matrices w [experts, matrix rows, K]: boxes of 128 rows x 64 elements of one expert.  Gated: of the matrix's
// `features` gate rows and as many up rows 64 each, in blocks of 8 in turn.  Kept like the other maps: an encode takes microseconds.
int weight_map(const void* w, int experts, int features, int K, bool gated, CUtensorMap* out) {
  static std::unordered_map<MapKey, CUtensorMap, MapHash> cache;
  static std::mutex lock;
  const MapKey key{w, experts, K, features, gated ? 1 : 0, 2};
  std::lock_guard<std::mutex> guard(lock);
  auto it = cache.find(key);
  if (it != cache.end()) { *out = it->second; return 0; }
  EncodeTiled encode = encode_fn();
  if (!encode) return sprout_fail("tensor map: cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t row = (cuuint64_t)K * 2;
  const cuuint64_t dims5[5] = {(cuuint64_t)K, 8, 2, (cuuint64_t)features / 8, (cuuint64_t)experts};
  const cuuint64_t strides5[4] = {row, row * features, row * 8, row * 2 * features};
  const cuuint32_t box5[5] = {BLOCK_K, 8, 2, BLOCK_M / 16, 1};
  const cuuint64_t dims3[3] = {(cuuint64_t)K, (cuuint64_t)features, (cuuint64_t)experts};
  const cuuint64_t strides3[2] = {row, row * features};
  const cuuint32_t box3[3] = {BLOCK_K, BLOCK_M, 1};
  const cuuint32_t steps[5] = {1, 1, 1, 1, 1};
  CUtensorMap map;
  CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, gated ? 5 : 3, const_cast<void*>(w), gated ? dims5 : dims3, gated ? strides5 : strides3,
                       gated ? box5 : box3, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return sprout_fail("experts_product: cuTensorMapEncodeTiled failed with code %d", (int)rc);
  if (cache.size() > 4096) cache.clear();
  cache.emplace(key, map);
  *out = map;
  return 0;
}

template <int KIND>
int launch_experts(const CUtensorMap& map_w, const RowMaps& maps_x, const ExpertsParams& p, long long work, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t err = cudaFuncSetAttribute(experts_tcgen05_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (err != cudaSuccess) return sprout_fail("experts_product: cannot reserve %d bytes of shared memory: %s", SMEM_BYTES, cudaGetErrorString(err));
    configured = true;
  }
  const long long pairs = work < sm_count() / 2 ? work : sm_count() / 2;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)(2 * pairs));
  config.blockDim = dim3(NUM_THREADS);
  config.dynamicSmemBytes = SMEM_BYTES;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = sprout_pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&config, experts_tcgen05_kernel<KIND>, map_w, maps_x, p);
  return sprout_check_launch("experts_product");
}

}  // namespace

int sprout_experts_product_tc(const void* rows, int row_stride, const int* offsets, const int* order, const void* w, void* out, int entries, int experts, int N,
                              int K, int unit, const float* row_weights, float limit, float alpha, int* status, cudaStream_t stream) {
  const bool gated = unit == sprout_experts::UNIT_CLAMPED || unit == sprout_experts::UNIT_SILU;
  SPROUT_REQUIRE(rows && w && out && status && entries > 0 && experts > 0 && (offsets ? (order != nullptr) : (experts == 1 && !row_weights)),
                 "experts_product: bad arguments");
  SPROUT_REQUIRE(N % 8 == 0 && K % 8 == 0 && experts <= MAX_EXPERTS, "experts_product: sizes in multiples of 8, up to 2,048 experts (N=%d K=%d, %d experts)", N, K, experts);
  const int features = gated ? BLOCK_M : 2 * BLOCK_M;                  // of a pair's tile
  const long long work = ((long long)entries / MAX_N + experts) * ((N + features - 1) / features);        // at most, whatever the routing
  SPROUT_REQUIRE((long long)experts * N * 2 <= 0x7fffffffLL && work <= 0x7fffffffLL, "experts_product: too many rows");
  const ExpertsParams p{out, N, K, experts, entries, offsets, order, row_weights, limit, alpha, status};
  CUtensorMap map_w;
  RowMaps maps_x;
  if (weight_map(w, experts, N, K, gated, &map_w)) return 1;
  for (int b = 0; b < ROW_MAPS; b++) {
    if (b > 0 && (8 << b) >= entries) maps_x.box[b] = maps_x.box[b - 1];       // no tile has so many rows: not used
    else if (tensor_map(rows, entries, K, row_stride, 8 << b, &maps_x.box[b])) return 1;
  }
  if (unit < 0) return launch_experts<KIND_DOWN>(map_w, maps_x, p, work, stream);
  if (unit == sprout_experts::UNIT_CLAMPED) return launch_experts<KIND_CLAMPED>(map_w, maps_x, p, work, stream);
  if (unit == sprout_experts::UNIT_SILU) return launch_experts<KIND_SILU>(map_w, maps_x, p, work, stream);
  return launch_experts<KIND_GELU>(map_w, maps_x, p, work, stream);
}
