// Paged causal attention, one block per (token, query head), float32 arithmetic throughout.
// It is the attention of the true 32-bit path and the plain device reference for the
// tensor-core attention kernels.  Query token t of sequence r, at position pos, attends the
// keys at positions 0..pos of r, found through r's block table; query head h reads key/value
// head h / (heads / kv_heads).  Keys are walked in chunks of 128 aligned to absolute position
// with a running maximum and sum, so the operations done for a query do not depend on how
// the tokens were cut into steps or on what else is in the batch.
//
// attention_tile (float32, head sizes 64 and 128, steps with prompt portions): the same operations in the same order for every
// query, for 32 tokens of a request at once, so that a chunk's keys and values are read once for all of them from shared memory
// instead of once per token from L2.  A warp has 4 tokens; a lane has 4 keys of the chunk in the scores and 2 (4) output
// elements in the values.  Bound by shared-memory reads.  512 tokens, 14 heads of 64: 557 us a token and head at a time, 70 us so.
#include "common.cuh"

namespace {

constexpr int CHUNK = 128;   // keys per pass == threads per block

template <typename T>
__global__ void __launch_bounds__(CHUNK)
attention_simple_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ k_cache,
                        const T* __restrict__ v_cache, const int* __restrict__ block_table, int table_stride,
                        const int* __restrict__ seq_of_token, const int* __restrict__ positions,
                        T* __restrict__ out, int out_stride, int heads, int kv_heads, int head_dim,
                        int page_tokens, int num_pages, int* status) {
  extern __shared__ float smem[];
  float* qs = smem;                       // head_dim
  float* probs = qs + head_dim;           // CHUNK
  float* scratch = probs + CHUNK;         // 33
  long long* row_offset = (long long*)(scratch + 34);   // CHUNK (8-byte aligned: sizes below are even)

  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int g = h / (heads / kv_heads);
  const int seq = seq_of_token[t];
  const int pos = positions[t];
  const int* table = block_table + (size_t)seq * table_stride;

  for (int d = tid; d < head_dim; d += CHUNK) qs[d] = to_float(q[(size_t)t * q_stride + h * head_dim + d]);
  __syncthreads();

  const float root = sqrtf((float)head_dim);
  float m_run = -INFINITY, l_run = 0.f;
  float acc0 = 0.f, acc1 = 0.f;           // output dims tid and tid + CHUNK

  for (int base = 0; base <= pos; base += CHUNK) {
    const int p = base + tid;
    bool valid = p <= pos;
    long long offset = 0;
    if (valid) {
      const int page = table[p / page_tokens];
      if (page < 0 || page >= num_pages) {
        atomicOr(status, SPROUT_STATUS_BAD_PAGE);
        valid = false;
      } else {
        offset = (((long long)page * kv_heads + g) * page_tokens + (p % page_tokens)) * head_dim;
      }
    }
    float s = -INFINITY;
    if (valid) {
      const T* key = k_cache + offset;
      float dot = 0.f;
      for (int d = 0; d < head_dim; d++) dot = fmaf(qs[d], to_float(key[d]), dot);
      s = dot / root;
    }
    row_offset[tid] = valid ? offset : -1;
    const float c_max = block_max(s, scratch);
    const float m_new = fmaxf(m_run, c_max);
    const float e = valid ? expf(s - m_new) : 0.f;
    probs[tid] = e;
    const float c_sum = block_sum(e, scratch);   // has barriers: probs and row_offset are visible after it
    const float alpha = (m_run == -INFINITY) ? 0.f : expf(m_run - m_new);
    l_run = l_run * alpha + c_sum;
    acc0 *= alpha;
    acc1 *= alpha;
    const int count = min(CHUNK, pos - base + 1);
    if (tid < head_dim) {
      for (int j = 0; j < count; j++) {
        const long long off = row_offset[j];
        if (off >= 0) acc0 = fmaf(probs[j], to_float(v_cache[off + tid]), acc0);
      }
    }
    if (tid + CHUNK < head_dim) {
      for (int j = 0; j < count; j++) {
        const long long off = row_offset[j];
        if (off >= 0) acc1 = fmaf(probs[j], to_float(v_cache[off + tid + CHUNK]), acc1);
      }
    }
    m_run = m_new;
    __syncthreads();
  }
  T* dst = out + (size_t)t * out_stride + h * head_dim;
  if (tid < head_dim) dst[tid] = from_float<T>(acc0 / l_run);
  if (tid + CHUNK < head_dim) dst[tid + CHUNK] = from_float<T>(acc1 / l_run);
}

constexpr int TILE = 32, TILE_THREADS = 256, TILE_ROWS = 4;      // tokens of a block, and of a warp

template <int HD>
constexpr size_t tile_smem() { return (size_t)(CHUNK * (HD + 4) + CHUNK * HD + TILE * HD + TILE * CHUNK) * sizeof(float) + CHUNK * sizeof(long long); }

template <int HD>
__global__ void __launch_bounds__(TILE_THREADS)
attention_tile_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                      const int* __restrict__ block_table, int table_stride, const int* __restrict__ q_start,
                      const int* __restrict__ positions, float* __restrict__ out, int out_stride, int requests, int heads, int kv_heads,
                      int page_tokens, int num_pages, int* status) {
  constexpr int K_STRIDE = HD + 4, DIMS = HD / 32;               // elements of the output a lane holds
  extern __shared__ __align__(16) float smem[];
  float* ks = smem;                                              // CHUNK x K_STRIDE
  float* vs = ks + CHUNK * K_STRIDE;                             // CHUNK x HD
  float* qs = vs + CHUNK * HD;                                   // TILE x HD
  float* probs = qs + TILE * HD;                                 // TILE x CHUNK
  long long* row_offset = (long long*)(probs + TILE * CHUNK);    // CHUNK; -1: no such key
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, g = h / (heads / kv_heads);
  int r, tile, tiles;
  if (!warp_find_piece(q_start, requests, TILE, blockIdx.x, r, tile, tiles)) return;
  const int first = q_start[r] + (tiles - 1 - tile) * TILE;      // a request's last tokens see most keys: they start first
  const int rows = min(TILE, q_start[r + 1] - first);
  const int* table = block_table + (size_t)r * table_stride;
  for (int i = tid; i < TILE * HD; i += TILE_THREADS) {
    const int row = i / HD, d = i % HD;
    qs[i] = row < rows ? q[(size_t)(first + row) * q_stride + h * HD + d] : 0.f;
  }
  const int own = lane < rows ? positions[first + lane] : -1;
  const int top = __reduce_max_sync(0xffffffffu, own);
  int pos[TILE_ROWS], most = -1, least = 0x7fffffff;             // this warp's rows; most and least among those that exist
#pragma unroll
  for (int i = 0; i < TILE_ROWS; i++) {
    pos[i] = __shfl_sync(0xffffffffu, own, warp * TILE_ROWS + i);
    most = max(most, pos[i]);
    if (warp * TILE_ROWS + i < rows) least = min(least, pos[i]);
  }
  const float root = sqrtf((float)HD);
  float m_run[TILE_ROWS], l_run[TILE_ROWS], acc[TILE_ROWS][DIMS];
#pragma unroll
  for (int i = 0; i < TILE_ROWS; i++) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int e = 0; e < DIMS; e++) acc[i][e] = 0.f;
  }
  for (int base = 0; base <= top; base += CHUNK) {
    __syncthreads();                                             // the chunk before has been used
    if (tid < CHUNK) {
      const int p = base + tid;
      long long offset = -1;
      if (p <= top) {
        const int page = table[p / page_tokens];
        if (page < 0 || page >= num_pages) atomicOr(status, SPROUT_STATUS_BAD_PAGE);
        else offset = (((long long)page * kv_heads + g) * page_tokens + (p % page_tokens)) * HD;
      }
      row_offset[tid] = offset;
    }
    __syncthreads();
    for (int i = tid; i < CHUNK * HD / 4; i += TILE_THREADS) {
      const int key = i / (HD / 4), d = 4 * (i % (HD / 4));
      const long long offset = row_offset[key];
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      *(float4*)&ks[key * K_STRIDE + d] = offset >= 0 ? *(const float4*)(k_cache + offset + d) : zero;
      *(float4*)&vs[key * HD + d] = offset >= 0 ? *(const float4*)(v_cache + offset + d) : zero;
    }
    __syncthreads();
    if (base > most) continue;                                   // no key of the chunk is this warp's
    float s[TILE_ROWS][4];
#pragma unroll
    for (int i = 0; i < TILE_ROWS; i++)
#pragma unroll
      for (int c = 0; c < 4; c++) s[i][c] = 0.f;
#pragma unroll 4
    for (int d = 0; d < HD; d += 4) {
      float4 key[4], query[TILE_ROWS];
#pragma unroll
      for (int c = 0; c < 4; c++) key[c] = *(const float4*)&ks[(lane + 32 * c) * K_STRIDE + d];
#pragma unroll
      for (int i = 0; i < TILE_ROWS; i++) query[i] = *(const float4*)&qs[(warp * TILE_ROWS + i) * HD + d];
#pragma unroll
      for (int i = 0; i < TILE_ROWS; i++)
#pragma unroll
        for (int c = 0; c < 4; c++)
          s[i][c] = fmaf(query[i].w, key[c].w, fmaf(query[i].z, key[c].z, fmaf(query[i].y, key[c].y, fmaf(query[i].x, key[c].x, s[i][c]))));
    }
    bool there[4];
#pragma unroll
    for (int c = 0; c < 4; c++) there[c] = row_offset[lane + 32 * c] >= 0;
#pragma unroll
    for (int i = 0; i < TILE_ROWS; i++) {
      float c_max = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        s[i][c] = there[c] && base + lane + 32 * c <= pos[i] ? s[i][c] / root : -INFINITY;
        c_max = fmaxf(c_max, s[i][c]);
      }
      c_max = warp_max(c_max);
      const float m_new = fmaxf(m_run[i], c_max);
      float sum[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float e = there[c] && base + lane + 32 * c <= pos[i] ? expf(s[i][c] - m_new) : 0.f;
        probs[(warp * TILE_ROWS + i) * CHUNK + lane + 32 * c] = e;
        sum[c] = warp_sum(e);
      }
      const float c_sum = (sum[0] + sum[2]) + (sum[1] + sum[3]);           // the order of block_sum over four warps
      const float alpha = (m_run[i] == -INFINITY) ? 0.f : expf(m_run[i] - m_new);
      l_run[i] = l_run[i] * alpha + c_sum;
#pragma unroll
      for (int e = 0; e < DIMS; e++) acc[i][e] *= alpha;
      m_run[i] = m_new;
    }
    __syncwarp();
    // a key that a row does not see is not multiplied into it (its value may be infinite): whole groups of four keys that all
    // rows see, then key by key
    const int count = min(CHUNK, most - base + 1), shared_count = min(count, least - base + 1) & ~3;
    for (int j = 0; j < count; j += 4) {
      float p[TILE_ROWS][4], v[4][DIMS];
#pragma unroll
      for (int i = 0; i < TILE_ROWS; i++) *(float4*)p[i] = *(const float4*)&probs[(warp * TILE_ROWS + i) * CHUNK + j];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if (DIMS == 2) *(float2*)v[e] = *(const float2*)&vs[(j + e) * HD + lane * 2];
        else *(float4*)v[e] = *(const float4*)&vs[(j + e) * HD + lane * 4];
      }
      const bool all = j < shared_count;
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int i = 0; i < TILE_ROWS; i++)
          if (all || base + j + e <= pos[i])
#pragma unroll
            for (int x = 0; x < DIMS; x++) acc[i][x] = fmaf(p[i][e], v[e][x], acc[i][x]);
    }
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < TILE_ROWS; i++) {
    const int row = warp * TILE_ROWS + i;
    if (row >= rows) continue;
#pragma unroll
    for (int e = 0; e < DIMS; e++) out[(size_t)(first + row) * out_stride + h * HD + lane * DIMS + e] = acc[i][e] / l_run[i];
  }
}

template <int HD>
int launch_tile(const float* q, int q_stride, const float* k_cache, const float* v_cache, const int* block_table, int table_stride,
                const int* q_start, const int* positions, float* out, int out_stride, int tokens, int requests, int heads, int kv_heads,
                int page_tokens, int num_pages, int* status, cudaStream_t stream) {
  const cudaError_t error = cudaFuncSetAttribute(attention_tile_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem<HD>());
  if (error != cudaSuccess) return sprout_fail("attention_tile: %s", cudaGetErrorString(error));
  // blocks for any cutting of the tokens into the requests: a captured launch is replayed for others than its own
  sprout_launch(attention_tile_kernel<HD>, dim3(tokens / TILE + requests, heads), dim3(TILE_THREADS), tile_smem<HD>(), stream,
                q, q_stride, k_cache, v_cache, block_table, table_stride, q_start, positions, out, out_stride, requests, heads, kv_heads, page_tokens,
                num_pages, status);
  return sprout_check_launch("attention_tile");
}

}  // namespace

// float32, head_dim 64 or 128; the caches' rows start on 16-byte boundaries.  q_start: the requests' first tokens and, last, the
// number of tokens (`tokens`).
SPROUT_API int sprout_attention_tile(const void* q, int q_stride, const void* k_cache, const void* v_cache, const int* block_table,
                                     int table_stride, const int* q_start, const int* positions, void* out, int out_stride, int tokens,
                                     int requests, int heads, int kv_heads, int head_dim, int page_tokens, int num_pages, int* status,
                                     cudaStream_t stream) {
  SPROUT_REQUIRE(requests > 0 && tokens > 0 && heads > 0 && kv_heads > 0 && page_tokens > 0 && num_pages > 0, "attention_tile: sizes must be positive");
  SPROUT_REQUIRE(heads % kv_heads == 0, "attention_tile: heads (%d) must be a multiple of kv_heads (%d)", heads, kv_heads);
  SPROUT_REQUIRE(heads <= 65535, "attention_tile: too many heads (%d)", heads);
  SPROUT_REQUIRE(q && k_cache && v_cache && block_table && q_start && positions && out && status, "attention_tile: null pointer");
  SPROUT_REQUIRE((uintptr_t)k_cache % 16 == 0 && (uintptr_t)v_cache % 16 == 0, "attention_tile: the caches must start on 16-byte boundaries");
  if (head_dim == 64)
    return launch_tile<64>((const float*)q, q_stride, (const float*)k_cache, (const float*)v_cache, block_table, table_stride, q_start, positions,
                           (float*)out, out_stride, tokens, requests, heads, kv_heads, page_tokens, num_pages, status, stream);
  if (head_dim == 128)
    return launch_tile<128>((const float*)q, q_stride, (const float*)k_cache, (const float*)v_cache, block_table, table_stride, q_start, positions,
                            (float*)out, out_stride, tokens, requests, heads, kv_heads, page_tokens, num_pages, status, stream);
  return sprout_fail("attention_tile: head_dim must be 64 or 128 (got %d)", head_dim);
}

SPROUT_API int sprout_attention_simple(const void* q, int q_stride, const void* k_cache, const void* v_cache,
                                       const int* block_table, int table_stride, const int* seq_of_token,
                                       const int* positions, void* out, int out_stride, int dtype,
                                       int num_tokens, int heads, int kv_heads, int head_dim, int page_tokens,
                                       int num_pages, int* status, cudaStream_t stream) {
  SPROUT_REQUIRE(num_tokens > 0 && heads > 0 && kv_heads > 0 && page_tokens > 0 && num_pages > 0,
                 "attention_simple: sizes must be positive");
  SPROUT_REQUIRE(heads % kv_heads == 0, "attention_simple: heads (%d) must be a multiple of kv_heads (%d)", heads, kv_heads);
  SPROUT_REQUIRE(head_dim > 0 && head_dim % 2 == 0 && head_dim <= 2 * CHUNK,
                 "attention_simple: head_dim must be even and at most %d (got %d)", 2 * CHUNK, head_dim);
  SPROUT_REQUIRE(heads <= 65535, "attention_simple: too many heads (%d)", heads);
  SPROUT_REQUIRE(q && k_cache && v_cache && block_table && seq_of_token && positions && out && status,
                 "attention_simple: null pointer");
  const size_t smem = (size_t)(head_dim + CHUNK + 34) * sizeof(float) + CHUNK * sizeof(long long);
  dim3 grid(num_tokens, heads);
  if (dtype == SPROUT_F32)
    sprout_launch(attention_simple_kernel<float>, grid, dim3(CHUNK), smem, stream, 
        (const float*)q, q_stride, (const float*)k_cache, (const float*)v_cache, block_table, table_stride,
        seq_of_token, positions, (float*)out, out_stride, heads, kv_heads, head_dim, page_tokens, num_pages, status);
  else if (dtype == SPROUT_BF16)
    sprout_launch(attention_simple_kernel<__nv_bfloat16>, grid, dim3(CHUNK), smem, stream, 
        (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache,
        block_table, table_stride, seq_of_token, positions, (__nv_bfloat16*)out, out_stride, heads, kv_heads,
        head_dim, page_tokens, num_pages, status);
  else
    return sprout_fail("attention_simple: unknown dtype %d", dtype);
  return sprout_check_launch("attention_simple");
}
