// Prompt attention over the paged cache on the fifth-generation tensor cores (sm_100a), one or two softmax maps per head
// over shared values: the bfloat16 kernel behind multimap_attention for steps with prompt portions.
//
// A CTA owns two Q tiles of 128 rows.  One map per head: 256 rows, a row being a (token, query head) pair of one request and one
// key/value head.  Two maps: 128 rows, the first tile their map 0, the second their map 1.  It walks the keys in tiles of 64:
//
//   S = Q K^T    tcgen05.mma, Q and K K-major in shared memory, S [128 x 64] in tensor memory, two buffers per Q tile
//   softmax      a warpgroup per Q tile, one thread per row: S into registers, masks, cap, P = exp2(..) as bfloat16 back into tensor
//                memory, over the first half of S's columns
//   O += P V     tcgen05.mma with P from tensor memory, V as it lies in the cache (MN-major); O stays in tensor memory
//
// S of the next tile is ready when a warpgroup has written P.  (128 keys a tile and one buffer of S: the warpgroups waited 1,800 of
// 4,500 cycles a tile for P V and S.)  A row's O and sum follow its maximum, so that the largest weight is 1 and those near it use
// the bfloat16 they multiply V in best: left behind until the maximum had grown by 2^8, which reads O back hardly ever, weights of up to
// 2^8 were rounded where the step is twice as wide, and results were 1 to 2 % further from 64-bit ones.  The sum is that of the weights in float32.
// S of tile j + 2 goes over the columns of P of tile j: one thread issues all products, and the tensor cores take them in order.
//
// What bounds it: the exponentials (16 an SM and cycle: 1,024 cycles for a pair of tiles, beside 900 to 1,280 of products).
// Measured, prompts of 2,048 tokens, 16 heads, two maps of 64 with values of 128: 167 us on mma.sync, 64 us here; layers: this one 297 and
// 144 us, one map with a window of 1,024, five prompts of 4,001 tokens together, 319 and 183 us.
//
// A piece (the CTA's rows) with many key tiles may be divided among `shares` CTAs, each taking every shares-th tile: partial sums
// go to scratch memory, and the CTA that finds all the others counted in merges them.  Nobody waits for anybody.
//
// K and V come by TMA, one box per page, through a ring of stages.  Every mbarrier wait is bounded: on a timeout the CTA sets
// the status word, waits (bounded) for its copies in flight, frees its tensor memory and returns.
#include <cuda_bf16.h>

#include "common.cuh"
#include "maps_attention.cuh"
#include "tcgen05.cuh"

using namespace sprout_maps;

namespace {

constexpr int ROWS = 128, KEYS = 64;        // rows of a Q tile (tensor-memory lanes), keys of a tile
constexpr int THREADS = 384;                // warpgroup 0: key copies, MMA, value copies (one warp idle); 1, 2: softmax of Q tile 0, 1
constexpr int ATOM = 128 * 128;             // bytes of a [128 rows, 64 bf16] swizzled tile
constexpr int KV_ATOM = KEYS * 128;         // and of [KEYS rows, 64 bf16]
constexpr int TMEM_COLS = 512;
constexpr int MAX_SHARES = 4;
constexpr int MIN_SHARE_TILES = 6;          // a share of fewer key tiles costs more than it saves

template <int DIM, int VDIM, int MAPS>
struct Layout {
  static constexpr int Q_BYTES = DIM / 64 * ATOM;                  // one Q tile
  static constexpr int K_BYTES = MAPS * DIM / 64 * KV_ATOM, V_BYTES = VDIM / 64 * KV_ATOM;
  static constexpr int STAGES = 5;
  static constexpr int OFF_K = 2 * Q_BYTES, OFF_V = OFF_K + STAGES * K_BYTES, OFF_BAR = OFF_V + STAGES * V_BYTES;
  static constexpr int OFF_SUMS = OFF_BAR + 512;                   // 128 pairs: map 1's maxima and sums
  static constexpr int SMEM = OFF_SUMS + 1024;
  static constexpr int O_COLUMN = 4 * KEYS;                        // tensor memory: S of the Q tiles, two buffers each, then their O
  static constexpr int CTA_ROWS = MAPS == 1 ? 2 * ROWS : ROWS;
  static constexpr int SHARE_FLOATS = 2 * ROWS * (VDIM + 4);       // a share's partial results
  static_assert(O_COLUMN + 2 * VDIM <= TMEM_COLS, "tensor memory columns");
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pair(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// 2^x, the hardware approximation; results below the normal range are zero
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// D (+)= A B from shared memory, the descriptors as words.
__device__ __forceinline__ void umma_bf16_words(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %6, 0;\n mov.b64 a, {%1, %2};\n mov.b64 b, {%3, %4};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
// The same with A [128 rows, 16] from tensor memory (two bfloat16 a 32-bit column).
__device__ __forceinline__ void umma_bf16_from_tmem_words(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 b;\n setp.ne.b32 p, %5, 0;\n mov.b64 b, {%2, %3};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void named_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Among how many CTAs a piece's key tiles go when the launch has `pieces` of them, a request's last piece `last` tiles and its first
// `first`.  As many as leave every CTA an SM; two where all pieces have one but lengths differ so much that the longest would run
// alone for long (a CTA takes some 9 us and 1.2 us a tile, 4 us more when it is divided, and a second round of CTAs starts late).
// Head size 128, 512 queries over 900 cached tokens, 64 heads over 8 (128 pieces of 15 to 23 tiles): undivided 46 us, two shares, which two
// rounds of CTAs take, about 65; 4,096 tokens, 8 heads over 1 (128 pieces of 1 to 64 tiles): about 97 and 77 us.
__device__ __forceinline__ int shares_of(int pieces, int last, int first, int sms) {
  if (pieces > sms) return 1;
  if (2 * pieces <= sms) return sms / pieces;
  const float undivided = 9.f + 1.2f * last, divided = fmaxf(pieces * (26.f + 0.6f * (last + first)) / sms + 13.f, 26.f + 1.2f * first);
  return divided < undivided ? 2 : 1;
}

struct Params {
  MultiMapParams m;                    // what every kernel of this attention takes
  int box_rows;                        // cache rows of a TMA box
  int shares, sms;                     // CTAs that a piece's key tiles may be divided among; SMs of the device
  float* scratch; int* counters;       // [pieces][shares] shares; [pieces][2], zero between launches
  // PACKED: the requests' keys and values lie side by side instead of in pages, each request's from its first visible tile on
  // (`packed_base`): a head's key is `key_atoms` times 64 columns of its own in map_k's rows and then the columns from `tail_col` of
  // map_v's rows, which the heads share; its values start at column `value_col` of map_k's rows
  int key_atoms, tail_col, value_col;
};

template <int DIM, int VDIM, int MAPS, bool PACKED>
__global__ void __launch_bounds__(THREADS, 1)
maps_attention_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const Params tc) {
  using L = Layout<DIM, VDIM, MAPS>;
  constexpr int KW = MAPS * DIM, NS = L::STAGES;
  const MultiMapParams& p = tc.m;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sK = smem + L::OFF_K;
  uint8_t* sV = smem + L::OFF_V;
  uint64_t* bars = (uint64_t*)(smem + L::OFF_BAR);
  uint64_t* k_full = bars;             // [NS] copies of a stage have landed
  uint64_t* k_empty = k_full + NS;     // the products that read a stage have completed
  uint64_t* v_full = k_empty + NS;
  uint64_t* v_empty = v_full + NS;
  uint64_t* s_full = v_empty + NS;     // [2 Q tiles][2 buffers] S is complete in tensor memory
  uint64_t* p_full = s_full + 4;       // [2][2] P is in tensor memory (4 warps arrive)
  uint64_t* o_done = p_full + 4;       // [2][2] P V of a Q tile's key tile is complete, for even and odd tiles (a waiter may be two behind)
  constexpr int BARS = 4 * NS + 12;
  static_assert(BARS * 8 + 16 <= 512, "room for the barriers");
  uint32_t* tmem_slot = (uint32_t*)(bars + BARS);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  int* seen = (int*)(tmem_slot + 2);   // [2]
  float2* sums1 = (float2*)(smem + L::OFF_SUMS);

  // before the wait for the step's earlier kernels: the request's bounds and positions and the block table, written before the
  // step's first kernel
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int piece_index = blockIdx.x / tc.shares, rank = blockIdx.x % tc.shares;
  const int g = piece_index % p.kv_heads, group = p.heads / p.kv_heads;
  // the pieces of a request are handed out from the last (the longest under the causal mask) to the first, the heads of a
  // piece side by side
  int r = 0, piece = piece_index / p.kv_heads;
  for (; r < p.requests; r++) {
    const int pieces = ((p.q_start[r + 1] - p.q_start[r]) * group + L::CTA_ROWS - 1) / L::CTA_ROWS;
    if (piece < pieces) { piece = pieces - 1 - piece; break; }
    piece -= pieces;
  }
  if (r >= p.requests) return;
  if ((smem_u32(smem) & 1023) != 0) {
    if (tid == 0) atomicOr(p.status, SPROUT_STATUS_BAD_LAYOUT);
    return;
  }
  const int q0 = p.q_start[r], rows_total = (p.q_start[r + 1] - q0) * group, row_base = piece * L::CTA_ROWS;
  const int* table = p.block_table + (size_t)r * p.table_stride;
  // positions grow with the row index, and so does the first visible key
  const bool two = MAPS == 2 || row_base + ROWS < rows_total;             // the second Q tile has rows
  const int limit_a = p.positions[q0 + (min(rows_total, row_base + ROWS) - 1) / group];
  const int max_limit = MAPS == 1 && two ? p.positions[q0 + (min(rows_total, row_base + L::CTA_ROWS) - 1) / group] : limit_a;
  const int min_lo = first_visible(p.mask_kind, p.mask_size, p.positions[q0 + row_base / group]);
  // the piece's key tiles: those of the kept first positions that lie before the window's, then the window's up to the last query
  const int tile_lo = min_lo / KEYS, keep_tiles = min((p.mask_keep + KEYS - 1) / KEYS, tile_lo);
  auto tile_of = [&](int i) { return i < keep_tiles ? i : tile_lo + (i - keep_tiles); };
  const int all_tiles = keep_tiles + max(0, max_limit / KEYS + 1 - tile_lo);
  const int all_tiles_a = min(all_tiles, keep_tiles + max(0, limit_a / KEYS + 1 - tile_lo));
  int shares = 1;
  if (tc.shares > 1) {
    // every thread takes the same decision: the launch's pieces, and the tiles of the request's last and first piece
    int pieces = 0;
    for (int base = 0; base < p.requests; base += 32) {
      const int i = base + lane;
      pieces += i < p.requests ? ((p.q_start[i + 1] - p.q_start[i]) * group + L::CTA_ROWS - 1) / L::CTA_ROWS : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pieces += __shfl_xor_sync(0xffffffffu, pieces, o);
    const int lo = first_visible(p.mask_kind, p.mask_size, p.positions[q0]), end = p.positions[p.q_start[r + 1] - 1];
    const int last_tiles = (end - first_visible(p.mask_kind, p.mask_size, end)) / KEYS + 1, first_tiles = (p.positions[q0] - lo) / KEYS + 1;
    shares = max(1, min(min(tc.shares, shares_of(pieces * p.kv_heads, last_tiles, first_tiles, tc.sms)), all_tiles / MIN_SHARE_TILES));
  }
  if (rank >= shares) return;
  // below, j counts the CTA's own tiles: rank + shares * j is the index among the piece's
  const int n_tiles = (all_tiles - rank + shares - 1) / shares;
  const int tiles_a = MAPS == 2 ? n_tiles : max(0, (all_tiles_a - rank + shares - 1) / shares);
  auto key_of = [&](int j) { return tile_of(rank + shares * j) * KEYS; };
  int packed_at = 0;                                  // the packed row of the request's position 0, if it were there
  if (PACKED) {
    for (int i = 0; i < r; i++)
      packed_at += p.positions[p.q_start[i + 1] - 1] + 1 - packed_base(p.mask_kind, p.mask_size, p.positions[p.q_start[i]]);
    packed_at -= packed_base(p.mask_kind, p.mask_size, p.positions[q0]);
  }

  // rows of a stage that no copy fills must hold finite numbers: their probabilities are zero, and zero times a NaN is not
  for (int i = tid; i < NS * L::V_BYTES / 16; i += THREADS) ((uint4*)sV)[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    for (int i = 0; i < BARS; i++) mbar_init(&bars[i], &bars[i] >= p_full && &bars[i] < o_done ? 4 : 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  pdl_wait();

  // Q rows -> shared memory, K-major with the 128-byte swizzle (16-byte chunk c of row r at position c ^ (r & 7))
  constexpr int CHUNKS = DIM / 8;
  for (int idx = tid; idx < 2 * ROWS * CHUNKS; idx += THREADS) {
    const int crow = idx / CHUNKS, c = idx % CHUNKS, q = crow >> 7, row = crow & (ROWS - 1);
    const int gi = row_base + (MAPS == 1 ? crow : row);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (gi < rows_total)
      v = *(const uint4*)(p.q + (size_t)(q0 + gi / group) * p.q_stride + (size_t)(g * group + gi % group) * KW + (MAPS == 2 ? q * DIM : 0) + c * 8);
    *(uint4*)(sQ + q * L::Q_BYTES + (c >> 3) * ATOM + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = v;
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  int issued = 0;                                     // tiles whose copies were issued (copy warps)
  auto gave_up = [&]() { *abort_flag = 1; atomicOr(p.status, SPROUT_STATUS_WAIT_TIMEOUT); };
  if (warp < 4) {
    warpgroup_regs_give<104>();
    if (warp == 0 || warp == 2) {
      // ---------------- copies, keys by warp 0 and values by warp 2 (the issue of one box takes some 60 cycles, and a tile of
      // 16-token pages has 8 to 16): one TMA box per page (or per KEYS keys of a larger page); lane b issues box b's copies, lane 0
      // waits for the stage and posts the bytes.  The page of a tile is looked up while the tile before waits and is copied.
      const bool keys = warp == 0;
      const CUtensorMap* map = keys ? &map_k : &map_v;
      uint64_t* full = keys ? k_full : v_full;
      uint64_t* empty = keys ? k_empty : v_empty;
      const uint32_t stages = smem_u32(keys ? sK : sV), stage_bytes = keys ? L::K_BYTES : L::V_BYTES;
      const int atoms = keys ? KW / 64 : VDIM / 64, boxes = PACKED ? 1 : KEYS / tc.box_rows;
      auto box_key = [&](int j) {                     // the first key of this lane's box of tile j, -1 if no row sees any of it
        if (lane >= boxes || j >= n_tiles) return -1;
        const int key = key_of(j) + lane * tc.box_rows;
        return key > max_limit || (key + tc.box_rows <= min_lo && key >= p.mask_keep) ? -1 : key;
      };
      int key = box_key(0);
      int page = !PACKED && key >= 0 ? table[key / p.page_tokens] : 0;
      for (int j = 0; j < n_tiles; j++) {
        const int s = j % NS;
        const bool bad = !PACKED && key >= 0 && (page < 0 || page >= p.num_pages);
        if (bad) atomicOr(p.status, SPROUT_STATUS_BAD_PAGE);
        const int row_at = key < 0 || bad ? -1 : PACKED ? packed_at + key : (page * p.kv_heads + g) * p.page_tokens + key % p.page_tokens;
        key = box_key(j + 1);
        if (!PACKED && key >= 0) page = table[key / p.page_tokens];
        const uint32_t bytes = (uint32_t)__popc(__ballot_sync(0xffffffffu, row_at >= 0)) * tc.box_rows * 128 * atoms;
        bool ok = true;
        if (lane == 0) {
          ok = !*abort_flag && mbar_wait(&empty[s], ((j / NS) & 1) ^ 1, abort_flag);
          if (ok) mbar_expect_tx(&full[s], bytes);
          else gave_up();
        }
        if (!__shfl_sync(0xffffffffu, ok, 0)) break;
        if (row_at >= 0)
          for (int a = 0; a < atoms; a++) {
            const uint32_t to = stages + s * stage_bytes + a * KV_ATOM + lane * tc.box_rows * 128;
            if (!PACKED) tma_load_2d_addr(to, map, smem_u32(&full[s]), a * 64, row_at);
            else if (!keys) tma_load_2d_addr(to, &map_k, smem_u32(&full[s]), tc.value_col + g * VDIM + a * 64, row_at);
            else if (a < tc.key_atoms) tma_load_2d_addr(to, &map_k, smem_u32(&full[s]), (g * tc.key_atoms + a) * 64, row_at);
            else tma_load_2d_addr(to, &map_v, smem_u32(&full[s]), tc.tail_col + (a - tc.key_atoms) * 64, row_at);
          }
        issued = j + 1;
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer: S(0) and S(1) of both Q tiles, then for every key tile and Q tile  [P(j)] P V(j), S(j + 2).
      // The second Q tile has at least the first one's tiles, or none; the last product that reads a stage releases it.
      // The whole warp walks the loop on values that are the same in all lanes (they stay in uniform registers, where the products
      // take them from); one elected lane issues.
      const uint32_t idesc_s = umma_idesc(ROWS, KEYS), idesc_o = umma_idesc_b_mn(ROWS, VDIM);
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      const int tiles_1 = __shfl_sync(0xffffffffu, n_tiles, 0), tiles_0 = __shfl_sync(0xffffffffu, tiles_a, 0);
      const bool both = __shfl_sync(0xffffffffu, (int)two, 0) != 0;
      const uint32_t k0 = (smem_u32(sK) & 0x3FFFF) >> 4, v0 = (smem_u32(sV) & 0x3FFFF) >> 4, q0_lo = (smem_u32(sQ) & 0x3FFFF) >> 4;
      const uint32_t bar0 = smem_u32(bars);
      auto bar_of = [&](const uint64_t* bar) { return bar0 + (uint32_t)((const char*)bar - (const char*)bars); };
      auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_addr(bar, parity, abort_flag)) != 0; };
      // descriptors: the start address / 16 in the low word, layout constants (umma_smem_desc, umma_smem_desc_mn) in the high one
      constexpr uint32_t DESC_HI = (1024 >> 4) | (1u << 14) | (2u << 29);
      auto issue_s = [&](int q, int stage, int buf) {
        if (elect_one()) {
#pragma unroll
          for (int a = 0; a < DIM / 64; a++)
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
              umma_bf16_words(tmem + (q * 2 + buf) * KEYS, q0_lo + (q * L::Q_BYTES + a * ATOM) / 16 + 2 * kk, DESC_HI,
                              k0 + stage * (L::K_BYTES / 16) + ((MAPS == 2 ? q * (DIM / 64) : 0) + a) * (KV_ATOM / 16) + 2 * kk, DESC_HI, idesc_s, (a | kk) != 0);
          umma_commit_addr(bar_of(s_full) + (q * 2 + buf) * 8);
          if (q == 1 || !both) umma_commit_addr(bar_of(k_empty) + stage * 8);
        }
        __syncwarp();
      };
      auto issue_pv = [&](int q, int stage, int buf, bool first) {
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < KEYS / 16; ks++)
            umma_bf16_from_tmem_words(tmem + L::O_COLUMN + q * VDIM, tmem + (q * 2 + buf) * KEYS + ks * 8,
                                      (v0 + stage * (L::V_BYTES / 16) + ks * 128) | ((uint32_t)(KV_ATOM >> 4) << 16), DESC_HI, idesc_o, !first || ks != 0);
          umma_commit_addr(bar_of(o_done) + (q * 2 + buf) * 8);
          if (q == 1 || !both) umma_commit_addr(bar_of(v_empty) + stage * 8);
        }
        __syncwarp();
      };
      bool ok = true;
      int k_stage = 0, v_stage = 0;                    // running stages and parities of the rings
      uint32_t k_parity = 0, v_parity = 0;
      for (int j = 0; j < min(2, tiles_1) && ok; j++) {
        ok = wait(bar_of(k_full) + k_stage * 8, 0);
        if (!ok) break;
        tc_fence_after();
        if (j < tiles_0) issue_s(0, k_stage, j);
        if (both) issue_s(1, k_stage, j);
        k_stage++;
      }
      for (int j = 0; j < tiles_1 && ok; j++) {
        const int buf = j & 1;
        const uint32_t parity = (j >> 1) & 1;
        ok = wait(bar_of(v_full) + v_stage * 8, v_parity);
        if (ok && j + 2 < tiles_1) ok = wait(bar_of(k_full) + k_stage * 8, k_parity);
        if (!ok) break;
        if (j < tiles_0) {
          ok = wait(bar_of(p_full) + buf * 8, parity);
          if (!ok) break;
          tc_fence_after();
          issue_pv(0, v_stage, buf, j == 0);
          if (j + 2 < tiles_0) issue_s(0, k_stage, buf);
        }
        if (both) {
          ok = wait(bar_of(p_full) + (2 + buf) * 8, parity);
          if (!ok) break;
          tc_fence_after();
          issue_pv(1, v_stage, buf, j == 0);
          if (j + 2 < tiles_1) issue_s(1, k_stage, buf);
        }
        if (++k_stage == NS) { k_stage = 0; k_parity ^= 1; }
        if (++v_stage == NS) { v_stage = 0; v_parity ^= 1; }
      }
      if (!ok && lane == 0) gave_up();
    }
  } else {
    // ---------------- softmax: a warpgroup per Q tile, one thread per row
    warpgroup_regs_take<200>();
    const int q = (warp >> 2) - 1;
    const int my_tiles = q == 0 ? tiles_a : (two ? n_tiles : 0);
    const int quarter = warp & 3, row = quarter * 32 + lane;         // a warp reads tensor-memory lanes 32 * (warp % 4) on
    const int gi = row_base + (MAPS == 1 ? q * ROWS : 0) + row;
    const bool row_valid = gi < rows_total;
    const int token = q0 + (row_valid ? gi / group : 0), head = g * group + gi % group;
    const int limit = row_valid ? p.positions[token] : -1;           // last visible key of the row
    const int lo = row_valid ? first_visible(p.mask_kind, p.mask_size, limit) : 0;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t o_addr = lane_addr + L::O_COLUMN + q * VDIM;
    const float scale_log2 = score_scale(p) * 1.4426950408889634f;
    const uint64_t scale2 = pair(scale_log2, scale_log2);
    float m = -INFINITY;                               // the maximum that the sums stand for (unscaled scores)
    uint64_t l2 = 0ull;                                // the sum, as two partial sums
    bool ok = true;
    for (int j = 0; j < my_tiles; j++) {
      const uint32_t s_addr = lane_addr + (q * 2 + (j & 1)) * KEYS;
      ok = !*abort_flag && mbar_wait(&s_full[q * 2 + (j & 1)], (j >> 1) & 1, abort_flag);
      if (!ok) gave_up();
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int kv0 = key_of(j);
      uint32_t sc[KEYS / 32][32];
#pragma unroll
      for (int c = 0; c < KEYS / 32; c++) tmem_load32_issue(s_addr + c * 32, sc[c]);
#pragma unroll
      for (int c = 0; c < KEYS / 32; c++) tmem_load_wait(sc[c]);
      if (p.softcap > 0.f) {
        const float cap = p.softcap, pre = p.scale, inv_cap = 1.0f / cap;
#pragma unroll
        for (int c = 0; c < KEYS / 32; c++)
#pragma unroll
          for (int i = 0; i < 32; i++) sc[c][i] = __float_as_uint(soft_cap_fast(__uint_as_float(sc[c][i]) * pre, cap, inv_cap));
      }
      if (kv0 + KEYS - 1 > limit) {                    // some key of the tile lies beyond this row's limit
#pragma unroll
        for (int c = 0; c < KEYS / 32; c++)
#pragma unroll
          for (int i = 0; i < 32; i++) if (kv0 + c * 32 + i > limit) sc[c][i] = 0xff800000u;          // -inf
      }
      if (kv0 < lo) {                                  // or before its window or chunk
#pragma unroll
        for (int c = 0; c < KEYS / 32; c++)
#pragma unroll
          for (int i = 0; i < 32; i++) {
            const int key = kv0 + c * 32 + i;
            if (key < lo && key >= p.mask_keep) sc[c][i] = 0xff800000u;
          }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < KEYS / 32; c++)
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          mx[0] = max3(mx[0], __uint_as_float(sc[c][i]), __uint_as_float(sc[c][i + 1]));
          mx[1] = max3(mx[1], __uint_as_float(sc[c][i + 2]), __uint_as_float(sc[c][i + 3]));
          mx[2] = max3(mx[2], __uint_as_float(sc[c][i + 4]), __uint_as_float(sc[c][i + 5]));
          mx[3] = max3(mx[3], __uint_as_float(sc[c][i + 6]), __uint_as_float(sc[c][i + 7]));
        }
      const float n = max3(m, fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      // the maximum moved: bring O and the sum to it
      const bool moved = n != m;
      if (__any_sync(0xffffffffu, moved)) {
        const float alpha = !moved ? 1.0f : m == -INFINITY ? 0.f : exp2_fast((m - n) * scale_log2);
        if (moved) m = n;
        float lo2, hi2;
        unpair(l2, lo2, hi2);
        l2 = pair(lo2 * alpha, hi2 * alpha);
        if (j > 0) {
          ok = !*abort_flag && mbar_wait(&o_done[q * 2 + ((j - 1) & 1)], ((j - 1) >> 1) & 1, abort_flag);
          if (!ok) gave_up();
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          for (int c = 0; c < VDIM; c += 16) {
            uint32_t o[16];
            tmem_load16(o_addr + c, o);
#pragma unroll
            for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_store16(o_addr + c, o);
          }
        }
      }
      const float base = m == -INFINITY ? 0.f : m * scale_log2;
      const uint64_t nbase2 = pair(-base, -base);
      // probabilities, their sum, and P as bfloat16 into tensor memory
#pragma unroll
      for (int c = 0; c < KEYS / 32; c++) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float x0, x1;
          unpair(fma2(pair(sc[c][i], sc[c][i + 1]), scale2, nbase2), x0, x1);
          const float p0 = exp2_fast(x0), p1 = exp2_fast(x1);
          __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
          packed[i >> 1] = *(uint32_t*)&h;
          l2 = add2(l2, pair(p0, p1));
        }
        tmem_store16(s_addr + c * 16, packed);
      }
      tmem_store_wait();
      // V rows of keys that no row of the CTA sees (beyond the last query, before the window) may hold anything, in slots that
      // held other tokens: their probabilities are zero, but zero times a NaN is not.  They are cleared once the copy has landed,
      // by each Q tile before it signals its P.
      if (kv0 + KEYS - 1 > max_limit || (kv0 < min_lo && kv0 + KEYS > p.mask_keep)) {
        const int key = kv0 + row, s = j % NS;
        if (row < KEYS && (key > max_limit || (key < min_lo && key >= p.mask_keep))) {
          if (*abort_flag || !mbar_wait(&v_full[s], (j / NS) & 1, abort_flag)) gave_up();
#pragma unroll
          for (int a = 0; a < VDIM / 64; a++)
#pragma unroll
            for (int c = 0; c < 8; c++) *(uint4*)(sV + s * L::V_BYTES + a * KV_ATOM + row * 128 + c * 16) = make_uint4(0, 0, 0, 0);
          fence_proxy_async();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[q * 2 + (j & 1)]);
    }
    if (ok && my_tiles > 0) {
      ok = !*abort_flag && mbar_wait(&o_done[q * 2 + ((my_tiles - 1) & 1)], ((my_tiles - 1) >> 1) & 1, abort_flag);
      if (!ok) gave_up();
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
    }
    float l_lo, l_hi;
    unpair(l2, l_lo, l_hi);
    float l = l_lo + l_hi;

    // this thread's row of O: `weight` times the tile in tensor memory (nothing where the CTA had no tile)
    auto own_columns = [&](uint32_t addr, bool any, int c, float weight, float (&v)[32]) {
      uint32_t o[32];
      tmem_load32(addr + c * 32, o);
#pragma unroll
      for (int i = 0; i < 32; i++) v[i] = any ? __uint_as_float(o[i]) * weight : 0.f;
    };
    // a share's partial results: VDIM / 4 + 1 planes of 128 rows of float4 per Q tile, the last (maximum, sum, -, -)
    auto share_at = [&](int share, int tile) {
      return (float4*)(tc.scratch + ((size_t)piece_index * tc.shares + share) * L::SHARE_FLOATS) + (size_t)tile * (VDIM / 4 + 1) * ROWS + row;
    };
    const bool has_rows = MAPS == 2 || q == 0 || two;
    bool finishes = MAPS == 1 ? has_rows : q == 0;
    if (shares > 1 && has_rows) {
      float4* mine = share_at(rank, q);
      for (int c = 0; c < VDIM / 32; c++) {
        float v[32];
        own_columns(o_addr, my_tiles > 0, c, 1.0f, v);
#pragma unroll
        for (int i = 0; i < 8; i++) mine[(c * 8 + i) * ROWS] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      }
      mine[VDIM / 4 * ROWS] = make_float4(ok ? m : -INFINITY, l, 0.f, 0.f);
      __threadfence();
      const int id = MAPS == 1 ? q : 0, threads = MAPS == 1 ? 128 : 256;
      named_barrier(1 + id, threads);                  // the warpgroup's (both warpgroups') rows are written
      const bool first_thread = MAPS == 1 ? (tid & 127) == 0 : tid == 128;
      int* counter = tc.counters + piece_index * 2 + id;
      if (first_thread) seen[id] = atomicAdd(counter, 1);
      named_barrier(1 + id, threads);
      finishes = finishes && seen[id] == shares - 1;
      if (finishes) {
        __threadfence();
        if (first_thread) *counter = 0;                // ready for the next launch
      }
    } else if (MAPS == 2 && shares == 1) {
      if (q == 1) sums1[row] = make_float2(m, l);
      tc_fence_before();
      named_barrier(1, 256);                           // both maps' O are complete, map 1's sums are in shared memory
      tc_fence_after();
    }
    if (ok && finishes) {
      // the denominators, and what every share's O is multiplied by on its way into the sum
      float weight[MAPS][MAX_SHARES], inv[MAPS];
      const float sink_log2 = p.sink != nullptr ? p.sink[row_valid ? head : 0] * 1.4426950408889634f : -INFINITY;
#pragma unroll
      for (int map = 0; map < MAPS; map++) {
        float sm[MAX_SHARES], sl[MAX_SHARES], top = sink_log2;
#pragma unroll
        for (int s = 0; s < MAX_SHARES; s++) {
          sm[s] = -INFINITY; sl[s] = 0.f;
          if (shares > 1 && s < shares) {
            const float4 ml = __ldcg(share_at(s, MAPS == 1 ? q : map) + VDIM / 4 * ROWS);
            sm[s] = ml.x; sl[s] = ml.y;
          } else if (s == 0) {
            sm[0] = MAPS == 2 && map == 1 ? sums1[row].x : m;
            sl[0] = MAPS == 2 && map == 1 ? sums1[row].y : l;
          }
        }
        if (shares == 1 && p.sink == nullptr) {
          weight[map][0] = 1.0f;
          inv[map] = 1.0f / sl[0];
          continue;
        }
#pragma unroll
        for (int s = 0; s < MAX_SHARES; s++) {
          sm[s] = sm[s] == -INFINITY ? -INFINITY : sm[s] * scale_log2;
          top = fmaxf(top, sm[s]);
        }
        float sum = sink_log2 == -INFINITY ? 0.f : exp2_fast(sink_log2 - top);
#pragma unroll
        for (int s = 0; s < MAX_SHARES; s++) {
          weight[map][s] = sm[s] == -INFINITY ? 0.f : exp2_fast(sm[s] - top);
          sum = fmaf(sl[s], weight[map][s], sum);
        }
        inv[map] = 1.0f / sum;
      }
      float o[VDIM], squares = 0.f;
#pragma unroll
      for (int c = 0; c < VDIM / 32; c++) {
        float v[32];
#pragma unroll
        for (int map = 0; map < MAPS; map++) {
          const int tile = MAPS == 1 ? q : map;
          const uint32_t addr = lane_addr + L::O_COLUMN + tile * VDIM;
          if (shares == 1) {
            own_columns(addr, my_tiles > 0, c, weight[map][0], v);
          } else {
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] = 0.f;
#pragma unroll
            for (int s = 0; s < MAX_SHARES; s++) {
              if (s >= shares) break;
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const float4 t = __ldcg(share_at(s, tile) + (c * 8 + i) * ROWS);
                v[4 * i] = fmaf(t.x, weight[map][s], v[4 * i]);
                v[4 * i + 1] = fmaf(t.y, weight[map][s], v[4 * i + 1]);
                v[4 * i + 2] = fmaf(t.z, weight[map][s], v[4 * i + 2]);
                v[4 * i + 3] = fmaf(t.w, weight[map][s], v[4 * i + 3]);
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; i++) {
            if (map == 0) o[c * 32 + i] = v[i] * inv[0];
            else o[c * 32 + i] -= p.lambda * (v[i] * inv[map]);
          }
        }
#pragma unroll
        for (int i = 0; i < 32; i++) squares = fmaf(o[c * 32 + i], o[c * 32 + i], squares);
      }
      float factor = p.out_scale;
      if (p.norm_eps > 0.f) factor *= 1.0f / sqrtf(squares / (float)VDIM + p.norm_eps);
      if (MAPS == 1 && p.turn.cos != nullptr) {
        // back by the query's position
        const size_t at = (size_t)min(max(limit, 0), p.turn.positions - 1) * (VDIM / 2);
#pragma unroll
        for (int i = 0; i < VDIM / 2; i++) {
          const float cs = p.turn.cos[at + i], sn = p.turn.sin[at + i];
          if (p.turn.interleaved) {
            const float a = o[2 * i], b = o[2 * i + 1];
            o[2 * i] = a * cs + b * sn;
            o[2 * i + 1] = b * cs - a * sn;
          } else {
            const float a = o[i], b = o[i + VDIM / 2];
            o[i] = a * cs + b * sn;
            o[i + VDIM / 2] = b * cs - a * sn;
          }
        }
      }
      if (row_valid) {
        const bool per_element = MAPS == 1 && p.gate != nullptr && p.gate_elements;
        if (p.gate != nullptr && !per_element) factor *= 1.0f / (1.0f + expf(-__bfloat162float(p.gate[(size_t)token * p.gate_stride + head])));
        __nv_bfloat16* dst = p.out + (size_t)token * p.out_stride + (size_t)head * VDIM;
#pragma unroll
        for (int i = 0; i < VDIM; i += 8) {
          uint32_t packed[4];
#pragma unroll
          for (int k = 0; k < 4; k++) {
            float a = o[i + 2 * k] * factor, b = o[i + 2 * k + 1] * factor;
            if (per_element) {
              a *= element_gate(p, token, head, VDIM, i + 2 * k);
              b *= element_gate(p, token, head, VDIM, i + 2 * k + 1);
            }
            __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
            packed[k] = *(uint32_t*)&h;
          }
          *(uint4*)(dst + i) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag && (warp == 0 || warp == 2) && lane == 0) {
    // copies already issued still write shared memory: wait for them (bounded) before leaving
    uint64_t* full = warp == 0 ? k_full : v_full;
    for (int j = max(0, issued - NS); j < issued; j++) mbar_wait(&full[j % NS], (j / NS) & 1);
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

bool tc_sizes(int maps, int dim, int vdim) {
  return (dim == 64 && (vdim == 64 || vdim == 128) && (maps == 1 || maps == 2)) || (dim == 128 && vdim == 128 && maps == 1);
}
int cta_rows(int maps) { return maps == 1 ? 2 * ROWS : ROWS; }
long long pieces_bound(int tokens, int requests, int heads, int kv_heads, int maps) {
  return ((long long)tokens * (heads / kv_heads) + (long long)requests * (cta_rows(maps) - 1)) / cta_rows(maps) * kv_heads;
}

template <int DIM, int VDIM, int MAPS, bool PACKED = false>
int launch(const CUtensorMap& map_k, const CUtensorMap& map_v, const Params& p, int ctas, cudaStream_t stream) {
  using L = Layout<DIM, VDIM, MAPS>;
  static bool configured = false;
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(maps_attention_tc_kernel<DIM, VDIM, MAPS, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (err != cudaSuccess) return sprout_fail("maps_attention (tcgen05): cannot reserve %d bytes of shared memory: %s", L::SMEM, cudaGetErrorString(err));
    configured = true;
  }
  sprout_launch(maps_attention_tc_kernel<DIM, VDIM, MAPS, PACKED>, dim3(ctas), dim3(THREADS), L::SMEM, stream, map_k, map_v, p);
  return sprout_check_launch("maps_attention (tcgen05)");
}

}  // namespace

// Whether the kernel takes these sizes; the output's rows start on 16-byte boundaries.
SPROUT_API int sprout_maps_attention_tc_supported(int maps, int dim, int vdim, int page_tokens, int out_stride) {
  const bool pages_ok = page_tokens == 8 || page_tokens == 16 || page_tokens == 32 || page_tokens == 64 || (page_tokens > 0 && page_tokens % 128 == 0);
  return tc_sizes(maps, dim, vdim) && pages_ok && out_stride % 8 == 0;
}

// How many CTAs a piece's key tiles are divided among at most in a launch of these sizes (the kernel knows the pieces exactly), and the
// floats of scratch that takes (none for one share).  A launch that divides has at most as many pieces as there are SMs, and two
// counters a piece.
SPROUT_API int sprout_maps_attention_tc_shares(int tokens, int requests, int heads, int kv_heads, int maps) {
  const long long pieces = pieces_bound(tokens, requests, heads, kv_heads, maps);
  const long long want = 2LL * sm_count() / (pieces > 0 ? pieces : 1);
  return (int)(want < 1 ? 1 : want > MAX_SHARES ? MAX_SHARES : want);
}
SPROUT_API long long sprout_maps_attention_tc_scratch_floats(int tokens, int requests, int heads, int kv_heads, int maps, int vdim) {
  const int shares = sprout_maps_attention_tc_shares(tokens, requests, heads, kv_heads, maps);
  return shares == 1 ? 0 : pieces_bound(tokens, requests, heads, kv_heads, maps) * shares * 2 * ROWS * (vdim + 4);
}

// The arguments of sprout_multimap_attention_mma, checked there.  `scratch` holds what the function above says, `counters` (zeroed) two
// numbers an SM, or they are null: then no piece is divided.
int sprout_maps_attention_tc(const MultiMapParams& m, int tokens, int maps, int dim, int vdim, float* scratch, int* counters, cudaStream_t stream) {
  SPROUT_REQUIRE(sprout_maps_attention_tc_supported(maps, dim, vdim, m.page_tokens, m.out_stride) && ((uintptr_t)m.out & 15) == 0,
                 "maps_attention (tcgen05): %d maps of %d with values of %d, page size %d or the output's alignment is not taken", maps, dim, vdim, m.page_tokens);
  const long long cache_rows = (long long)m.num_pages * m.kv_heads * m.page_tokens;
  SPROUT_REQUIRE(cache_rows <= 0x7fffffffLL, "maps_attention (tcgen05): the cache has too many rows for a tensor map coordinate");
  Params p{};
  p.m = m;
  p.box_rows = m.page_tokens < KEYS ? m.page_tokens : KEYS;
  p.shares = scratch && counters ? sprout_maps_attention_tc_shares(tokens, m.requests, m.heads, m.kv_heads, maps) : 1;
  p.scratch = scratch; p.counters = counters; p.sms = sm_count();
  CUtensorMap map_k, map_v;
  if (tensor_map(m.k_cache, (int)cache_rows, maps * dim, maps * dim, p.box_rows, &map_k)) return 1;
  if (tensor_map(m.v_cache, (int)cache_rows, vdim, vdim, p.box_rows, &map_v)) return 1;
  const long long ctas = pieces_bound(tokens, m.requests, m.heads, m.kv_heads, maps) * p.shares;
  SPROUT_REQUIRE(ctas <= 0x7fffffffLL, "maps_attention (tcgen05): too many tokens");
  if (maps == 2) return vdim == 64 ? launch<64, 64, 2>(map_k, map_v, p, (int)ctas, stream) : launch<64, 128, 2>(map_k, map_v, p, (int)ctas, stream);
  if (dim == 64) return vdim == 64 ? launch<64, 64, 1>(map_k, map_v, p, (int)ctas, stream) : launch<64, 128, 1>(map_k, map_v, p, (int)ctas, stream);
  return launch<128, 128, 1>(map_k, map_v, p, (int)ctas, stream);
}

// Attention of queries [tokens, heads * (dim + tail)] over packed rows: `unfolded` bfloat16 [rows, heads * dim + heads * vdim] (every
// head's own key part, then every head's values) and `latent` [rows, latent_width], whose columns from tail_col on are the key part that
// the heads share.  Rows of a request lie in the order of its positions from packed_base on, the requests' one behind the other.
SPROUT_API int sprout_latent_unfolded_attention(const void* q, int q_stride, const void* unfolded, const void* latent, int rows, int latent_width,
                                                int tail_col, const int* q_start, const int* positions, const float* sink, void* out, int out_stride,
                                                int tokens, int requests, int heads, int dim, int tail, int vdim, float scale, int window,
                                                float* scratch, int* counters, int* status, cudaStream_t stream) {
  SPROUT_REQUIRE(q && unfolded && latent && q_start && positions && out && status, "latent_unfolded_attention: null pointer");
  SPROUT_REQUIRE(rows > 0 && tokens > 0 && requests > 0 && heads > 0 && dim > 0 && tail >= 0 && dim % 64 == 0 && tail % 64 == 0 && tc_sizes(1, dim + tail, vdim),
                 "latent_unfolded_attention: bad sizes (keys of %d + %d, values of %d)", dim, tail, vdim);
  SPROUT_REQUIRE(q_stride % 8 == 0 && out_stride % 8 == 0 && latent_width % 8 == 0 && tail_col % 8 == 0 && tail_col + tail <= latent_width &&
                 (((uintptr_t)q | (uintptr_t)unfolded | (uintptr_t)latent | (uintptr_t)out) & 15) == 0, "latent_unfolded_attention: rows must start on 16-byte boundaries");
  Params p{};
  p.m.q = (const __nv_bfloat16*)q; p.m.q_stride = q_stride; p.m.q_start = q_start; p.m.positions = positions;
  p.m.block_table = q_start; p.m.page_tokens = KEYS; p.m.num_pages = 1;                     // not read
  p.m.out = (__nv_bfloat16*)out; p.m.out_stride = out_stride; p.m.requests = requests; p.m.heads = p.m.kv_heads = heads;
  p.m.scale = scale; p.m.out_scale = 1.0f; p.m.status = status; p.m.ksplit = 1; p.m.sink = sink;
  p.m.mask_kind = window > 0 ? MASK_WINDOW : MASK_CAUSAL; p.m.mask_size = window;
  p.box_rows = KEYS;
  p.shares = scratch && counters ? sprout_maps_attention_tc_shares(tokens, requests, heads, heads, 1) : 1;
  p.scratch = scratch; p.counters = counters; p.sms = sm_count();
  p.key_atoms = dim / 64; p.tail_col = tail_col; p.value_col = heads * dim;
  const int width = heads * (dim + vdim);
  CUtensorMap map_k, map_v;
  if (tensor_map(unfolded, rows, width, width, KEYS, &map_k)) return 1;
  if (tensor_map(latent, rows, latent_width, latent_width, KEYS, &map_v)) return 1;
  const long long ctas = pieces_bound(tokens, requests, heads, heads, 1) * p.shares;
  SPROUT_REQUIRE(ctas <= 0x7fffffffLL, "latent_unfolded_attention: too many tokens");
  if (dim + tail == 64) return vdim == 64 ? launch<64, 64, 1, true>(map_k, map_v, p, (int)ctas, stream) : launch<64, 128, 1, true>(map_k, map_v, p, (int)ctas, stream);
  return launch<128, 128, 1, true>(map_k, map_v, p, (int)ctas, stream);
}

// The arguments of sprout_attention_prefill, checked there; scratch and counters may be null.
int sprout_attention_prefill_maps(const void* q, int q_stride, const void* k_cache, const void* v_cache, const int* block_table, int table_stride,
                                  const int* q_start, const int* positions, void* out, int out_stride, int num_tokens, int requests, int heads,
                                  int kv_heads, int head_dim, int page_tokens, int num_pages, float* scratch, long long scratch_floats, int* counters,
                                  int* status, cudaStream_t stream) {
  MultiMapParams m{};
  m.q = (const __nv_bfloat16*)q; m.q_stride = q_stride; m.k_cache = (const __nv_bfloat16*)k_cache; m.v_cache = (const __nv_bfloat16*)v_cache;
  m.block_table = block_table; m.table_stride = table_stride; m.q_start = q_start; m.positions = positions;
  m.out = (__nv_bfloat16*)out; m.out_stride = out_stride; m.requests = requests; m.heads = heads; m.kv_heads = kv_heads;
  m.page_tokens = page_tokens; m.num_pages = num_pages; m.scale = 1.0f / sqrtf((float)head_dim); m.out_scale = 1.0f; m.status = status; m.ksplit = 1;
  const bool fits = scratch && counters && sprout_maps_attention_tc_scratch_floats(num_tokens, requests, heads, kv_heads, 1, head_dim) <= scratch_floats;
  return sprout_maps_attention_tc(m, num_tokens, 1, head_dim, head_dim, fits ? scratch : nullptr, fits ? counters : nullptr, stream);
}
