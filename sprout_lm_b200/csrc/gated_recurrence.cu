// Recurrent mixers whose decay comes from the input, and the row kernels around them.  All arithmetic is float32;
// the element type of the projections (float or bfloat16) is a template parameter.
//
//  * gated_scan:   per request and head, token by token:
//                      S_t = diag(a_t) S_(t-1) + (c_t k_t) v_t^T,   o_t = S_t^T (q_scale q_t) + skip_h v_t
//                  with S [dim, vdim] float32 in the request's state slot.  Two ways to make a_t and c_t:
//                    per key channel (gated linear attention): a_t[i] = sigmoid(z_t[i] + bias[i])^(1/tau), c_t = 1;
//                    per head (a selective state space):      dt = softplus(z_t[h] + bias[h]), a_t[i] = exp(-exp(a_log[h]) dt),
//                                                             c_t = dt;
//                    a floor (a forget gate that also decides what is written): w_t[i] = (1 - floor[i]) sigmoid(-(z_t[i] + bias[i])),
//                                                             a_t[i] = 1 - w_t[i]; w_t takes the place of c_t k_t;
//                    a bonus (the RWKV recurrence): a_t[i] = exp(-exp(z_t[i] + bias[i])), c_t = 1, and the output reads the state before
//                                                             the token plus the token's own write weighed by a bonus u[i] per channel:
//                                                             o_t = (S_(t-1) + diag(u) k_t v_t^T)^T (q_scale q_t);
//                    given (a matrix memory with exponential gates): a_t and c_t per head come ready-made from the
//                                                             caller (`da`, `dc`), whatever the portion's length.
//                  With `ones_col` the value row gets one more column that is always 1 (column `v_cols` of the state
//                  and of the output): the state's extra column is then sum of the decayed c_t k_t, a normaliser.
//                  q and k may be shared by the heads of a group (`groups` <= heads).  One block per (request, head,
//                  block of value columns) with its part of the state in registers; the tokens' vectors come through
//                  shared memory a few tokens at a time.  The order of operations per element is the tokens' order:
//                  the result does not depend on the cutting or on the batch.
//  * causal_conv:  y_t[c] = act(bias[c] + sum_j w[c][j] x_(t - (taps - 1 - j))[c]), zeros before the start of the
//                  sequence; the last taps - 1 inputs of a request live in its state slot [taps - 1, channels] and are
//                  read at the start of a portion and replaced at its end.
//  * token_blend:  row t of part s = h_t + (h_(t-1) - h_t) * mu_s, several blends of every row with the row before it; the row
//                  before a portion's first lives in the request's state slot (zeros at the start of the sequence).
//  * gated_group_norm: rows in `groups` equal parts, each divided by its own root mean square, times a weight that
//                  repeats every `period` elements, times act(gate) before or after the norm (or without a gate).
//  * scaled_sum:   x += a y_1 + b y_2.
#include "gated_scan.cuh"

using namespace sprout_scan;

namespace {

__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float silu_g(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float sigmoid_g(float z) { return 1.0f / (1.0f + expf(-z)); }

// Forms of the scan's kernel (the others share FORM_PLAIN), so that each keeps its own registers.
enum ScanForm : int { FORM_PLAIN = 0, FORM_FLOOR = 1, FORM_BONUS = 2 };

__device__ __forceinline__ float double_exp_decay(float z) { return expf(-expf(z)); }

// What a forget gate with a floor writes: 1 - f for f = floor + (1 - floor) sigmoid(z).
__device__ __forceinline__ float write_share(float z, float floor) { return (1.0f - floor) * sigmoid_g(-z); }

// Eight neighbouring elements of a row that start on a 16-byte boundary.
__device__ __forceinline__ void fetch8(const float* p, float (&v)[8]) {
  const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void fetch8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *(const uint4*)p;
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// Two float32 in a register pair: sm_100a multiplies, adds and fuses them pairwise in one instruction.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

constexpr int SCAN_THREADS = 128, SCAN_MAX_TOKENS = 8;

// A block of SCAN_THREADS threads owns (request, head, `cb` value columns).  A thread keeps a tile of ROWS x COLS
// elements of the state in registers from the first token to the last: the state's rows are dealt to `slices` lanes
// of a warp (a power of two; the thread of slice s has rows s, s + slices, s + 2 slices, ...), the columns in groups of
// COLS to the threads of equal slice, so every (q, k, a) triple read from shared memory serves COLS columns.
// Tokens come `batch` at a time: while the threads walk a batch's tokens over their registers, the next batch's q, k,
// decay inputs and values are on their way from memory into registers; at the batch's end they are turned into
// float32 vectors in shared memory ([q_scale q | c k | a] per row).  The slices of a column add their parts of o with
// shuffles.  The bfloat16 path's walks over chunks of key sizes 64, 128 and 256, whose rows fill the slices (PAIRS), go two rows at a
// time in packed arithmetic: a thread's rows are then neighbours, fetched 16 bytes at a time, and q, c k and a lie in planes of their
// own, so that a 16-byte read is two pairs of one of them (2,048 tokens of 16 heads of 128 x 128, with the decays and the carry: 443 us
// with a number at a time, (q, c k, a) triples and 2-byte fetches, 296 us so).  Decays per channel or per head at key sizes 64 and 128 run in
// gated_scan_mma.cu where their rows allow it, in the same three launches around the same carry.  Other sizes and rows off 16-byte boundaries keep a
// number at a time: pairs without the wide fetches cost 12 % (four heads of 96 x 96), and with two slices or one, 4 % (8 x 512, 16 x 64).
// Each element of S sees S <- fma(a, S, (c k) v) once per token in the tokens' order.  An output's sum over the rows has one order in
// the 32-bit path, whatever the cutting and the batch; with PAIRS it is added in pairs, without in turn.  A bfloat16 request's last bits
// depend on the whole step: whether its portions are walked whole or in chunks and, in gated_scan_mma.cu, on the chunks' length, which
// follows from the step's tokens, number of portions and longest portion and from the SMs (a replayed step keeps that of the step it was
// recorded for).
//
// Long portions are cut into chunks of `p.chunk` tokens so that more blocks than (request, head, columns) have work, in
// three launches: SCAN_CHUNK_SUMS walks every chunk but a request's last from a zero state and leaves the chunk's own
// sums and the product of its decays; scan_carry_kernel turns them, in the chunks' order, into the state before each
// chunk; SCAN_CHUNK_OUT walks every chunk from that state, writes the outputs, and the last chunk writes the
// request's state.  The decays of these two walks are made beforehand by scan_decay_kernel (each is needed by all
// blocks of columns and in both walks).  Against the single walk only the association of the decays' products
// differs: (a_n ... a_1) S + sums instead of a_n (... (a_1 S)).
// FORM: FORM_FLOOR is the forget gate with a floor (DECAY_FLOOR), FORM_BONUS the output that reads the state before the token
// (DECAY_BONUS): the fourth number of a row's vector is then q_scale q u k, whose sum over the rows weighs the token's value.
template <typename T, int ROWS, int COLS, int PHASE, int FORM, bool PAIRS>
__global__ void __launch_bounds__(SCAN_THREADS, ROWS == 8 ? 4 : 2)
gated_scan_kernel(const ScanParams<T> p, int slices_log2, int batch) {
  constexpr int ROWS_LOG2 = ROWS == 8 ? 3 : 5;
  static_assert(ROWS == 8 || ROWS == 32, "rows of a thread's tile");
  constexpr int EPT = ROWS == 8 ? 8 : 16;            // row vectors a thread fetches per batch: batch * slices * ROWS / threads
  constexpr int VPT = SCAN_MAX_TOKENS;               // values a thread fetches per batch: batch * cb / threads
  extern __shared__ float4 scan_smem[];
  const int slices = 1 << slices_log2, dim = p.dim;
  const int rows_log2 = slices_log2 + ROWS_LOG2, rows_pad = 1 << rows_log2;
  const int cb_log2 = 7 - slices_log2 + (COLS == 4 ? 2 : 0), cb = 1 << cb_log2;
  static_assert(COLS == 1 || COLS == 4, "columns of a thread's tile");
  static_assert(!PAIRS || (ROWS == 8 && COLS == 4 && PHASE != SCAN_WHOLE), "pairs of rows in tiles of 8 x 4, over ready-made decays");
  float4* tok = scan_smem;                                             // [batch][rows_pad]: (q, k, a, -)
  // PAIRS: [batch][4 planes: q, k, a, -][2 halves of every 8 rows][slices][4], a half padded so that the two halves' banks differ
  const int half_stride = rows_pad / 2 + 16, plane = 2 * half_stride;
  float* tok2 = reinterpret_cast<float*>(scan_smem);
  float* vt = PAIRS ? tok2 + (size_t)batch * 4 * plane : reinterpret_cast<float*>(tok + (size_t)batch * rows_pad);  // [batch][cb]
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, tid = threadIdx.x;
  int r = blockIdx.x, chunk_at = 0, chunk_count = 1;
  if (PHASE != SCAN_WHOLE && p.sums != nullptr) {      // without scratch every request is one chunk: block x walks request x
    if (!find_chunk(p.q_start, p.requests, p.chunk, blockIdx.x, r, chunk_at, chunk_count)) return;
    if (PHASE == SCAN_CHUNK_SUMS && chunk_at == chunk_count - 1) return;      // nothing comes after it
  }
  const bool last_chunk = chunk_at == chunk_count - 1;
  const int slice = tid & (slices - 1), col_local = (tid >> slices_log2) * COLS;
  const int col = blockIdx.z * cb + col_local;                          // the first of the thread's columns
  const int slot = p.state_slots[r];
  if (slot < 0 || slot >= p.num_slots) {
    if (tid == 0) atomicOr(p.status, SPROUT_STATUS_BAD_PAGE);
    return;
  }
  const int g = h / (p.heads / p.groups);
  constexpr bool floored = FORM == FORM_FLOOR, bonus = FORM == FORM_BONUS;                     // a decay per channel, and no keys
  const bool per_head = FORM == FORM_PLAIN && p.mode != DECAY_PER_CHANNEL;
  float* mine = p.state + (((size_t)slot * p.heads + h) * dim) * p.vdim;
  // the chunk's place in the scratch: the blocks before it belong to the requests before r and to r's earlier chunks
  float* held = PHASE == SCAN_WHOLE ? nullptr : p.sums + (((size_t)(blockIdx.x) * p.heads + h) * dim) * p.vdim;
  const float* from = (PHASE == SCAN_WHOLE || chunk_count == 1) ? mine : held;
  const bool vectors = (p.vdim & 3) == 0;             // rows of the state start on 16-byte boundaries
  float S[ROWS][COLS], P[PHASE == SCAN_CHUNK_SUMS ? ROWS : 1];
  auto row_of = [&](int j) { return PAIRS ? slice * ROWS + j : j * slices + slice; };
#pragma unroll
  for (int j = 0; j < ROWS; j++) {
    const int row = row_of(j);
    if (COLS == 4 && vectors) {                       // four columns of a row in one access
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (PHASE != SCAN_CHUNK_SUMS && col < p.vdim && row < dim) x = *reinterpret_cast<const float4*>(from + (size_t)row * p.vdim + col);
      S[j][0] = x.x; S[j][1 % COLS] = x.y; S[j][2 % COLS] = x.z; S[j][3 % COLS] = x.w;
    } else {
#pragma unroll
      for (int c = 0; c < COLS; c++)
        S[j][c] = (PHASE != SCAN_CHUNK_SUMS && col + c < p.vdim && row < dim) ? from[(size_t)row * p.vdim + col + c] : 0.f;
    }
    if (PHASE == SCAN_CHUNK_SUMS) P[j] = 1.f;
  }
  unsigned long long S2[PAIRS ? ROWS / 2 : 1][COLS], P2[PAIRS ? ROWS / 2 : 1];      // PAIRS: rows 2 j and 2 j + 1
  if (PAIRS) {
#pragma unroll
    for (int j = 0; j < ROWS / 2; j++) {
      P2[j] = pack2(1.f, 1.f);
#pragma unroll
      for (int c = 0; c < COLS; c++) S2[j][c] = pack2(S[2 * j][c], S[2 * j + 1][c]);
    }
  }
  const float skip = p.skip ? p.skip[h] : 0.f;
  const float rate = p.mode == DECAY_PER_HEAD ? expf(p.a_log[h]) : 0.f;
  const int first = p.q_start[r] + chunk_at * (PHASE == SCAN_WHOLE ? 0 : p.chunk);
  const int last = PHASE == SCAN_WHOLE ? p.q_start[r + 1] : min(p.q_start[r + 1], first + p.chunk);
  auto z_at = [&](size_t index) { return p.z_f32 ? ((const float*)p.z)[index] : to_float(((const T*)p.z)[index]); };

  float rq[EPT], rk[EPT], rz[EPT], rc[PHASE == SCAN_WHOLE ? 1 : EPT], rv[VPT];
  // PAIRS: a thread's eight elements are the rows 8 (tid % slices) on of token tid / slices of the batch, its values neighbours too
  // (32 slices: a batch of 4 tokens over 16 columns has a value for every second thread only)
  const int wide_token = tid >> slices_log2, wide_values = max(1, (batch << cb_log2) / SCAN_THREADS);
  auto fetch = [&](int t0) {                          // loads only: nothing waits for them here
    const int n = min(batch, last - t0);
    if (PAIRS) {
      if (wide_token < n) {
        const size_t t = (size_t)t0 + wide_token;
        const int i = slice * 8;
        float x[8];
        if (PHASE != SCAN_CHUNK_SUMS) {
          fetch8(p.q + t * p.q_stride + (size_t)g * dim + i, x);
#pragma unroll
          for (int u = 0; u < 8; u++) rq[u % EPT] = x[u];
        }
        if (!floored) {
          fetch8(p.k + t * p.k_stride + (size_t)g * dim + i, x);
#pragma unroll
          for (int u = 0; u < 8; u++) rk[u % EPT] = x[u];
        }
        if (per_head) {
          const float a = p.da[t * p.heads + h];
#pragma unroll
          for (int u = 0; u < 8; u++) rz[u % EPT] = a;
          rc[0] = p.dc[t * p.heads + h];
        } else {
          fetch8(p.da + (t * p.heads + h) * dim + i, x);
#pragma unroll
          for (int u = 0; u < 8; u++) rz[u % EPT] = x[u];
          rc[0] = 1.f;
        }
      }
#pragma unroll
      for (int u = 0; u < VPT; u++) {
        if (u >= wide_values) break;
        const int e = tid * wide_values + u, tt = e >> cb_log2, column = blockIdx.z * cb + (e & (cb - 1));
        rv[u] = (tt < n && column < p.v_cols) ? to_float(p.v[(size_t)(t0 + tt) * p.v_stride + (size_t)h * p.v_cols + column])
                                              : (p.ones_col && tt < n && column == p.v_cols) ? 1.f : 0.f;
      }
      return;
    }
    // the batch's first rows once in 64-bit; within the batch 32-bit offsets do (at most SCAN_MAX_TOKENS rows further)
    const size_t tb = (size_t)t0;
    const T* qrow = p.q + tb * p.q_stride + (size_t)g * dim;
    const T* krow = p.k + tb * p.k_stride + (size_t)g * dim;
    const T* vrow = p.v + tb * p.v_stride + (size_t)h * p.v_cols;
    const float* arow = PHASE == SCAN_WHOLE ? nullptr : p.da + (per_head ? tb * p.heads + h : (tb * p.heads + h) * dim);
    const float* crow = (PHASE == SCAN_WHOLE || !per_head) ? nullptr : p.dc + tb * p.heads + h;
#pragma unroll
    for (int u = 0; u < EPT; u++) {
      const int e = tid + u * SCAN_THREADS, tt = e >> rows_log2, i = e & (rows_pad - 1);
      rq[u] = rk[u] = rz[u] = 0.f;
      if (PHASE != SCAN_WHOLE) rc[u] = 0.f;
      if (tt < n && i < dim) {
        if (PHASE != SCAN_CHUNK_SUMS) rq[u] = to_float(qrow[tt * p.q_stride + i]);
        rk[u] = floored ? 0.f : to_float(krow[tt * p.k_stride + i]);
        if (PHASE == SCAN_WHOLE) {
          const size_t t = tb + tt;
          rz[u] = per_head ? z_at(t * p.z_stride + h) : z_at(t * p.z_stride + (size_t)h * dim + i);
        } else {
          rz[u] = per_head ? arow[tt * p.heads] : arow[tt * p.heads * dim + i];
          rc[u] = per_head ? crow[tt * p.heads] : 1.f;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < VPT; u++) {
      const int e = tid + u * SCAN_THREADS, tt = e >> cb_log2, column = blockIdx.z * cb + (e & (cb - 1));
      rv[u] = (tt < n && column < p.v_cols) ? to_float(vrow[tt * p.v_stride + column]) : (p.ones_col && tt < n && column == p.v_cols) ? 1.f : 0.f;
    }
  };
  if (first < last) fetch(first);
  for (int t0 = first; t0 < last; t0 += batch) {
    const int n = min(batch, last - t0);
    __syncthreads();                                   // the batch before has been read by everyone
    if (PAIRS) {
      if (wide_token < n) {
        float4* to = reinterpret_cast<float4*>(tok2 + (size_t)wide_token * 4 * plane + slice * 4);
        const int half4 = half_stride / 4, plane4 = plane / 4;
        float x[4][8];                                 // q, k, a, -
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const float decay = rz[u % EPT];
          x[0][u] = PHASE == SCAN_CHUNK_SUMS ? 0.f : (floored && p.q_silu ? silu_g(rq[u % EPT]) : rq[u % EPT]) * p.q_scale;
          x[1][u] = floored ? decay : rk[u % EPT] * rc[0];
          x[2][u] = floored ? 1.0f - decay : decay;
          if (bonus && PHASE != SCAN_CHUNK_SUMS) x[3][u] = x[0][u] * p.bonus[(size_t)h * dim + slice * 8 + u] * x[1][u];
        }
#pragma unroll
        for (int which = 0; which < 4; which++) {
          if ((which == 0 && PHASE == SCAN_CHUNK_SUMS) || (which == 3 && (!bonus || PHASE == SCAN_CHUNK_SUMS))) continue;
          to[which * plane4] = make_float4(x[which][0], x[which][1], x[which][2], x[which][3]);
          to[which * plane4 + half4] = make_float4(x[which][4], x[which][5], x[which][6], x[which][7]);
        }
      }
#pragma unroll
      for (int u = 0; u < VPT; u++) {
        if (u >= wide_values) break;
        if (tid * wide_values + u < (batch << cb_log2)) vt[tid * wide_values + u] = rv[u];
      }
    } else {
#pragma unroll
    for (int u = 0; u < EPT; u++) {
      const int e = tid + u * SCAN_THREADS, tt = e >> rows_log2, i = e & (rows_pad - 1);
      if (tt >= n) break;
      float4 x = make_float4(0.f, 0.f, 1.f, 0.f);      // rows beyond dim stay zero
      if (i < dim) {
        float step = 1.0f, decay;
        if (PHASE != SCAN_WHOLE) {
          step = rc[u];
          decay = rz[u];
        } else if (per_head) {
          step = softplus_f(rz[u] + p.bias[h]);
          decay = expf(-rate * step);
        } else if (floored) {
          decay = write_share(rz[u] + p.bias[(size_t)h * dim + i], p.a_log[(size_t)h * dim + i]);
        } else if (bonus) {
          decay = double_exp_decay(rz[u] + p.bias[(size_t)h * dim + i]);
        } else {
          decay = expf(-softplus_f(-(rz[u] + p.bias[(size_t)h * dim + i])) * p.inv_tau);  // sigmoid(z)^(1/tau) through its logarithm
        }
        x.x = (floored && p.q_silu ? silu_g(rq[u]) : rq[u]) * p.q_scale;
        x.y = floored ? decay : rk[u] * step;
        x.z = floored ? 1.0f - decay : decay;
        if (bonus && PHASE != SCAN_CHUNK_SUMS) x.w = x.x * p.bonus[(size_t)h * dim + i] * x.y;
      }
      tok[e] = x;
    }
#pragma unroll
    for (int u = 0; u < VPT; u++) {
      const int e = tid + u * SCAN_THREADS;
      if (e < (n << cb_log2)) vt[e] = rv[u];
    }
    }
    __syncthreads();
    if (t0 + batch < last) fetch(t0 + batch);          // in flight while this batch is applied
    float* out_rows = p.out + (size_t)t0 * p.heads * p.vdim + (size_t)h * p.vdim + col;
    for (int tt = 0; tt < n; tt++) {
      float v[COLS], o[COLS];
      if (COLS == 4) {
        const float4 v4 = *reinterpret_cast<const float4*>(vt + (tt << cb_log2) + col_local);
        v[0] = v4.x; v[1 % COLS] = v4.y; v[2 % COLS] = v4.z; v[3 % COLS] = v4.w;
      } else {
#pragma unroll
        for (int c = 0; c < COLS; c++) v[c] = vt[(tt << cb_log2) + col_local + c];
      }
#pragma unroll
      for (int c = 0; c < COLS; c++) o[c] = 0.f;
      const float4* cur = tok + ((size_t)tt << rows_log2) + slice;
      float own = 0.f;                                 // the weight of the token's own value
      if (PAIRS) {
        const float* at = tok2 + (size_t)tt * 4 * plane + slice * 4;
        unsigned long long q2[4], k2[4], a2[4], v2[COLS], o2[COLS];
        auto four = [&](int which, unsigned long long (&to)[4]) {
          const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(at + which * plane), hi = *reinterpret_cast<const ulonglong2*>(at + which * plane + half_stride);
          to[0] = lo.x; to[1] = lo.y; to[2] = hi.x; to[3] = hi.y;
        };
        four(1, k2);
        four(2, a2);
        if (PHASE != SCAN_CHUNK_SUMS) four(0, q2);
#pragma unroll
        for (int c = 0; c < COLS; c++) { v2[c] = pack2(v[c], v[c]); o2[c] = 0ull; }
#pragma unroll
        for (int j = 0; j < 4; j++) {
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            const unsigned long long s = fma2(a2[j], S2[PAIRS ? j : 0][c], mul2(k2[j], v2[c]));
            if (PHASE != SCAN_CHUNK_SUMS) o2[c] = fma2(bonus ? S2[PAIRS ? j : 0][c] : s, q2[j], o2[c]);
            S2[PAIRS ? j : 0][c] = s;
          }
          if (PHASE == SCAN_CHUNK_SUMS) P2[PAIRS ? j : 0] = mul2(P2[PAIRS ? j : 0], a2[j]);
        }
        if (PHASE != SCAN_CHUNK_SUMS) {
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            float lo, hi;
            unpack2(o2[c], lo, hi);
            o[c] = lo + hi;
          }
          if (bonus) {
            const float4 w0 = *reinterpret_cast<const float4*>(at + 3 * plane), w1 = *reinterpret_cast<const float4*>(at + 3 * plane + half_stride);
            own = ((w0.x + w0.y) + (w0.z + w0.w)) + ((w1.x + w1.y) + (w1.z + w1.w));
          }
        }
      } else
#pragma unroll
      for (int j = 0; j < ROWS; j++) {
        const float4 x = cur[j << slices_log2];
#pragma unroll
        for (int c = 0; c < COLS; c++) {
          const float s = fmaf(x.z, S[j][c], x.y * v[c]);
          if (PHASE != SCAN_CHUNK_SUMS) o[c] = fmaf(bonus ? S[j][c] : s, x.x, o[c]);
          S[j][c] = s;
        }
        if (bonus && PHASE != SCAN_CHUNK_SUMS) own += x.w;
        if (PHASE == SCAN_CHUNK_SUMS) P[j] *= x.z;
      }
      if (PHASE == SCAN_CHUNK_SUMS) continue;
      if (bonus) {
#pragma unroll
        for (int c = 0; c < COLS; c++) o[c] = fmaf(own, v[c], o[c]);
      }
      float* dst = out_rows + tt * p.heads * p.vdim;
      if (COLS == 4 && slices_log2 >= 2) {
        // four sums over the slices with five shuffles instead of four per sum: neighbours split the columns between
        // them (the even lane takes 0 and 1, the odd one 2 and 3), then pairs two apart split again; lane (b0, b1)
        // ends with column 2 b0 + b1, added up over the remaining lanes as usual
        const bool odd = slice & 1, upper = slice & 2;
        float keep0 = odd ? o[2 % COLS] : o[0], keep1 = odd ? o[3 % COLS] : o[1 % COLS];
        keep0 += __shfl_xor_sync(0xffffffffu, odd ? o[0] : o[2 % COLS], 1);
        keep1 += __shfl_xor_sync(0xffffffffu, odd ? o[1 % COLS] : o[3 % COLS], 1);
        float keep = upper ? keep1 : keep0;
        keep += __shfl_xor_sync(0xffffffffu, upper ? keep0 : keep1, 2);
        for (int d = 4; d < slices; d <<= 1) keep += __shfl_xor_sync(0xffffffffu, keep, d);
        const int c = 2 * (slice & 1) + ((slice >> 1) & 1);
        const float vc = c == 0 ? v[0] : c == 1 ? v[1 % COLS] : c == 2 ? v[2 % COLS] : v[3 % COLS];
        if (slice < 4 && col + c < p.vdim) dst[c] = fmaf(skip, vc, keep);
      } else {
#pragma unroll
        for (int c = 0; c < COLS; c++) {
          for (int d = slices >> 1; d > 0; d >>= 1) o[c] += __shfl_xor_sync(0xffffffffu, o[c], d);
          if (slice == 0 && col + c < p.vdim) dst[c] = fmaf(skip, v[c], o[c]);
        }
      }
    }
  }
  if (PHASE == SCAN_CHUNK_OUT && !last_chunk) return;
  float* to = PHASE == SCAN_CHUNK_SUMS ? held : mine;
  if (PAIRS) {
#pragma unroll
    for (int j = 0; j < ROWS / 2; j++) {
#pragma unroll
      for (int c = 0; c < COLS; c++) unpack2(S2[PAIRS ? j : 0][c], S[2 * j][c], S[2 * j + 1][c]);
      if (PHASE == SCAN_CHUNK_SUMS) unpack2(P2[PAIRS ? j : 0], P[(2 * j) % (PHASE == SCAN_CHUNK_SUMS ? ROWS : 1)], P[(2 * j + 1) % (PHASE == SCAN_CHUNK_SUMS ? ROWS : 1)]);
    }
  }
#pragma unroll
  for (int j = 0; j < ROWS; j++) {
    const int row = row_of(j);
    if (COLS == 4 && vectors) {
      if (col < p.vdim && row < dim)
        *reinterpret_cast<float4*>(to + (size_t)row * p.vdim + col) = make_float4(S[j][0], S[j][1 % COLS], S[j][2 % COLS], S[j][3 % COLS]);
    } else {
#pragma unroll
      for (int c = 0; c < COLS; c++)
        if (col + c < p.vdim && row < dim) to[(size_t)row * p.vdim + col + c] = S[j][c];
    }
    if (PHASE == SCAN_CHUNK_SUMS && blockIdx.z == 0 && col_local == 0 && row < dim)
      p.prods[((size_t)blockIdx.x * p.heads + h) * dim + row] = P[j];
  }
}

// The decays of every token of the step, once: per key channel a = sigmoid(z + bias)^(1 / tau); per head
// dt = softplus(z + bias), a = exp(-exp(a_log) dt), c = dt; with a floor what is written, 1 - a (`a_log` holds the floors);
// with a bonus a = exp(-exp(z + bias)).
// Threads own four neighbouring numbers of a row and walk the tokens: 16-byte accesses where rows lie on them (`vec`), and no division.
// 2,500 tokens of 2,048: 21 us with an element a thread and its place from a 64-bit division, 13 us so.
__global__ void __launch_bounds__(128)
scan_decay_kernel(const void* __restrict__ z, int z_stride, int z_f32, int is_bf16, const float* __restrict__ bias, const float* __restrict__ a_log,
                  float inv_tau, int mode, int heads, int dim, int tokens, int vec, float* __restrict__ da, float* __restrict__ dc) {
  pdl_launch_dependents();
  pdl_wait();
  const int per_token = mode == DECAY_PER_HEAD ? heads : heads * dim, c0 = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (c0 >= per_token) return;
  const bool wide = z_f32 || !is_bf16;
  const int n = min(4, per_token - c0);
  float b[4], al[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    b[i] = i < n ? bias[c0 + i] : 0.f;
    al[i] = i < n && a_log ? a_log[c0 + i] : 0.f;
  }
  for (int t = blockIdx.y; t < tokens; t += gridDim.y) {
    const size_t at = (size_t)t * z_stride + c0, to = (size_t)t * per_token + c0;
    float zv[4], a[4], d[4];
    if (vec && wide) {
      const float4 x = *(const float4*)((const float*)z + at);
      zv[0] = x.x; zv[1] = x.y; zv[2] = x.z; zv[3] = x.w;
    } else if (vec) {
      const uint2 x = *(const uint2*)((const __nv_bfloat16*)z + at);
      zv[0] = __uint_as_float(x.x << 16); zv[1] = __uint_as_float(x.x & 0xffff0000u);
      zv[2] = __uint_as_float(x.y << 16); zv[3] = __uint_as_float(x.y & 0xffff0000u);
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++)
        zv[i] = i >= n ? 0.f : wide ? ((const float*)z)[at + i] : to_float(((const __nv_bfloat16*)z)[at + i]);
    }
    if (mode == DECAY_PER_HEAD) {
#pragma unroll
      for (int i = 0; i < 4; i++) { d[i] = softplus_f(zv[i] + b[i]); a[i] = expf(-expf(al[i]) * d[i]); }
    } else if (mode == DECAY_FLOOR) {
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = write_share(zv[i] + b[i], al[i]);
    } else if (mode == DECAY_BONUS) {
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = double_exp_decay(zv[i] + b[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = expf(-softplus_f(-(zv[i] + b[i])) * inv_tau);
    }
    if (vec) {
      *(float4*)(da + to) = make_float4(a[0], a[1], a[2], a[3]);
      if (mode == DECAY_PER_HEAD) *(float4*)(dc + to) = make_float4(d[0], d[1], d[2], d[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i < n) {
          da[to + i] = a[i];
          if (mode == DECAY_PER_HEAD) dc[to + i] = d[i];
        }
    }
  }
}

// In the chunks' order, per element of a request's state: the scratch's entry of chunk c (the chunk's own sums)
// becomes the state before chunk c; requests of one chunk are left alone (their walk starts from the state slot).
__global__ void scan_carry_kernel(float* __restrict__ sums, const float* __restrict__ prods, const float* __restrict__ state,
                                  const int* __restrict__ q_start, const int* __restrict__ state_slots, int num_slots, int chunk,
                                  int heads, int dim, int vdim) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.z, h = blockIdx.y;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = (q_start[r + 1] - q_start[r] + chunk - 1) / chunk;
  const int slot = state_slots[r];
  if (n < 2 || e >= dim * vdim || slot < 0 || slot >= num_slots) return;
  int base = 0;
  for (int i = 0; i < r; i++) base += (q_start[i + 1] - q_start[i] + chunk - 1) / chunk;
  const int row = e / vdim;
  const size_t per = (size_t)heads * dim * vdim;
  float* mine = sums + (size_t)base * per + (size_t)h * dim * vdim + e;
  const float* decays = prods + ((size_t)base * heads + h) * dim + row;
  float S = state[((size_t)slot * heads + h) * dim * vdim + e];
  const size_t decay_step = (size_t)heads * dim;
  for (int c0 = 0; c0 + 1 < n; c0 += 8) {              // eight chunks' loads are in flight before the first is used
    float own[8], a[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const bool there = c0 + u + 1 < n;
      own[u] = there ? mine[(size_t)(c0 + u) * per] : 0.f;
      a[u] = there ? decays[(size_t)(c0 + u) * decay_step] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      if (c0 + u + 1 >= n) break;
      mine[(size_t)(c0 + u) * per] = S;
      S = fmaf(a[u], S, own[u]);
    }
  }
  mine[(size_t)(n - 1) * per] = S;
}

constexpr int CONV_MAX_TAPS = 8, CONV_TOKENS = 32;

// grid (blocks of CONV_TOKENS tokens of one request, numbered over the requests in order; blocks of 128 channels); a thread walks
// its channel through its tokens with the last taps - 1 inputs in registers.  As many tokens as requests are one each.  The block of
// a request's first tokens reads the state (before anything writes it) and is the one that writes the new state at its end.
template <typename T>
__global__ void __launch_bounds__(128)
causal_conv_kernel(const T* __restrict__ in, int in_stride, const float* __restrict__ weight, const float* __restrict__ bias,
                   T* __restrict__ out, int out_stride, const int* __restrict__ q_start, const int* __restrict__ state_slots,
                   float* __restrict__ state, int num_slots, int tokens, int requests, int channels, int taps, int act, int* status) {
  pdl_launch_dependents();
  pdl_wait();
  int r = blockIdx.x, part = 0, parts;
  if (tokens != requests && !warp_find_piece(q_start, requests, CONV_TOKENS, blockIdx.x, r, part, parts)) return;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const int begin = q_start[r], end = q_start[r + 1];
  const int first = begin + part * CONV_TOKENS;
  if (c >= channels) return;
  const int slot = state_slots[r];
  if (slot < 0 || slot >= num_slots) {
    if (threadIdx.x == 0) atomicOr(status, SPROUT_STATUS_BAD_PAGE);
    return;
  }
  float* mine = state + (size_t)slot * (taps - 1) * channels + c;       // [taps - 1, channels], oldest first
  float w[CONV_MAX_TAPS], hist[CONV_MAX_TAPS];                           // hist[b]: the input b tokens back
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; j++) {
    w[j] = j < taps ? weight[(size_t)c * taps + j] : 0.f;
    hist[j] = 0.f;
  }
#pragma unroll
  for (int b = 1; b < CONV_MAX_TAPS; b++) {
    if (b >= taps) break;
    const int j = first - b;
    hist[b] = j >= begin ? to_float(in[(size_t)j * in_stride + c]) : mine[(size_t)(taps - 1 + (j - begin)) * channels];
  }
  float old[CONV_MAX_TAPS];                                              // the state as it was: old[b] is b tokens before the portion
#pragma unroll
  for (int b = 0; b < CONV_MAX_TAPS; b++) old[b] = hist[b];
  const float offset = bias ? bias[c] : 0.f;
  const int stop = min(first + CONV_TOKENS, end);
  for (int t = first; t < stop; t++) {
    hist[0] = to_float(in[(size_t)t * in_stride + c]);
    float y = offset;
#pragma unroll
    for (int b = CONV_MAX_TAPS - 1; b >= 0; b--)
      if (b < taps) y = fmaf(w[taps - 1 - b], hist[b], y);               // oldest input first
    out[(size_t)t * out_stride + c] = from_float<T>(act ? silu_g(y) : y);
#pragma unroll
    for (int b = CONV_MAX_TAPS - 1; b > 0; b--) hist[b] = hist[b - 1];
  }
  if (part != 0) return;
  // the new state: the last taps - 1 inputs of what the request has seen, oldest first
#pragma unroll
  for (int s = 0; s < CONV_MAX_TAPS - 1; s++) {
    if (s >= taps - 1) break;
    const int j = end - (taps - 1) + s;
    float value;
    if (j >= begin) {
      value = to_float(in[(size_t)j * in_stride + c]);
    } else {
      const int back = begin - j;                                        // 1 .. taps - 1 tokens before the portion
      value = 0.f;
#pragma unroll
      for (int b = 1; b < CONV_MAX_TAPS; b++)
        if (b == back) value = old[b];
    }
    mine[(size_t)s * channels] = value;
  }
}

// A thread takes VEC neighbouring elements of one row in every part.  The thread of a portion's first token reads the row before
// it from the request's state and then puts the request's last row there (no other thread touches that element).
template <typename T, int VEC>
__global__ void __launch_bounds__(256)
token_blend_kernel(const T* __restrict__ h, const float* __restrict__ mu, T* __restrict__ out, const int* __restrict__ q_start,
                   const int* __restrict__ seq_of_token, const int* __restrict__ state_slots, float* __restrict__ state, int num_slots,
                   int tokens, int width, int parts, int* status) {
  pdl_launch_dependents();
  pdl_wait();
  const int per_row = width / VEC;
  const long long count = (long long)tokens * per_row;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < count; e += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(e / per_row), c = (int)(e - (long long)t * per_row) * VEC;
    const int r = seq_of_token[t], begin = q_start[r];
    float now[VEC], delta[VEC];
    auto row = [&](int token, float (&v)[VEC]) {
      const T* src = h + (size_t)token * width + c;
      if (VEC == 8 && sizeof(T) == 2) {
        const uint4 raw = *reinterpret_cast<const uint4*>(src);
        const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int i = 0; i < VEC / 2; i++) {
          const float2 f = __bfloat1622float2(pairs[i]);
          v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < VEC; i++) v[i] = to_float(src[i]);
      }
    };
    auto floats = [&](const float* src, float (&v)[VEC]) {
      if (VEC == 8) {
        const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
        v[0] = a.x; v[1 % VEC] = a.y; v[2 % VEC] = a.z; v[3 % VEC] = a.w;
        v[4 % VEC] = b.x; v[5 % VEC] = b.y; v[6 % VEC] = b.z; v[7 % VEC] = b.w;
      } else {
#pragma unroll
        for (int i = 0; i < VEC; i++) v[i] = src[i];
      }
    };
    row(t, now);
    if (t > begin) {
      row(t - 1, delta);
    } else {
      const int slot = state_slots[r];
      if (slot < 0 || slot >= num_slots) {
        if (c == 0) atomicOr(status, SPROUT_STATUS_BAD_PAGE);
#pragma unroll
        for (int i = 0; i < VEC; i++) delta[i] = 0.f;
      } else {
        float* mine = state + (size_t)slot * width + c;
        float last[VEC];
        row(q_start[r + 1] - 1, last);
        floats(mine, delta);
        if (VEC == 8) {
          reinterpret_cast<float4*>(mine)[0] = make_float4(last[0], last[1 % VEC], last[2 % VEC], last[3 % VEC]);
          reinterpret_cast<float4*>(mine)[1] = make_float4(last[4 % VEC], last[5 % VEC], last[6 % VEC], last[7 % VEC]);
        } else {
#pragma unroll
          for (int i = 0; i < VEC; i++) mine[i] = last[i];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < VEC; i++) delta[i] -= now[i];
#pragma unroll 5
    for (int s = 0; s < parts; s++) {
      float m[VEC];
      floats(mu + (size_t)s * width + c, m);
      T* dst = out + ((size_t)t * parts + s) * width + c;
      if (VEC == 8 && sizeof(T) == 2) {
        uint4 packed;
        __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
        for (int i = 0; i < VEC / 2; i++)
          pairs[i] = __floats2bfloat162_rn(fmaf(delta[2 * i], m[2 * i], now[2 * i]), fmaf(delta[2 * i + 1], m[2 * i + 1], now[2 * i + 1]));
        *reinterpret_cast<uint4*>(dst) = packed;
      } else {
#pragma unroll
        for (int i = 0; i < VEC; i++) dst[i] = from_float<T>(fmaf(delta[i], m[i], now[i]));
      }
    }
  }
}

// grid (rows, groups).  o float32 [rows, width]; gate rows of TG with their own stride; out rows of T.
template <typename TG, typename T>
__global__ void __launch_bounds__(128)
gated_group_norm_kernel(const float* __restrict__ o, const TG* __restrict__ gate, int gate_stride, const float* __restrict__ weight,
                        int period, T* __restrict__ out, int width, int groups, float eps, int gate_first, int act) {
  __shared__ float scratch[33];
  pdl_launch_dependents();
  pdl_wait();
  const int part = width / groups, base = blockIdx.y * part;
  const float* src = o + (size_t)blockIdx.x * width + base;
  const TG* grow = gate ? gate + (size_t)blockIdx.x * gate_stride + base : nullptr;
  float q = 0.f;
  for (int i = threadIdx.x; i < part; i += blockDim.x) {
    float v = src[i];
    if (gate_first) {
      const float gv = to_float(grow[i]);
      v *= act ? silu_g(gv) : sigmoid_g(gv);
    }
    q = fmaf(v, v, q);
  }
  const float r = 1.0f / sqrtf(block_sum(q, scratch) / (float)part + eps);
  T* dst = out + (size_t)blockIdx.x * width + base;
  for (int i = threadIdx.x; i < part; i += blockDim.x) {
    const float gv = grow ? to_float(grow[i]) : 0.f;
    const float factor = !grow ? 1.0f : act ? silu_g(gv) : sigmoid_g(gv);
    const float v = gate_first ? (src[i] * factor) * r * weight[(base + i) % period] : src[i] * r * weight[(base + i) % period] * factor;
    dst[i] = from_float<T>(v);
  }
}

// The same for parts that a warp's lanes hold (up to 128 elements in multiples of 4, up to 256 in multiples of 8) whose rows start on 16
// bytes: the lanes of a warp share PARTS parts of a row (32 / LANES of them, LANES = part / VEC rounded up to a power of two), VEC elements a lane in 16-byte accesses, the part in registers
// between its sum and its scaling, no block-wide barrier.  Bound by memory: 2,500 rows of 16 parts of 128: 45 us as a block of 128
// threads per part, 19 us with 4 elements a lane placed by 64-bit divisions, 13 us so.
template <typename TG, int VEC>
__global__ void __launch_bounds__(256)
gated_group_norm_warp_kernel(const float* __restrict__ o, const TG* __restrict__ gate, int gate_stride, const float* __restrict__ weight,
                             int period, __nv_bfloat16* __restrict__ out, int width, int groups, int lanes_log2, unsigned parts, float eps, int gate_first, int act) {
  pdl_launch_dependents();
  pdl_wait();
  const int part = width / groups, lanes = 1 << lanes_log2, lane = threadIdx.x & (lanes - 1);
  const unsigned index = (blockIdx.x * (256u >> lanes_log2)) + (threadIdx.x >> lanes_log2);
  const bool active = index < parts && lane * VEC < part;
  const unsigned row = active ? index / (unsigned)groups : 0;
  const int base = active ? (int)(index - row * (unsigned)groups) * part + lane * VEC : 0;
  float v[VEC], factor[VEC];
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < VEC; i++) { v[i] = 0.f; factor[i] = 1.f; }
  if (active) {
    const float4* src = (const float4*)(o + (size_t)row * width + base);
#pragma unroll
    for (int i = 0; i < VEC / 4; i++) {
      const float4 x = src[i];
      v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
    }
    if (gate) {
      const TG* g = gate + (size_t)row * gate_stride + base;
      float gv[VEC];
      if (sizeof(TG) == 4) {
#pragma unroll
        for (int i = 0; i < VEC / 4; i++) {
          const float4 x = ((const float4*)g)[i];
          gv[4 * i] = x.x; gv[4 * i + 1] = x.y; gv[4 * i + 2] = x.z; gv[4 * i + 3] = x.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < VEC / 4; i++) {
          const uint2 x = ((const uint2*)g)[i];
          gv[4 * i] = __uint_as_float(x.x << 16); gv[4 * i + 1] = __uint_as_float(x.x & 0xffff0000u);
          gv[4 * i + 2] = __uint_as_float(x.y << 16); gv[4 * i + 3] = __uint_as_float(x.y & 0xffff0000u);
        }
      }
#pragma unroll
      for (int i = 0; i < VEC; i++) factor[i] = act ? silu_g(gv[i]) : sigmoid_g(gv[i]);
    }
#pragma unroll
    for (int i = 0; i < VEC; i++) {
      if (gate_first) v[i] *= factor[i];
      q = fmaf(v[i], v[i], q);
    }
  }
  for (int d = lanes >> 1; d > 0; d >>= 1) q += __shfl_xor_sync(0xffffffffu, q, d);
  if (!active) return;
  const float r = 1.0f / sqrtf(q / (float)part + eps);
  __nv_bfloat16* dst = out + (size_t)row * width + base;
  const int first = base % period;                     // a lane's weights follow one another unless the period ends among them
  const bool run = first + VEC <= period;
#pragma unroll
  for (int i = 0; i < VEC; i += 4) {
    float y[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float w = weight[run ? first + i + e : (first + i + e) % period];
      y[e] = gate_first ? v[i + e] * r * w : v[i + e] * r * w * factor[i + e];
    }
    __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[1]), hi = __floats2bfloat162_rn(y[2], y[3]);
    *(uint2*)(dst + i) = make_uint2(*(uint32_t*)&lo, *(uint32_t*)&hi);
  }
}

template <typename TG, typename T>
int launch_group_norm(const float* o, const void* gate, int gate_stride, const float* weight, int period, void* out, int rows, int width,
                      int groups, float eps, int gate_first, int act, cudaStream_t stream) {
  const int part = width / groups;
  const bool aligned = part % 4 == 0 && part <= 256 && (!gate || gate_stride % 4 == 0) && ((uintptr_t)o & 15) == 0 && ((uintptr_t)out & 15) == 0 &&
                       ((uintptr_t)gate & 15) == 0;
  // the 32-bit path keeps one order of additions for all its calls: the block kernel's.  Below 1,024 parts either kernel is one short wave
  // and the block kernel's is shorter (256 parts of 256: 2.95 against 3.37 us; 512 of 64: 2.36 and 2.45; 1,024 of 128: 2.87 and 2.52).
  if constexpr (sizeof(T) == 2) if (aligned && (long long)rows * groups >= 1024) {
    const int vec = part % 8 == 0 && part >= 64 ? 8 : 4;
    int lanes_log2 = 0;
    while ((vec << lanes_log2) < part) lanes_log2++;
    const long long parts = (long long)rows * groups, blocks = ((parts << lanes_log2) + 255) / 256;
    if (part % vec == 0 && lanes_log2 <= 5 && parts <= 0x7fffffffLL) {        // a part is one warp's: 132 to 252 in fours that are not eights are not
      SPROUT_REQUIRE(blocks <= 0x7fffffffLL, "gated_group_norm: too many rows");
      if (vec == 8)
        sprout_launch(gated_group_norm_warp_kernel<TG, 8>, dim3((unsigned)blocks), dim3(256), 0, stream, o, (const TG*)gate, gate_stride, weight,
                      period, (T*)out, width, groups, lanes_log2, (unsigned)parts, eps, gate_first, act);
      else
        sprout_launch(gated_group_norm_warp_kernel<TG, 4>, dim3((unsigned)blocks), dim3(256), 0, stream, o, (const TG*)gate, gate_stride, weight,
                      period, (T*)out, width, groups, lanes_log2, (unsigned)parts, eps, gate_first, act);
      return sprout_check_launch("gated_group_norm");
    }
  }
  sprout_launch(gated_group_norm_kernel<TG, T>, dim3(rows, groups), dim3(128), 0, stream, o, (const TG*)gate, gate_stride, weight, period, (T*)out,
                width, groups, eps, gate_first, act);
  return sprout_check_launch("gated_group_norm");
}

__global__ void scaled_sum_kernel(float* __restrict__ x, const float* __restrict__ y1, float a, const float* __restrict__ y2,
                                  float b, long long count) {
  pdl_launch_dependents();
  pdl_wait();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
    x[i] += a * y1[i] + (y2 ? b * y2[i] : 0.f);
}

template <typename T, int ROWS, int COLS, int FORM>
int launch_scan_tiles(const ScanParams<T>& p, bool pairs, int requests, int max_chunks, cudaStream_t stream) {
  int slices_log2 = 0;
  while ((ROWS << slices_log2) < p.dim) slices_log2++;
  SPROUT_REQUIRE(slices_log2 <= 5, "gated_scan: key vectors too long (%d)", p.dim);
  const int slices = 1 << slices_log2, cb = SCAN_THREADS / slices * COLS;
  // tokens of a batch: what a thread stages in registers bounds it (row vectors: ROWS * slices * batch / threads <= 8 or 16;
  // values: cb * batch / threads <= SCAN_MAX_TOKENS)
  int batch = SCAN_MAX_TOKENS;
  const int by_rows = (ROWS == 8 ? 128 : 64) / slices, by_values = SCAN_MAX_TOKENS * slices / COLS;
  if (batch > by_rows) batch = by_rows;
  if (batch > by_values) batch = by_values;
  // single walks (few tokens: the state's way in and out is most of their time, and rows dealt in turn read it faster: 64 single tokens
  // of 16 heads 46 against 52 us) keep a number at a time, and so does the 32-bit path, whose sums have one order in both walks
  constexpr bool PAIRED = ROWS == 8 && COLS == 4 && sizeof(T) == 2;
  pairs = pairs && PAIRED;
  const size_t smem = (size_t)batch * ((size_t)ROWS * slices * sizeof(float4) + (size_t)cb * sizeof(float));
  const size_t smem_chunks = pairs ? (size_t)batch * ((size_t)4 * 2 * (ROWS * slices / 2 + 16) + cb) * sizeof(float) : smem;
  const dim3 grid(requests, p.heads, (p.vdim + cb - 1) / cb);
  SPROUT_REQUIRE(grid.z <= 65535, "gated_scan: too many value columns");
  if (p.sums == nullptr && p.mode == DECAY_GIVEN) {
    sprout_launch(gated_scan_kernel<T, ROWS, COLS, SCAN_CHUNK_OUT, FORM, false>, grid, dim3(SCAN_THREADS), smem, stream, p, slices_log2, batch);
    return sprout_check_launch("gated_scan");
  }
  if (p.sums == nullptr) {
    sprout_launch(gated_scan_kernel<T, ROWS, COLS, SCAN_WHOLE, FORM, false>, grid, dim3(SCAN_THREADS), smem, stream, p, slices_log2, batch);
    return sprout_check_launch("gated_scan");
  }
  // `max_chunks` blocks per (head, columns): the chunks of all requests, found by their number
  const dim3 chunks(max_chunks, p.heads, grid.z);
  bool mma = false;                                    // 16 tokens at a time on tensor cores
  if constexpr (sizeof(T) == 2 && FORM == FORM_PLAIN) mma = scan_mma_takes(p);
  auto walk = [&](int phase) {
    if constexpr (sizeof(T) == 2 && FORM == FORM_PLAIN)
      if (mma) return launch_scan_mma(p, phase, max_chunks, stream);
    auto* kernel = phase == SCAN_CHUNK_SUMS ? (pairs ? gated_scan_kernel<T, ROWS, COLS, SCAN_CHUNK_SUMS, FORM, PAIRED> : gated_scan_kernel<T, ROWS, COLS, SCAN_CHUNK_SUMS, FORM, false>)
                                            : (pairs ? gated_scan_kernel<T, ROWS, COLS, SCAN_CHUNK_OUT, FORM, PAIRED> : gated_scan_kernel<T, ROWS, COLS, SCAN_CHUNK_OUT, FORM, false>);
    sprout_launch(kernel, chunks, dim3(SCAN_THREADS), smem_chunks, stream, p, slices_log2, batch);
    return sprout_check_launch(phase == SCAN_CHUNK_SUMS ? "gated_scan (chunk sums)" : "gated_scan (chunk outputs)");
  };
  if (int rc = walk(SCAN_CHUNK_SUMS)) return rc;
  SPROUT_REQUIRE(requests <= 65535, "gated_scan: too many requests");
  sprout_launch(scan_carry_kernel, dim3((p.dim * p.vdim + 255) / 256, p.heads, requests), dim3(256), 0, stream, p.sums,
                (const float*)p.prods, (const float*)p.state, p.q_start, p.state_slots, p.num_slots, p.chunk, p.heads, p.dim, p.vdim);
  if (int rc = sprout_check_launch("gated_scan (carry)")) return rc;
  return walk(SCAN_CHUNK_OUT);
}

template <typename T>
int launch_scan(const ScanParams<T>& p, int requests, int max_chunks, cudaStream_t stream) {
  // pairs of rows: the key's rows fill the tile's slices, and every row starts on a 16-byte boundary
  constexpr int per16 = 16 / (int)sizeof(T);
  auto on16 = [](const void* x) { return ((uintptr_t)x & 15) == 0; };
  const bool pairs = (p.dim == 64 || p.dim == 128 || p.dim == 256) && p.q_stride % per16 == 0 && (!p.k || p.k_stride % per16 == 0) && on16(p.q) &&
                     on16(p.k) && on16(p.da);
  // a thread's tile of the state: 8 rows x 4 columns up to 256 key channels, 32 rows of one column up to 1024
  const bool narrow = p.dim <= 8 * 32;
  if (p.mode == DECAY_FLOOR)
    return narrow ? launch_scan_tiles<T, 8, 4, FORM_FLOOR>(p, pairs, requests, max_chunks, stream) : launch_scan_tiles<T, 32, 1, FORM_FLOOR>(p, pairs, requests, max_chunks, stream);
  if (p.mode == DECAY_BONUS)
    return narrow ? launch_scan_tiles<T, 8, 4, FORM_BONUS>(p, pairs, requests, max_chunks, stream) : launch_scan_tiles<T, 32, 1, FORM_BONUS>(p, pairs, requests, max_chunks, stream);
  return narrow ? launch_scan_tiles<T, 8, 4, FORM_PLAIN>(p, pairs, requests, max_chunks, stream) : launch_scan_tiles<T, 32, 1, FORM_PLAIN>(p, pairs, requests, max_chunks, stream);
}

}  // namespace

SPROUT_API int sprout_gated_scan(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                                 const void* z, int z_stride, int z_f32, int dtype, const float* bias, const float* a_log, const float* skip, const float* bonus,
                                 float inv_tau, float q_scale, int mode, int requests, int heads, int groups, int dim, int vdim,
                                 const int* q_start, const int* state_slots, float* state, int num_slots, float* out, int* status,
                                 int tokens, int chunk, int max_chunks, float* da, float* dc, float* sums, float* prods,
                                 int v_cols, int ones_col, int q_silu, cudaStream_t stream) {
  SPROUT_REQUIRE(q && (k || mode == DECAY_FLOOR) && v && q_start && state_slots && state && out && status, "gated_scan: null pointer");
  SPROUT_REQUIRE(mode == DECAY_GIVEN ? (da && dc) : (z && bias), "gated_scan: the decay's inputs are missing");
  SPROUT_REQUIRE(v_cols > 0 && v_cols <= vdim && (!ones_col || v_cols < vdim), "gated_scan: the value rows' columns do not fit the state's");
  if (mode == DECAY_GIVEN && !sums) {
    // one walk per request over ready-made decays: the outputs' walk of the chunked form with a chunk that holds any portion
    chunk = 1 << 30;
    max_chunks = requests;
  }
  if (sums && mode != DECAY_GIVEN) {
    // portions in chunks: scratch for the decays of every token and for every chunk's sums and decay product
    SPROUT_REQUIRE(chunk > 0 && max_chunks > 0 && tokens > 0 && da && prods && (mode != DECAY_PER_HEAD || dc),
                   "gated_scan: the chunked form needs its scratch");
    const int per_token = mode == DECAY_PER_HEAD ? heads : heads * dim, item = z_f32 || dtype != SPROUT_BF16 ? 4 : 2;
    const int vec = per_token % 4 == 0 && z_stride % 4 == 0 && ((uintptr_t)z & (4 * item - 1)) == 0 && (((uintptr_t)da | (uintptr_t)dc) & 15) == 0;
    const int columns = (per_token + 511) / 512, walkers = 16 * sprout_sm_count() / columns;
    sprout_launch(scan_decay_kernel, dim3(columns, tokens < walkers ? tokens : walkers < 1 ? 1 : walkers), dim3(128), 0, stream, z, z_stride, z_f32,
                  dtype == SPROUT_BF16 ? 1 : 0, bias, a_log, inv_tau, mode, heads, dim, tokens, vec, da, dc);
    if (int rc = sprout_check_launch("gated_scan (decays)")) return rc;
  }
  SPROUT_REQUIRE(requests > 0 && heads > 0 && groups > 0 && heads % groups == 0 && dim > 0 && vdim > 0 && num_slots > 0,
                 "gated_scan: bad sizes");
  SPROUT_REQUIRE(mode == DECAY_PER_CHANNEL || ((mode == DECAY_PER_HEAD || mode == DECAY_FLOOR) && a_log) || mode == DECAY_GIVEN ||
                 (mode == DECAY_BONUS && bonus), "gated_scan: unknown decay form");
  SPROUT_REQUIRE(!q_silu || mode == DECAY_FLOOR, "gated_scan: silu on the queries goes with a floor");
  SPROUT_REQUIRE((mode != DECAY_FLOOR && mode != DECAY_BONUS) || groups == heads, "gated_scan: a forget gate with a floor or a bonus has query vectors per head");
  SPROUT_REQUIRE(heads <= 65535, "gated_scan: too many heads");
  if (dtype == SPROUT_F32) {
    ScanParams<float> p{(const float*)q, q_stride, (const float*)k, k_stride, (const float*)v, v_stride, z, z_stride, z_f32,
                        bias, a_log, skip, bonus, inv_tau, q_scale, mode, heads, groups, dim, vdim, q_start, state_slots, state,
                        num_slots, out, status, da, dc, sums, prods, chunk, requests, q_silu, v_cols, ones_col};
    return launch_scan(p, requests, max_chunks, stream);
  }
  if (dtype == SPROUT_BF16) {
    ScanParams<__nv_bfloat16> p{(const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k, k_stride, (const __nv_bfloat16*)v,
                                v_stride, z, z_stride, z_f32, bias, a_log, skip, bonus, inv_tau, q_scale, mode, heads,
                                groups, dim, vdim, q_start, state_slots, state, num_slots, out, status, da, dc, sums, prods, chunk,
                                requests, q_silu, v_cols, ones_col};
    return launch_scan(p, requests, max_chunks, stream);
  }
  return sprout_fail("gated_scan: unknown dtype %d", dtype);
}

// The grid follows `tokens` and `requests` alone: a captured launch is replayed for other cuttings of the same tokens.
SPROUT_API int sprout_causal_conv(const void* in, int in_stride, const float* weight, const float* bias, void* out, int out_stride,
                                  int dtype, const int* q_start, const int* state_slots, float* state, int num_slots, int requests,
                                  int tokens, int channels, int taps, int act, int* status, cudaStream_t stream) {
  SPROUT_REQUIRE(in && weight && out && q_start && state_slots && state && status, "causal_conv: null pointer");
  SPROUT_REQUIRE(requests > 0 && tokens > 0 && channels > 0 && num_slots > 0, "causal_conv: bad sizes");
  SPROUT_REQUIRE(taps >= 2 && taps <= CONV_MAX_TAPS, "causal_conv: 2 to %d taps (got %d)", CONV_MAX_TAPS, taps);
  SPROUT_REQUIRE(in_stride >= channels && out_stride >= channels, "causal_conv: rows shorter than the channels");
  const dim3 grid(tokens == requests ? requests : tokens / CONV_TOKENS + requests, (channels + 127) / 128);
  SPROUT_REQUIRE(grid.y <= 65535, "causal_conv: too many channels");
  if (dtype == SPROUT_F32)
    sprout_launch(causal_conv_kernel<float>, grid, dim3(128), 0, stream, (const float*)in, in_stride, weight, bias, (float*)out,
                  out_stride, q_start, state_slots, state, num_slots, tokens, requests, channels, taps, act, status);
  else if (dtype == SPROUT_BF16)
    sprout_launch(causal_conv_kernel<__nv_bfloat16>, grid, dim3(128), 0, stream, (const __nv_bfloat16*)in, in_stride, weight, bias,
                  (__nv_bfloat16*)out, out_stride, q_start, state_slots, state, num_slots, tokens, requests, channels, taps, act, status);
  else
    return sprout_fail("causal_conv: unknown dtype %d", dtype);
  return sprout_check_launch("causal_conv");
}

// out [tokens, parts, width]: row t of part s = h_t + (h_(t-1) - h_t) * mu[s]; state float32 [slots, width], the last row of
// every request.
SPROUT_API int sprout_token_blend(const void* h, const float* mu, void* out, int dtype, const int* q_start, const int* seq_of_token,
                                  const int* state_slots, float* state, int num_slots, int tokens, int width, int parts, int* status,
                                  cudaStream_t stream) {
  SPROUT_REQUIRE(h && mu && out && q_start && seq_of_token && state_slots && state && status, "token_blend: null pointer");
  SPROUT_REQUIRE(tokens > 0 && width > 0 && parts > 0 && num_slots > 0, "token_blend: bad sizes");
  const bool vec = dtype == SPROUT_BF16 && width % 8 == 0 && (((uintptr_t)h | (uintptr_t)out | (uintptr_t)mu | (uintptr_t)state) & 15) == 0;
  // few tokens: small blocks, so that more SMs have one
  const long long threads = (long long)tokens * (width / (vec ? 8 : 1));
  const int block = threads < 148 * 256 ? 64 : 256;
  const long long blocks = (threads + block - 1) / block;
  const dim3 grid((unsigned)(blocks < 148 * 16 ? blocks : 148 * 16));
  if (dtype == SPROUT_F32)
    sprout_launch(token_blend_kernel<float, 1>, grid, dim3(block), 0, stream, (const float*)h, mu, (float*)out, q_start, seq_of_token,
                  state_slots, state, num_slots, tokens, width, parts, status);
  else if (vec)
    sprout_launch(token_blend_kernel<__nv_bfloat16, 8>, grid, dim3(block), 0, stream, (const __nv_bfloat16*)h, mu, (__nv_bfloat16*)out,
                  q_start, seq_of_token, state_slots, state, num_slots, tokens, width, parts, status);
  else if (dtype == SPROUT_BF16)
    sprout_launch(token_blend_kernel<__nv_bfloat16, 1>, grid, dim3(block), 0, stream, (const __nv_bfloat16*)h, mu, (__nv_bfloat16*)out,
                  q_start, seq_of_token, state_slots, state, num_slots, tokens, width, parts, status);
  else
    return sprout_fail("token_blend: unknown dtype %d", dtype);
  return sprout_check_launch("token_blend");
}

SPROUT_API int sprout_gated_group_norm(const float* o, const void* gate, int gate_stride, int gate_dtype, const float* weight, int period, void* out,
                                       int dtype, int rows, int width, int groups, float eps, int gate_first, int act,
                                       cudaStream_t stream) {
  SPROUT_REQUIRE(o && (gate || !gate_first) && weight && out && rows > 0 && width > 0 && eps > 0, "gated_group_norm: bad arguments");
  SPROUT_REQUIRE(groups > 0 && groups <= 65535 && width % groups == 0 && period > 0 && (!gate || gate_stride >= width),
                 "gated_group_norm: the row must divide into the groups, gate rows must hold the row");
  SPROUT_REQUIRE(!gate || gate_dtype == dtype || gate_dtype == SPROUT_F32, "gated_group_norm: the gate is of out's type or float32");
  if (dtype == SPROUT_F32)
    return launch_group_norm<float, float>(o, gate, gate_stride, weight, period, out, rows, width, groups, eps, gate_first, act, stream);
  if (dtype == SPROUT_BF16 && gate && gate_dtype == SPROUT_F32)
    return launch_group_norm<float, __nv_bfloat16>(o, gate, gate_stride, weight, period, out, rows, width, groups, eps, gate_first, act, stream);
  if (dtype == SPROUT_BF16)
    return launch_group_norm<__nv_bfloat16, __nv_bfloat16>(o, gate, gate_stride, weight, period, out, rows, width, groups, eps, gate_first, act, stream);
  return sprout_fail("gated_group_norm: unknown dtype %d", dtype);
}

SPROUT_API int sprout_scaled_sum(float* x, const float* y1, float a, const float* y2, float b, long long count, cudaStream_t stream) {
  SPROUT_REQUIRE(x && y1 && count > 0, "scaled_sum: bad arguments");
  const long long blocks = (count + 255) / 256;
  sprout_launch(scaled_sum_kernel, dim3((unsigned)(blocks < 148 * 8 ? blocks : 148 * 8)), dim3(256), 0, stream, x, y1, a, y2, b, count);
  return sprout_check_launch("scaled_sum");
}
