// The gated scan's walks over chunks on tensor cores (bfloat16 q, k, v; key sizes 64 and 128; decays per channel or per head), 16 tokens
// at a time.  With a_t the decay of a key channel, P(j, i) = a_(j+1) ... a_i and the state S before the 16 tokens,
//
//   o_i = (q_i P(0, i))^T S + sum_(j <= i) A_ij v_j,   A_ij = sum_d q_i k_j P(j, i),       S <- P(0, 16) S + sum_j (k_j P(j, 16)) v_j^T.
//
// Every P is a product of decays (at most 1), never a quotient, so decays of any strength pass.
//
// Nothing is rounded to 16 bits on the way: a float32 operand of the tensor cores goes in as three bfloat16 terms (value = high + middle
// + low, 24 bits together), the products of which down to 2^-24 are added up in float32 (3 of them against the values v, which are
// bfloat16 as they come, 6 between two such operands).  The triangle A is float32 on the CUDA cores: P(j, i) by running products, a
// key row's 128 channels over a warp's lanes.
//
// A block of four warps owns (chunk, head, 4 WC value columns); a warp keeps S^T for its WC columns in the accumulators' registers, where
// it has the layout of the A operand of o^T = S^T q^T, so it is split into terms without leaving the registers.  The vectors of the next
// 16 tokens come by cp.async while these are worked on.
//
// Infinities and NaN: the terms of an infinity are not one (infinity - infinity), and the tensor cores multiply the triangle's zeros with
// the values of tokens that an output does not see.  Either way what comes out is NaN, never a wrong number, and only in the value columns
// of such a value or state, or in all columns from a token on.  So such columns' 16 tokens are walked again in turn (`walk`), which gives
// the outputs that are not finite and the state; the outputs that are finite stay as they came.  A value reaches its own column from its
// own token on, as in the walk token by token.  Looking for them costs 2,500 tokens of three requests 8 of 263 us (the layer).
//
// Bound by the issue of instructions (some 300 products and 1,700 others a warp and 16 tokens) at eight warps an SM; walking token by
// token, every element of S took a packed multiply and multiply-add a token.  2,500 tokens of three requests, 16 heads of 128 x 128: in
// chunks of 64 the sums' walk 106 us there and 29 here, the outputs' 243 and 105; in the chunks of 160 that `kernels.scan_mma_chunk` gives
// them, cold caches, 28 and 99, the layer 262 (565 token by token); the outputs' error against 64 bits 1.5e-7 in both, the states' 1.4e-7
// and 1.3e-7.
#include "attention_bf16.cuh"
#include "gated_scan.cuh"

using namespace sprout_scan;
using namespace sprout_attn;

namespace {

constexpr int STEP = 16, THREADS = 128;

template <int DIM, int WC, bool PER_HEAD>
struct Shape {
  static constexpr int COLS = 4 * WC;                          // value columns of a block
  static constexpr int ROW = DIM * 2 + 16, V_ROW = COLS * 2 + 16, A_ROW = STEP * 2 + 16;     // padded rows: ldmatrix without conflicts
  static constexpr int Q_BYTES = STEP * DIM * 2, DECAY_BYTES = PER_HEAD ? 2 * STEP * 4 : STEP * DIM * 4, V_BYTES = STEP * V_ROW;
  static constexpr int STAGE = 2 * Q_BYTES + DECAY_BYTES + V_BYTES;                           // q, k, decays (and factors), v of a step
  static constexpr int OFF_QS = 2 * STAGE, OFF_KS = OFF_QS + 3 * STEP * ROW, OFF_A = OFF_KS + 3 * STEP * ROW, OFF_D = OFF_A + 3 * STEP * A_ROW;
  static constexpr int BYTES = OFF_D + DIM * 4;
};

// x0, x1 as three pairs of bfloat16 terms.
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& high, uint32_t& mid, uint32_t& low) {
  high = pack_bf16(x0, x1);
  const float r0 = x0 - __uint_as_float(high << 16), r1 = x1 - __uint_as_float(high & 0xffff0000u);
  mid = pack_bf16(r0, r1);
  low = pack_bf16(r0 - __uint_as_float(mid << 16), r1 - __uint_as_float(mid & 0xffff0000u));
}

// C = A B from zero.  The tensor cores cut off where float32 sums are rounded to nearest: at most a few products go into one of their
// sums, and those sums are added on the CUDA cores (o of 2,500 tokens with all products in one sum: 6.4e-7 off 64 bits, 1.6e-7 so).
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ void cp_async16_or_zero(void* smem, const void* gmem, bool there) {
  const int bytes = there ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes));
}

template <int DIM, int WC, bool PER_HEAD, int PHASE>
__global__ void __launch_bounds__(THREADS, 2)
scan_mma_kernel(const ScanParams<__nv_bfloat16> p) {
  using L = Shape<DIM, WC, PER_HEAD>;
  constexpr bool OUT = PHASE == SCAN_CHUNK_OUT;
  constexpr int MT = WC / 16, KT = DIM / 16, LANE_DIMS = DIM / 32;
  extern __shared__ __align__(16) uint8_t smem[];
  float* total = (float*)(smem + L::OFF_D);                    // P(0, 16) per channel
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c2 = 2 * (lane & 3);
  const int h = blockIdx.y, col0 = blockIdx.z * L::COLS;
  int r, chunk_at, chunk_count;
  if (!find_chunk(p.q_start, p.requests, p.chunk, blockIdx.x, r, chunk_at, chunk_count)) return;
  const bool last_chunk = chunk_at == chunk_count - 1;
  if (!OUT && last_chunk) return;                              // nothing comes after it
  const int slot = p.state_slots[r];
  if (slot < 0 || slot >= p.num_slots) {
    if (tid == 0) atomicOr(p.status, SPROUT_STATUS_BAD_PAGE);
    return;
  }
  const int group = h / (p.heads / p.groups);
  const int first = p.q_start[r] + chunk_at * p.chunk, last = min(p.q_start[r + 1], first + p.chunk);
  float* mine = p.state + ((size_t)slot * p.heads + h) * DIM * p.vdim;
  float* held = p.sums + ((size_t)blockIdx.x * p.heads + h) * DIM * p.vdim;
  const float* from = chunk_count == 1 ? mine : held;
  const int wcol = col0 + warp * WC;                           // the warp's first column

  // S^T: rows are value columns (wcol + 16 m + g, + 8), columns key channels (8 n + c2, + 1)
  float S[MT][2 * KT][4];
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int n = 0; n < 2 * KT; n++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int col = wcol + 16 * m + g + 8 * (e >> 1), d = 8 * n + c2 + (e & 1);
        S[m][n][e] = OUT && col < p.vdim ? from[(size_t)d * p.vdim + col] : 0.f;
      }
  unsigned walked_before = 0;                                  // SUMS: columns that have been walked in turn
  float prod0 = 1.f, prod1 = 1.f;                              // SUMS: the chunk's decays of two channels (threads of the keys)

  auto fetch = [&](int t0, int stage) {
    uint8_t* to = smem + stage * L::STAGE;
    constexpr int PER_ROW = DIM / 8;
#pragma unroll
    for (int i = tid; i < STEP * PER_ROW; i += THREADS) {
      const int t = i / PER_ROW, d = 8 * (i % PER_ROW);
      const bool there = t0 + t < last;
      const size_t row = there ? t0 + t : t0;
      if (OUT) cp_async16_or_zero(to + t * DIM * 2 + d * 2, p.q + row * p.q_stride + (size_t)group * DIM + d, there);
      cp_async16_or_zero(to + L::Q_BYTES + t * DIM * 2 + d * 2, p.k + row * p.k_stride + (size_t)group * DIM + d, there);
    }
    uint8_t* decays = to + 2 * L::Q_BYTES;
    if (PER_HEAD) {
      if (tid < STEP) {
        const bool there = t0 + tid < last;
        ((float*)decays)[tid] = there ? p.da[(size_t)(t0 + tid) * p.heads + h] : 1.f;
        ((float*)decays)[STEP + tid] = there ? p.dc[(size_t)(t0 + tid) * p.heads + h] : 0.f;
      }
    } else {
#pragma unroll
      for (int i = tid; i < STEP * DIM / 4; i += THREADS) {
        const int t = i / (DIM / 4), d = 4 * (i % (DIM / 4));
        const bool there = t0 + t < last;
        cp_async16_or_zero(decays + t * DIM * 4 + d * 4, p.da + ((size_t)(there ? t0 + t : t0) * p.heads + h) * DIM + d, there);
      }
    }
    uint8_t* values = decays + L::DECAY_BYTES;
    constexpr int V_CHUNKS = L::COLS / 8;
#pragma unroll
    for (int i = tid; i < STEP * V_CHUNKS; i += THREADS) {
      const int t = i / V_CHUNKS, c = 8 * (i % V_CHUNKS);
      const bool there = t0 + t < last && col0 + c < p.v_cols;
      uint8_t* dst = values + t * L::V_ROW + c * 2;
      if (p.ones_col && col0 + c == p.v_cols)                  // the column of ones, and nothing beyond it
        *(uint4*)dst = make_uint4(t0 + t < last ? 0x3f80u : 0u, 0u, 0u, 0u);
      else
        cp_async16_or_zero(dst, p.v + (there ? (size_t)(t0 + t) * p.v_stride + (size_t)h * p.v_cols + col0 + c : 0), there);
    }
    cp_async_commit();
  };

  const float skip = OUT && p.skip ? p.skip[h] : 0.f;
  fetch(first, 0);
  for (int t0 = first, stage = 0; t0 < last; t0 += STEP, stage ^= 1) {
    const int n_tokens = min(STEP, last - t0);
    cp_async_wait<0>();
    __syncthreads();                                           // the vectors are there; the step before has read its terms
    if (t0 + STEP < last) fetch(t0 + STEP, stage ^ 1);
    const uint8_t* in = smem + stage * L::STAGE;
    const __nv_bfloat16* q_in = (const __nv_bfloat16*)in;
    const __nv_bfloat16* k_in = (const __nv_bfloat16*)(in + L::Q_BYTES);
    const float* a_in = (const float*)(in + 2 * L::Q_BYTES);
    const uint8_t* v_in = in + 2 * L::Q_BYTES + L::DECAY_BYTES;
    auto two = [](const __nv_bfloat16* at, float& x0, float& x1) {
      const uint32_t raw = *(const uint32_t*)at;
      x0 = __uint_as_float(raw << 16);
      x1 = __uint_as_float(raw & 0xffff0000u);
    };
    auto decay2 = [&](int t, int d, float& a0, float& a1) {    // tokens that do not exist keep everything
      if (PER_HEAD) { a0 = a1 = a_in[t]; return; }
      const float2 a = *(const float2*)(a_in + t * DIM + d);
      a0 = t < n_tokens ? a.x : 1.f;
      a1 = t < n_tokens ? a.y : 1.f;
    };
    bool k_bad = false;                                        // a key's term or a decay that is not finite
    // ---- the terms of k_j P(j, 16) and q_i P(0, i): two channels a thread, half of the threads (a quarter each at 64) for either
    constexpr int HALF = DIM / 2;
    if (tid < HALF) {
      const int d = 2 * tid;
      float s0 = 1.f, s1 = 1.f;
      __nv_bfloat162 most = __floats2bfloat162_rn(0.f, 0.f);   // NaN once a term is not finite
#pragma unroll
      for (int t = STEP - 1; t >= 0; t--) {
        float x0, x1, a0, a1;
        two(k_in + t * DIM + d, x0, x1);
        decay2(t, d, a0, a1);
        const float factor = PER_HEAD ? a_in[STEP + t] : 1.f;
        uint32_t high, mid, low;
        split3(x0 * factor * s0, x1 * factor * s1, high, mid, low);
        most = __hfma2(*(const __nv_bfloat162*)&high, __floats2bfloat162_rn(0.f, 0.f), most);
        uint8_t* to = smem + L::OFF_KS + t * L::ROW + d * 2;
        *(uint32_t*)to = high;
        *(uint32_t*)(to + STEP * L::ROW) = mid;
        *(uint32_t*)(to + 2 * STEP * L::ROW) = low;
        s0 *= a0;
        s1 *= a1;
      }
      k_bad = fmaf(s0, 0.f, fmaf(s1, 0.f, __low2float(most) + __high2float(most))) != 0.f;
      *(float2*)(total + d) = make_float2(s0, s1);
      prod0 *= s0;
      prod1 *= s1;
    } else if (OUT && tid < 2 * HALF) {
      const int d = 2 * (tid - HALF);
      float s0 = p.q_scale, s1 = p.q_scale;
#pragma unroll
      for (int t = 0; t < STEP; t++) {
        float x0, x1, a0, a1;
        two(q_in + t * DIM + d, x0, x1);
        decay2(t, d, a0, a1);
        s0 *= a0;
        s1 *= a1;
        uint32_t high, mid, low;
        split3(x0 * s0, x1 * s1, high, mid, low);
        uint8_t* to = smem + L::OFF_QS + t * L::ROW + d * 2;
        *(uint32_t*)to = high;
        *(uint32_t*)(to + STEP * L::ROW) = mid;
        *(uint32_t*)(to + 2 * STEP * L::ROW) = low;
      }
    }
    // ---- the triangle A: keys j = warp, 7 - warp, 8 + warp, 15 - warp (34 pairs a warp), LANE_DIMS channels a lane
    if (OUT) {
#pragma unroll 1
      for (int u = 0; u < 4; u++) {
        const int j = u == 0 ? warp : u == 1 ? 7 - warp : u == 2 ? 8 + warp : 15 - warp;
        const int d = lane * LANE_DIMS;
        float w[LANE_DIMS], sum[STEP];
#pragma unroll
        for (int e = 0; e < LANE_DIMS; e += 2) two(k_in + j * DIM + d + e, w[e], w[e + 1]);
#pragma unroll
        for (int i = 0; i < STEP; i++) {
          sum[i] = 0.f;
          if (i < j) continue;                                 // the same for the whole warp
          float q[LANE_DIMS];
#pragma unroll
          for (int e = 0; e < LANE_DIMS; e += 2) {
            float a0, a1;
            two(q_in + i * DIM + d + e, q[e], q[e + 1]);
            decay2(i, d + e, a0, a1);
            if (i > j) { w[e] *= a0; w[e + 1] *= a1; }
          }
#pragma unroll
          for (int e = 0; e < LANE_DIMS; e++) sum[i] = fmaf(q[e], w[e], sum[i]);
        }
        // 16 sums over the lanes: halves are exchanged until a lane pair has one of them, row lane / 2
#pragma unroll
        for (int width = 8, mask = 16; width > 0; width >>= 1, mask >>= 1) {
          const bool upper = lane & mask;
#pragma unroll
          for (int i = 0; i < width; i++) {
            const float send = upper ? sum[i] : sum[i + width], keep = upper ? sum[i + width] : sum[i];
            sum[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
          }
        }
        float x = sum[0] + __shfl_xor_sync(0xffffffffu, sum[0], 1);
        x *= p.q_scale * (PER_HEAD ? a_in[STEP + j] : 1.f);
        if ((lane >> 1) == j) x += skip;
        uint32_t high, mid, low;
        split3(x, 0.f, high, mid, low);
        if ((lane & 1) == 0) {
          uint8_t* to = smem + L::OFF_A + (lane >> 1) * L::A_ROW + j * 2;
          *(uint16_t*)to = (uint16_t)high;
          *(uint16_t*)(to + STEP * L::A_ROW) = (uint16_t)mid;
          *(uint16_t*)(to + 2 * STEP * L::A_ROW) = (uint16_t)low;
        }
      }
    }
    k_bad = __syncthreads_or(k_bad);
    // ---- tensor cores
    const uint8_t* own_values = v_in + (warp * WC) * 2;
    uint32_t v[MT][4];                                         // v^T: rows value columns, columns tokens
#pragma unroll
    for (int m = 0; m < MT; m++)
      ldmatrix_x4_trans(v[m], own_values + ((lane & 7) + ((lane >> 4) & 1) * 8) * L::V_ROW + (16 * m + ((lane >> 3) & 1) * 8) * 2);
    // one bit for every column of the thread (16 m + g, + 8), the same in the four lanes that share it: walk this column in turn
    unsigned walked = k_bad ? (1u << 2 * MT) - 1 : 0;
    auto votes = [&](bool yes) { return (__ballot_sync(0xffffffffu, yes) >> (lane & 28) & 15u) != 0; };
    if (!OUT) {                                                // values that are not finite; a column once walked stays so
      uint32_t seen[MT][2], any = 0;
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
          seen[m][half] = ((v[m][half] & 0x7f807f80u) + 0x00800080u) | ((v[m][half + 2] & 0x7f807f80u) + 0x00800080u);
          any |= seen[m][half];
        }
      if (__any_sync(0xffffffffu, any & 0x80008000u)) {
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
          for (int half = 0; half < 2; half++) walked |= (unsigned)votes(seen[m][half] & 0x80008000u) << (2 * m + half);
      }
      walked |= walked_before;
      walked_before = walked;
    }
    // the 16 tokens in turn for the columns in `walked`: the state, and of the outputs those that are not finite
    auto walk = [&](float (&o)[MT][2][4]) {
#pragma unroll 1
      for (int t = 0; t < n_tokens; t++) {
        float value[MT][2], part[MT][2];
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
          for (int half = 0; half < 2; half++) {
            value[m][half] = __bfloat162float(*(const __nv_bfloat16*)(own_values + t * L::V_ROW + (16 * m + 8 * half + g) * 2));
            part[m][half] = 0.f;
          }
        const float factor = PER_HEAD ? a_in[STEP + t] : 1.f;
#pragma unroll
        for (int n = 0; n < 2 * KT; n++) {
          float k[2], a[2], q[2] = {0.f, 0.f};
          two(k_in + t * DIM + 8 * n + c2, k[0], k[1]);
          decay2(t, 8 * n + c2, a[0], a[1]);
          if (OUT) two(q_in + t * DIM + 8 * n + c2, q[0], q[1]);
#pragma unroll
          for (int m = 0; m < MT; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const int half = e >> 1, x = e & 1;
              if (walked >> (2 * m + half) & 1) S[m][n][e] = fmaf(a[x], S[m][n][e], k[x] * factor * value[m][half]);
              if (OUT) part[m][half] = fmaf(p.q_scale * q[x], S[m][n][e], part[m][half]);
            }
        }
        if (OUT) {
#pragma unroll
          for (int m = 0; m < MT; m++)
#pragma unroll
            for (int half = 0; half < 2; half++) {
              float sum = part[m][half] + __shfl_xor_sync(0xffffffffu, part[m][half], 1);
              sum += __shfl_xor_sync(0xffffffffu, sum, 2);
              sum = fmaf(skip, value[m][half], sum);
#pragma unroll
              for (int n = 0; n < 2; n++)
#pragma unroll
                for (int x = 0; x < 2; x++) {
                  float& at = o[m][n][2 * half + x];
                  if (8 * n + c2 + x == t && (walked >> (2 * m + half) & 1) && !isfinite(at)) at = sum;
                }
            }
        }
      }
    };
    const int nt_row = (lane & 7) + ((lane >> 4) & 1) * 8, nt_col = ((lane >> 3) & 1) * 8;
    if (OUT) {
      float o[MT][2][4], small[MT][2][4];                      // o^T: rows value columns, columns tokens (8 n + c2, + 1); the lesser terms' part
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) o[m][n][e] = small[m][n][e] = 0.f;
#pragma unroll
      for (int kt = 0; kt < KT; kt++) {
        uint32_t q[3][4];
#pragma unroll
        for (int x = 0; x < 3; x++) ldmatrix_x4(q[x], smem + L::OFF_QS + (x * STEP + nt_row) * L::ROW + (16 * kt + nt_col) * 2);
#pragma unroll
        for (int m = 0; m < MT; m++) {
          uint32_t s[3][4];
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float* pair = &S[m][2 * kt + (e >> 1)][2 * (e & 1)];
            split3(pair[0], pair[1], s[0][e], s[1][e], s[2][e]);
          }
#pragma unroll
          for (int n = 0; n < 2; n++) {
            float c[4];
            mma_bf16(small[m][n], s[0], q[2][2 * n], q[2][2 * n + 1]);
            mma_bf16(small[m][n], s[2], q[0][2 * n], q[0][2 * n + 1]);
            mma_bf16(small[m][n], s[1], q[1][2 * n], q[1][2 * n + 1]);
            mma_bf16(small[m][n], s[0], q[1][2 * n], q[1][2 * n + 1]);
            mma_bf16(small[m][n], s[1], q[0][2 * n], q[0][2 * n + 1]);
            mma_bf16_first(c, s[0], q[0][2 * n], q[0][2 * n + 1]);
#pragma unroll
            for (int e = 0; e < 4; e++) o[m][n][e] += c[e];
          }
        }
      }
      uint32_t a[3][4];
#pragma unroll
      for (int x = 0; x < 3; x++) ldmatrix_x4(a[x], smem + L::OFF_A + (x * STEP + nt_row) * L::A_ROW + nt_col * 2);
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < 2; n++) {
          float c[4];
          mma_bf16(small[m][n], v[m], a[2][2 * n], a[2][2 * n + 1]);
          mma_bf16(small[m][n], v[m], a[1][2 * n], a[1][2 * n + 1]);
          mma_bf16_first(c, v[m], a[0][2 * n], a[0][2 * n + 1]);
#pragma unroll
          for (int e = 0; e < 4; e++) o[m][n][e] += c[e] + small[m][n][e];
        }
      float probe = 0.f;                                       // NaN if an output is not finite: as all of a column's are if its state or a value is not
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) probe = fmaf(o[m][n][e], 0.f, probe);
      if (__any_sync(0xffffffffu, probe != 0.f)) {
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
          for (int half = 0; half < 2; half++) {
            float of_column = 0.f;
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
              for (int x = 0; x < 2; x++) of_column = fmaf(o[m][n][2 * half + x], 0.f, of_column);
            walked |= (unsigned)votes(of_column != 0.f) << (2 * m + half);
          }
      }
      if (__any_sync(0xffffffffu, walked)) walk(o);
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int col = wcol + 16 * m + g + 8 * (e >> 1), t = 8 * n + c2 + (e & 1);
            if (t < n_tokens && col < p.vdim) p.out[((size_t)(t0 + t) * p.heads + h) * p.vdim + col] = o[m][n][e];
          }
      if (last_chunk ? false : t0 + STEP >= last) break;       // the state after the chunk is the next one's, made by the carry
    } else if (__any_sync(0xffffffffu, walked)) {
      float none[MT][2][4];
      walk(none);
    }
#pragma unroll
    for (int kt = 0; kt < KT; kt++) {
      const float2 d0 = *(const float2*)(total + 16 * kt + c2), d1 = *(const float2*)(total + 16 * kt + 8 + c2);
      uint32_t k[3][4];
#pragma unroll
      for (int x = 0; x < 3; x++) ldmatrix_x4_trans(k[x], smem + L::OFF_KS + (x * STEP + (lane & 15)) * L::ROW + (16 * kt + (lane >> 4) * 8) * 2);
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < 2; n++) {
          float c[4];
          mma_bf16_first(c, v[m], k[2][2 * n], k[2][2 * n + 1]);
          mma_bf16(c, v[m], k[1][2 * n], k[1][2 * n + 1]);
          mma_bf16(c, v[m], k[0][2 * n], k[0][2 * n + 1]);
          const float2 d = n == 0 ? d0 : d1;
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (!(walked >> (2 * m + (e >> 1)) & 1)) S[m][2 * kt + n][e] = fmaf(S[m][2 * kt + n][e], e & 1 ? d.y : d.x, c[e]);
        }
    }
  }
  if (OUT && !last_chunk) return;
  float* to = OUT ? mine : held;
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int n = 0; n < 2 * KT; n++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int col = wcol + 16 * m + g + 8 * (e >> 1), d = 8 * n + c2 + (e & 1);
        if (col < p.vdim) to[(size_t)d * p.vdim + col] = S[m][n][e];
      }
  if (!OUT && blockIdx.z == 0 && tid < DIM / 2)
    *(float2*)(p.prods + ((size_t)blockIdx.x * p.heads + h) * DIM + 2 * tid) = make_float2(prod0, prod1);
}

template <int DIM, int WC, bool PER_HEAD, int PHASE>
int launch_phase(const ScanParams<__nv_bfloat16>& p, int max_chunks, cudaStream_t stream) {
  using L = Shape<DIM, WC, PER_HEAD>;
  auto* kernel = scan_mma_kernel<DIM, WC, PER_HEAD, PHASE>;
  static bool configured = false;
  if (!configured) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
    if (err != cudaSuccess) return sprout_fail("gated_scan: cannot reserve %d bytes of shared memory: %s", L::BYTES, cudaGetErrorString(err));
    configured = true;
  }
  const dim3 grid(max_chunks, p.heads, (p.vdim + L::COLS - 1) / L::COLS);
  SPROUT_REQUIRE(grid.z <= 65535, "gated_scan: too many value columns");
  sprout_launch(kernel, grid, dim3(THREADS), L::BYTES, stream, p);
  return sprout_check_launch(PHASE == SCAN_CHUNK_OUT ? "gated_scan (chunk outputs)" : "gated_scan (chunk sums)");
}

template <int DIM, int WC>
int launch_sizes(const ScanParams<__nv_bfloat16>& p, int phase, int max_chunks, cudaStream_t stream) {
  const bool per_head = p.mode != DECAY_PER_CHANNEL;
  if (phase == SCAN_CHUNK_OUT)
    return per_head ? launch_phase<DIM, WC, true, SCAN_CHUNK_OUT>(p, max_chunks, stream) : launch_phase<DIM, WC, false, SCAN_CHUNK_OUT>(p, max_chunks, stream);
  return per_head ? launch_phase<DIM, WC, true, SCAN_CHUNK_SUMS>(p, max_chunks, stream) : launch_phase<DIM, WC, false, SCAN_CHUNK_SUMS>(p, max_chunks, stream);
}

}  // namespace

namespace sprout_scan {

bool scan_mma_takes(const ScanParams<__nv_bfloat16>& p) {
  auto on16 = [](const void* x) { return ((uintptr_t)x & 15) == 0; };
  return (p.dim == 64 || p.dim == 128) && (p.mode == DECAY_PER_CHANNEL || p.mode == DECAY_PER_HEAD || p.mode == DECAY_GIVEN) && p.sums && p.prods &&
         p.v_cols % 8 == 0 && p.v_stride % 8 == 0 && p.q_stride % 8 == 0 && p.k_stride % 8 == 0 && on16(p.q) && on16(p.k) && on16(p.v) &&
         (p.mode != DECAY_PER_CHANNEL || on16(p.da));
}

int launch_scan_mma(const ScanParams<__nv_bfloat16>& p, int phase, int max_chunks, cudaStream_t stream) {
  const bool narrow = p.vdim <= 64;                            // blocks of 64 value columns, else of 128
  if (p.dim == 64) return narrow ? launch_sizes<64, 16>(p, phase, max_chunks, stream) : launch_sizes<64, 32>(p, phase, max_chunks, stream);
  return narrow ? launch_sizes<128, 16>(p, phase, max_chunks, stream) : launch_sizes<128, 32>(p, phase, max_chunks, stream);
}

}  // namespace sprout_scan
