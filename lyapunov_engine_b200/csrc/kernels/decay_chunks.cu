// Linear recurrences over a matrix of state per head whose decay is one number
// per head and token, over chunks of tokens on the tensor cores: the form of
// the state-space duality (state_space.cu) and of the mLSTM's matrix memory
// (mlstm.cu) for requests that bring several tokens in bfloat16, from each
// request's state row and back into it.  Those files' scans take decoded
// tokens, other types and other sizes; the mathematics and the state's layout
// are theirs.
//
// Per head, with k, q [dim], v [vdim], a decay a_t and a weight w_t per token:
//
//   S <- a_t S + w_t k_t v_t^T                 o_t = S^T q_t
//
// state-space duality: a = exp(-exp(A_log) dt), w = dt, k = B, q = C (shared by
// the heads of a group), v = x; the output is (o + D x) silu(z).
// matrix memory: a = e^(f + m - m'), w = e^(i - m'); n runs along as one more
// column (v = 1), and the output is o / (max(|n . q|, e^(-m')) + 1e-6).
//
// In a chunk of 64 tokens, with L_i the logarithms of its decays summed up to
// token i, and S the state before the chunk:
//
//   o_i = e^(L_i) S^T q_i + sum_{j <= i} e^(L_i - L_j) w_j (q_i . k_j) v_j
//   S  <- e^(L_last) S + sum_j e^(L_last - L_j) w_j k_j v_j^T
//
// k, q and v are exact bfloat16 operands.  The 32-bit numbers that meet them in a
// product (S, the weighted scores, the weighted values) are split into three
// bfloat16 parts that keep all their 24 bits, and every part is multiplied; all
// sums are 32-bit and S is never rounded.  The L are summed in 64 bits and kept as
// two floats, so that differences of them are as good as the decays themselves.
//
// What bounds it, and the layout that follows: token by token (one request, 64 heads of 64 x 128,
// 2,048 tokens) a prompt is 2,048 steps of load, multiply-add, shuffle, each as long as their latencies
// (1,268 us, over chunks 165; the matrix memory of 8 heads of 128 x 256 1,019 us, 126).  A chunk is one step
// instead, and segments of SEGMENT tokens run side by side: every segment's own sum first (SUMS), then the states
// they start from, element by element, then the outputs (35, 11 and 135 us cold; the tensor pipes are busy for a
// third and a fifth of them).  A block is one segment, one head and 64 columns of S; S^T stays in the
// accumulators of its four warps (16 columns each, all of dim), whose layout is that of the left operand of the
// next product, so the state never passes through shared memory.
#include "chunk_mma.cuh"

namespace {

using bf16 = __nv_bfloat16;
using le::add4, le::high_of, le::ldsm4, le::ldsm4_trans, le::low_of, le::mma, le::mma_first, le::mma_split3, le::split_pair3, le::split_state3;

constexpr int CHUNK = 64;
constexpr int SEGMENT = 256;
constexpr int COLS = 64;            // columns of S a block takes
constexpr int THREADS = 128;
constexpr int LDV = COLS + 8;       // rows of v, of the weighted scores (bfloat16) and of outputs (float) in shared
constexpr int LDP = CHUNK + 8;      // memory: padded so that eight rows' 16-byte pieces fall into different banks
constexpr int LDO = COLS + 4;
constexpr float SMALLEST_LOG = -1.0e4f;   // of one token's decay: its exponential is exp_unbiased's smallest, 1.6e-38, and sums stay finite

__device__ __forceinline__ float softplus_f32(float v) { return v > 20.0f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float log_sigmoid_f32(float x) {
  return x >= 0.0f ? -log1pf(expf(-x)) : x - log1pf(expf(x));
}

template <int N> struct Int { static constexpr int value = N; };

struct DecayArgs {
  float *out; int64_t out_stride;
  const bf16 *q, *k, *v; int64_t q_stride, k_stride, v_stride;   // at head 0's entries of token 0
  int heads_per_group;               // heads that share q and k
  float4 *gates; int64_t tokens;     // [heads, tokens]: L (high part, low part), w, e^(-m')
  float *keeps;                      // [segments, heads]: the product of a segment's decays
  float *starts_n;                   // [segments, heads, dim]: n before the request's first token, at its first segment
  float *state; int num_state_rows;
  float *scratch;                    // [segments, heads, vdim (+ 1: n), dim], or null: every request is one segment
  const int32_t *state_slots, *cu_q, *tile_request, *tile_q0;
  int heads, dim, vdim, part_rows;   // part_rows: columns per part of the matrix memory's state layout
  int vector;                        // 16-byte pieces are whole and aligned
  const bf16 *z; int64_t z_stride; const float *d_skip; float out_scale;   // state-space duality
  float q_scale;                                                           // matrix memory
};

// Where column c of a head's S lies in the state (its entries are consecutive).
template <bool MEMORY>
__device__ __forceinline__ int64_t column_at(const DecayArgs &p, int slot, int head, int c) {
  const int64_t h = static_cast<int64_t>(slot) * p.heads + head;
  if constexpr (MEMORY) {
    const int R = p.part_rows;
    return (h * (p.vdim / R) * (R + 2) + (c / R) * (R + 2) + c % R) * p.dim;
  } else {
    return (h * p.vdim + c) * p.dim;
  }
}
// A part's copy of n; m is the first number of the row behind it.
__device__ __forceinline__ int64_t n_at(const DecayArgs &p, int slot, int head, int part) {
  const int R = p.part_rows;
  return ((static_cast<int64_t>(slot) * p.heads + head) * (p.vdim / R) * (R + 2) + part * (R + 2) + R) * p.dim;
}

// L of this thread's token from every token's logarithm: sums over the chunk's 64 tokens (two warps) up to it.
// `totals` [8] of shared memory receives the warps' sums; a block meets once.
__device__ __forceinline__ double chunk_sum(double x, double *totals) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) totals[warp] = x;
  __syncthreads();
  return (warp & 1) ? x + totals[warp - 1] : x;
}
// e^L for a sum in 64 bits: both of its floats count.
__device__ __forceinline__ float exp_of_sum(float high, float low) {
  const float e = le::exp_unbiased(high);
  return fmaf(e, low, e);                                  // (low is no more than a rounding of high)
}
__device__ __forceinline__ float exp_of_sum(double L) {
  const float high = static_cast<float>(L);
  return exp_of_sum(high, static_cast<float>(L - static_cast<double>(high)));
}
__device__ __forceinline__ float4 gate_of(double L, float w, float floor) {
  const float high = static_cast<float>(L);
  return make_float4(high, static_cast<float>(L - static_cast<double>(high)), w, floor);
}

// State-space duality: one block per segment and head, a thread per token.
__global__ void __launch_bounds__(SEGMENT)
duality_gates_kernel(DecayArgs p, const bf16 *dt_rows, int64_t dt_stride, const float *dt_bias, const float *a_log) {
  __shared__ double totals[8];
  le::let_successor_start();
  const int seg = blockIdx.x, head = blockIdx.y;
  const float rate = expf(a_log[head]), bias = dt_bias[head];
  const int b = p.tile_request[seg], q0 = p.tile_q0[seg];
  const int tokens = min(SEGMENT, p.cu_q[b + 1] - p.cu_q[b] - q0);
  const int64_t at = static_cast<int64_t>(p.cu_q[b]) + q0 + threadIdx.x;
  le::wait_for_predecessor();
  float dt = 0.0f, log_decay = 0.0f;
  if (threadIdx.x < tokens) {
    dt = softplus_f32(__bfloat162float(dt_rows[at * dt_stride + head]) + bias);
    log_decay = fmaxf(-dt * rate, SMALLEST_LOG);
  }
  const double L = chunk_sum(static_cast<double>(log_decay), totals);
  if (threadIdx.x < tokens) p.gates[head * p.tokens + at] = gate_of(L, dt, 0.0f);
  if (threadIdx.x == 0) {
    double all = 0.0;
#pragma unroll
    for (int w = 0; w < SEGMENT / 32; ++w) all += totals[w];
    p.keeps[static_cast<int64_t>(seg) * p.heads + head] = exp_of_sum(all);
  }
}

// Matrix memory: one block per request (at its first segment) and head.  The running maximum m' = max(f + m, i) is a
// scan of pairs (sum of f, largest i plus the f behind it); whatever its rounding, the decays and weights are made from
// the m that results, in 64 bits, so S, n and e^(-m') stay in the same units.  It also moves m and keeps a copy of n.
__global__ void __launch_bounds__(SEGMENT)
memory_gates_kernel(DecayArgs p, const bf16 *rows, int64_t row_stride, int i_col, int f_col, const float *i_bias,
                    const float *f_bias, float cap, int num_segments) {
  __shared__ double totals[8];
  __shared__ float s_f[8], s_m[8], s_run;
  le::let_successor_start();
  const int seg = blockIdx.x, head = blockIdx.y;
  if (p.tile_q0[seg] != 0) return;               // (the step's integers are older than the kernel before this one)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = p.tile_request[seg];
  const int64_t first = p.cu_q[b];
  const int q_len = p.cu_q[b + 1] - p.cu_q[b];
  const int slot = p.state_slots[b];
  const bool has_state = slot >= 0 && slot < p.num_state_rows;
  const float bias_i = i_bias[head], bias_f = f_bias[head];
  le::wait_for_predecessor();
  for (int d = tid; d < p.dim; d += SEGMENT)
    p.starts_n[(static_cast<int64_t>(seg) * p.heads + head) * p.dim + d] = has_state ? p.state[n_at(p, slot, head, 0) + d] : 0.0f;
  float run = has_state ? p.state[n_at(p, slot, head, 0) + p.dim] : 0.0f;
  int at = seg;                                   // the request's next segment in the list
  for (int s0 = 0; s0 < q_len; s0 += SEGMENT) {
    const bool live = s0 + tid < q_len;
    float gi = -INFINITY, gf = 0.0f;
    if (live) {
      const bf16 *row = rows + (first + s0 + tid) * row_stride;
      gi = cap * tanhf((__bfloat162float(row[i_col + head]) + bias_i) / cap);
      gf = log_sigmoid_f32(cap * tanhf((__bfloat162float(row[f_col + head]) + bias_f) / cap));
    }
    float F = gf, M = gi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float f = __shfl_up_sync(0xffffffffu, F, o), m = __shfl_up_sync(0xffffffffu, M, o);
      if (lane >= o) M = fmaxf(M, m + F), F += f;
    }
    if (lane == 31) s_f[warp] = F, s_m[warp] = M;
    __syncthreads();
    float before = run;
    for (int w = 0; w < warp; ++w) before = fmaxf(before + s_f[w], s_m[w]);
    const float m_new = fmaxf(before + F, M);
    float m_old = __shfl_up_sync(0xffffffffu, m_new, 1);
    if (lane == 0) m_old = before;
    if (tid == SEGMENT - 1) s_run = m_new;
    const double step = live ? static_cast<double>(gf) + static_cast<double>(m_old) - static_cast<double>(m_new) : 0.0;
    const double L = chunk_sum(step, totals);     // (a meeting: s_run is there behind it)
    if (live) {
      p.gates[head * p.tokens + first + s0 + tid] = gate_of(L, le::exp_unbiased(gi - m_new), le::exp_unbiased(-m_new));
    }
    while (at < num_segments && p.tile_request[at] != b) ++at;
    if (tid == 0 && at < num_segments) {
      double all = 0.0;
#pragma unroll
      for (int w = 0; w < SEGMENT / 32; ++w) all += totals[w];
      p.keeps[static_cast<int64_t>(at) * p.heads + head] = exp_of_sum(all);
    }
    ++at;
    run = s_run;
    __syncthreads();                              // totals, s_f, s_m and s_run are read
  }
  if (has_state)
    for (int part = tid; part < p.vdim / p.part_rows; part += SEGMENT) p.state[n_at(p, slot, head, part) + p.dim] = run;
}

template <int DP, bool SUMS>
constexpr size_t decay_smem() {
  return sizeof(bf16) * ((SUMS ? 1 : 2) * CHUNK * (DP + 8) + CHUNK * LDV + (SUMS ? 0 : 3 * CHUNK * LDP)) +
         sizeof(float) * (10 * CHUNK + 16 + DP);
}

// DP: dim, padded to 64 or 128 (zeros behind the real entries).
template <int DP, bool MEMORY, bool SUMS>
__global__ void __launch_bounds__(THREADS, SUMS ? 4 : 3)
decay_chunk_kernel(DecayArgs p) {
  extern __shared__ __align__(16) unsigned char dc_smem[];
  constexpr int LD = DP + 8, KSTEPS = DP / 16, NT = DP / 8;
  bf16 *s_k = reinterpret_cast<bf16 *>(dc_smem);           // [CHUNK][LD]
  bf16 *s_v = s_k + CHUNK * LD;                            // [CHUNK][LDV]
  bf16 *s_q = s_v + CHUNK * LDV;                           // [CHUNK][LD]
  bf16 *s_p = s_q + (SUMS ? 0 : CHUNK * LD);               // [3][CHUNK][LDP]: weighted scores, high, middle, low parts
  float *s_o = reinterpret_cast<float *>(s_p);             // [CHUNK][LDO]: outputs, once the scores are used
  float *s_hi = reinterpret_cast<float *>(s_p + (SUMS ? 0 : 3 * CHUNK * LDP)), *s_lo = s_hi + CHUNK, *s_w = s_lo + CHUNK;
  float *s_from = s_w + CHUNK, *s_to = s_from + CHUNK;     // e^(L_i), e^(L_last - L_j) w_j
  // Of a pair of tokens in different sixteens the weight is a product: from the key to the end of its sixteen (times the
  // key's w), from there to the start of the query's, from there to the query; none of the three decays is above 1, and
  // none is an exponential per pair.
  float *s_in = s_to + CHUNK, *s_out = s_in + CHUNK, *s_over = s_out + CHUNK;      // s_over [4][4]
  float *s_floor = s_over + 16, *s_row = s_floor + CHUNK, *s_den = s_row + CHUNK;
  float *s_n = s_den + CHUNK;                              // [DP]
  int *s_bad = reinterpret_cast<int *>(s_out);             // [COLS]: the first token with NaN or infinity, once s_out is used
  le::let_successor_start();
  const int slices = (p.vdim + COLS - 1) / COLS;
  const int head = blockIdx.x / slices, e0 = (blockIdx.x % slices) * COLS;
  const int seg = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3, j8 = lane >> 3, r8 = lane & 7;
  const int D = p.dim, cols = min(COLS, p.vdim - e0), group = head / p.heads_per_group;
  const int b = p.tile_request[seg], q0 = p.tile_q0[seg];
  const int tokens = min(SEGMENT, p.cu_q[b + 1] - p.cu_q[b] - q0);
  const int64_t first = static_cast<int64_t>(p.cu_q[b]) + q0;
  const int slot = p.state_slots[b];
  const bool has_state = slot >= 0 && slot < p.num_state_rows;
  const bool mine = 16 * warp < cols;                      // this warp has columns
  const bool with_n = MEMORY && (!SUMS || e0 == 0);
  const int64_t parts = p.vdim + (MEMORY ? 1 : 0);
  float *piece = p.scratch != nullptr ? p.scratch + (static_cast<int64_t>(seg) * p.heads + head) * parts * D : nullptr;
  le::wait_for_predecessor();

  // S^T: tile i holds columns 16 warp + g (entries 0, 1) and + 8 (2, 3) of S, entries 8 i + 2 t4 and the next of dim
  float S[NT][4];
  const int c_row[2] = {16 * warp + g, 16 * warp + g + 8};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float *from = nullptr;
    if (!SUMS && c_row[h] < cols) {
      if (piece != nullptr) from = piece + static_cast<int64_t>(e0 + c_row[h]) * D;
      else if (has_state) from = p.state + column_at<MEMORY>(p, slot, head, e0 + c_row[h]);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int d = 8 * i + 2 * t4;
      S[i][2 * h] = from != nullptr && d < D ? from[d] : 0.0f;
      S[i][2 * h + 1] = from != nullptr && d + 1 < D ? from[d + 1] : 0.0f;
    }
  }
  float n_mine = 0.0f;                                     // entry tid of n
  if (with_n && !SUMS && tid < D)
    n_mine = piece != nullptr ? piece[static_cast<int64_t>(p.vdim) * D + tid]
                              : p.starts_n[(static_cast<int64_t>(seg) * p.heads + head) * D + tid];

  // A chunk's rows of k, q or v into shared memory; rows beyond the tokens and entries beyond the sizes are zeros.
  auto copy_rows = [&](bf16 *dst, auto pieces_of, int ld, const bf16 *src0, int64_t stride, int limit, int c0) {
    constexpr int PIECES = decltype(pieces_of)::value, STEP = THREADS / PIECES;
    const int at = (tid % PIECES) * 8, t0 = tid / PIECES;
    const bf16 *src = src0 + (first + c0 + t0) * stride + at;
    bf16 *to = dst + t0 * ld + at;
    const int rows = at < limit ? tokens - c0 - t0 : 0;    // of those this thread copies a row each STEP
    if (p.vector) {
#pragma unroll
      for (int i = 0; i < CHUNK / STEP; ++i) le::copy16_async(to + i * STEP * ld, i * STEP < rows ? src + i * STEP * stride : src0, i * STEP < rows);
    } else {
      for (int i = 0; i < CHUNK / STEP; ++i)
#pragma unroll
        for (int u = 0; u < 8; ++u)
          to[i * STEP * ld + u] = i * STEP < rows && at + u < limit ? src[i * STEP * stride + u] : __float2bfloat16_rn(0.0f);
    }
  };
  const bf16 *k0 = p.k + group * D, *q_rows = p.q + group * D, *v0 = p.v + static_cast<int64_t>(head) * p.vdim + e0;
  auto fetch_k = [&](int c0) { copy_rows(s_k, Int<DP / 8>(), LD, k0, p.k_stride, D, c0); };
  auto fetch_q = [&](int c0) { copy_rows(s_q, Int<DP / 8>(), LD, q_rows, p.q_stride, D, c0); };
  auto fetch_v = [&](int c0) { copy_rows(s_v, Int<COLS / 8>(), LDV, v0, p.v_stride, cols, c0); };
  fetch_k(0);
  if constexpr (!SUMS) fetch_q(0);
  fetch_v(0);
  le::commit_copies();
  const float skip = !MEMORY && !SUMS && p.d_skip != nullptr ? p.d_skip[head] : 0.0f;

  for (int c0 = 0; c0 < tokens; c0 += CHUNK) {
    const int len = min(CHUNK, tokens - c0);
    const float4 *gates = p.gates + head * p.tokens + first + c0;
    const float4 last = gates[len - 1];
    const float keep = exp_of_sum(last.x, last.y);
    if (tid < CHUNK) {
      const float4 gate = tid < len ? gates[tid] : make_float4(last.x, last.y, 0.0f, 1.0f);
      s_hi[tid] = gate.x, s_lo[tid] = gate.y, s_w[tid] = gate.z;
      s_to[tid] = le::exp_unbiased((last.x - gate.x) + (last.y - gate.y)) * gate.z;
      if constexpr (!SUMS) {
        s_floor[tid] = gate.w;
        s_from[tid] = exp_of_sum(gate.x, gate.y);
        const int before = (tid & ~15) - 1;                // the last token before this sixteen, the last one of it
        const float4 start = before < 0 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : gates[min(before, len - 1)];
        const float4 end = gates[min(tid | 15, len - 1)];
        s_in[tid] = le::exp_unbiased((gate.x - start.x) + (gate.y - start.y));
        s_out[tid] = le::exp_unbiased((end.x - gate.x) + (end.y - gate.y)) * gate.z;
      }
    } else if (!SUMS && tid < CHUNK + 16) {
      const int ib = (tid >> 2) & 3, kb = tid & 3;
      float over = 0.0f;
      if (kb < ib) {
        const float4 start = gates[min(16 * ib - 1, len - 1)], end = gates[min(16 * kb + 15, len - 1)];
        over = le::exp_unbiased((start.x - end.x) + (start.y - end.y));
      }
      s_over[tid - CHUNK] = over;
    }
    if (with_n && tid < DP) s_n[tid] = n_mine;
    le::wait_for_copies();
    __syncthreads();

    float o[CHUNK / 8][4];
    float nq = 0.0f;
    if constexpr (!SUMS) {
#pragma unroll
      for (int i = 0; i < CHUNK / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
      // this warp's 16 tokens' scores with the keys up to them, weighted and split, for all warps
      {
        const int i0 = 16 * warp, row[2] = {i0 + g, i0 + g + 8};
        float sum[2] = {0.0f, 0.0f};
        uint32_t qf[KSTEPS][4];
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) ldsm4(qf[ks], s_q + (i0 + (j8 & 1) * 8 + r8) * LD + ks * 16 + (j8 >> 1) * 8);
        for (int kb = 0; kb <= i0; kb += 16) {
          float s[2][4] = {};
#pragma unroll
          for (int ks = 0; ks < KSTEPS; ++ks) {
            uint32_t kf[4];
            ldsm4(kf, s_k + (kb + (j8 >> 1) * 8 + r8) * LD + ks * 16 + (j8 & 1) * 8);
            float x[2][4];
            mma_first(x[0], qf[ks], kf[0], kf[1]);
            mma_first(x[1], qf[ks], kf[2], kf[3]);
            add4(s[0], x[0]);
            add4(s[1], x[1]);
          }
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const int j = kb + nt * 8 + 2 * t4;
            if (kb < i0) {
              const float over = s_over[warp * 4 + kb / 16];
              const float2 out_j = *reinterpret_cast<const float2 *>(s_out + j);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float in = s_in[row[h]] * over;
                s[nt][2 * h] *= in * out_j.x, s[nt][2 * h + 1] *= in * out_j.y;
              }
            } else {
              const float2 hj = *reinterpret_cast<const float2 *>(s_hi + j), lj = *reinterpret_cast<const float2 *>(s_lo + j);
              const float2 wj = *reinterpret_cast<const float2 *>(s_w + j);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float x = le::exp_unbiased((s_hi[row[h]] - hj.x) + (s_lo[row[h]] - lj.x)) * wj.x;
                const float y = le::exp_unbiased((s_hi[row[h]] - hj.y) + (s_lo[row[h]] - lj.y)) * wj.y;
                // (the query's own key: D x, where there is one, joins it)
                s[nt][2 * h] = j < row[h] ? s[nt][2 * h] * x : j == row[h] ? fmaf(s[nt][2 * h], wj.x, skip) : 0.0f;
                s[nt][2 * h + 1] = j + 1 < row[h] ? s[nt][2 * h + 1] * y : j + 1 == row[h] ? fmaf(s[nt][2 * h + 1], wj.y, skip) : 0.0f;
              }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if constexpr (MEMORY) sum[h] += s[nt][2 * h] + s[nt][2 * h + 1];
              uint32_t part[3];
              split_pair3(s[nt][2 * h], s[nt][2 * h + 1], part[0], part[1], part[2]);
#pragma unroll
              for (int u = 0; u < 3; ++u) *reinterpret_cast<uint32_t *>(s_p + u * CHUNK * LDP + row[h] * LDP + j) = part[u];
            }
          }
        }
        if constexpr (MEMORY) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
            sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
            if (t4 == 0) s_row[row[h]] = sum[h];
          }
        }
      }
      // what the state before the chunk gives
      if (mine) {
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
          uint32_t a[3][4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            split_state3(S[2 * ks + (u >> 1)][2 * (u & 1)], S[2 * ks + (u >> 1)][2 * (u & 1) + 1], a[0][u], a[1][u], a[2][u]);
#pragma unroll
          for (int tb = 0; tb < CHUNK / 16; ++tb) {
            uint32_t qb[4];
            ldsm4(qb, s_q + (tb * 16 + (j8 >> 1) * 8 + r8) * LD + ks * 16 + (j8 & 1) * 8);
            mma_split3(o[2 * tb], a, qb[0], qb[1]);
            mma_split3(o[2 * tb + 1], a, qb[2], qb[3]);
          }
        }
#pragma unroll
        for (int i = 0; i < CHUNK / 8; ++i) {
          const float2 f = *reinterpret_cast<const float2 *>(s_from + 8 * i + 2 * t4);
          o[i][0] *= f.x, o[i][1] *= f.y, o[i][2] *= f.x, o[i][3] *= f.y;
        }
      }
      if constexpr (MEMORY) {                              // n before the chunk times q, two threads a token
        const uint32_t *q_row = reinterpret_cast<const uint32_t *>(s_q + (tid >> 1) * LD);
#pragma unroll 8
        for (int i = tid & 1; i < DP / 2; i += 2) {
          const uint32_t q2 = q_row[i];
          nq = fmaf(s_n[2 * i], low_of(q2), fmaf(s_n[2 * i + 1], high_of(q2), nq));
        }
        nq += __shfl_xor_sync(0xffffffffu, nq, 1);
      }
    }
    // the state behind the chunk (tokens beyond it have weight zero)
    uint32_t odd = 0;                                      // a NaN or an infinity among this warp's values
    if (mine) {
#pragma unroll
      for (int i = 0; i < NT; ++i) S[i][0] *= keep, S[i][1] *= keep, S[i][2] *= keep, S[i][3] *= keep;
#pragma unroll
      for (int kb = 0; kb < CHUNK / 16; ++kb) {
        if (kb * 16 >= len) break;
        const float2 f0 = *reinterpret_cast<const float2 *>(s_to + kb * 16 + 2 * t4);
        const float2 f1 = *reinterpret_cast<const float2 *>(s_to + kb * 16 + 2 * t4 + 8);
        uint32_t va[4], a[3][4];
        ldsm4_trans(va, s_v + (kb * 16 + (j8 >> 1) * 8 + r8) * LDV + 16 * warp + (j8 & 1) * 8);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 f = u < 2 ? f0 : f1;
          odd |= (va[u] & 0x7f807f80u) + 0x00800080u;      // (bits 15 and 31: all bits of an exponent)
          split_pair3(low_of(va[u]) * f.x, high_of(va[u]) * f.y, a[0][u], a[1][u], a[2][u]);
        }
#pragma unroll
        for (int db = 0; db < NT / 2; ++db) {
          uint32_t kf[4];
          ldsm4_trans(kf, s_k + (kb * 16 + (j8 & 1) * 8 + r8) * LD + db * 16 + (j8 >> 1) * 8);
          mma_split3(S[2 * db], a, kf[0], kf[1]);
          mma_split3(S[2 * db + 1], a, kf[2], kf[3]);
        }
      }
    }
    if (with_n && tid < DP) {
      n_mine *= keep;
#pragma unroll 8
      for (int t = 0; t < CHUNK; ++t) n_mine = fmaf(s_to[t], __bfloat162float(s_k[t * LD + tid]), n_mine);
    }
    bool poisoned = false;
    if constexpr (SUMS) __syncthreads();                   // k is used
    else poisoned = __syncthreads_or((odd & 0x80008000u) != 0);   // the weighted scores are there; k and q are used
    if (c0 + CHUNK < tokens) {
      fetch_k(c0 + CHUNK);
      if constexpr (!SUMS) fetch_q(c0 + CHUNK);
    }
    if constexpr (!SUMS) {
      if constexpr (MEMORY) {
        if ((tid & 1) == 0) {
          const int t = tid >> 1;
          s_den[t] = fmaxf(fabsf(p.q_scale * fmaf(s_from[t], nq, s_row[t])), s_floor[t]) + 1e-6f;
        }
      }
      // The weights of keys behind a query are zeros, and zero times NaN or infinity would reach back in time: such
      // values leave the product, and their columns are NaN from the first of them on.
      if (poisoned) {
        if (tid < COLS) {
          int from = CHUNK;
          for (int t = CHUNK - 1; t >= 0; --t) {
            bf16 &v = s_v[t * LDV + tid];
            if (!(fabsf(__bfloat162float(v)) < INFINITY)) from = t, v = __float2bfloat16_rn(0.0f);
          }
          s_bad[tid] = from;
        }
        __syncthreads();
      }
      if (mine) {
#pragma unroll
        for (int kb = 0; kb < CHUNK / 16; ++kb) {
          uint32_t va[4];
          ldsm4_trans(va, s_v + (kb * 16 + (j8 >> 1) * 8 + r8) * LDV + 16 * warp + (j8 & 1) * 8);
#pragma unroll
          for (int ib = kb; ib < CHUNK / 16; ++ib) {
            float x[2][4];
#pragma unroll
            for (int u = 2; u >= 0; --u) {
              uint32_t pb[4];
              ldsm4(pb, s_p + u * CHUNK * LDP + (ib * 16 + (j8 >> 1) * 8 + r8) * LDP + kb * 16 + (j8 & 1) * 8);
              if (u == 2) {
                mma_first(x[0], va, pb[0], pb[1]);
                mma_first(x[1], va, pb[2], pb[3]);
              } else {
                mma(x[0], va, pb[0], pb[1]);
                mma(x[1], va, pb[2], pb[3]);
              }
            }
            add4(o[2 * ib], x[0]);
            add4(o[2 * ib + 1], x[1]);
          }
        }
      }
      __syncthreads();                                     // the weighted scores and v are used
      if (c0 + CHUNK < tokens) fetch_v(c0 + CHUNK);
      if (mine) {
#pragma unroll
        for (int i = 0; i < CHUNK / 8; ++i) {
          const int t = 8 * i + 2 * t4;
          s_o[t * LDO + c_row[0]] = o[i][0], s_o[(t + 1) * LDO + c_row[0]] = o[i][1];
          s_o[t * LDO + c_row[1]] = o[i][2], s_o[(t + 1) * LDO + c_row[1]] = o[i][3];
        }
      }
    }

    if constexpr (!SUMS) {
      const int c = (tid % (COLS / 4)) * 4, t0 = tid / (COLS / 4);
      constexpr int STEP = THREADS / (COLS / 4), N_OUT = CHUNK / STEP;
      uint2 z4[N_OUT];
      const bf16 *z = nullptr;
      if constexpr (!MEMORY) {                             // (the gates are asked for before the block meets)
        if (p.z != nullptr) z = p.z + (first + c0 + t0) * p.z_stride + static_cast<int64_t>(head) * p.vdim + e0 + c;
#pragma unroll
        for (int i = 0; i < N_OUT; ++i) {
          z4[i] = make_uint2(0u, 0u);
          if (z != nullptr && p.vector && t0 + i * STEP < len && c < cols) z4[i] = *reinterpret_cast<const uint2 *>(z + i * STEP * p.z_stride);
        }
      }
      __syncthreads();                                     // the outputs are in shared memory
      float *dst = p.out + (first + c0 + t0) * p.out_stride + static_cast<int64_t>(head) * p.vdim + e0 + c;
#pragma unroll
      for (int i = 0; i < N_OUT; ++i) {
        const int t = t0 + i * STEP;
        if (t >= len || c >= cols) break;
        const float4 o4 = *reinterpret_cast<const float4 *>(s_o + t * LDO + c);
        float y[4] = {o4.x, o4.y, o4.z, o4.w};
        if (poisoned) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (t >= s_bad[c + u]) y[u] = NAN;
        }
        if constexpr (MEMORY) {
          const float den = s_den[t];
#pragma unroll
          for (int u = 0; u < 4; ++u) y[u] = y[u] * p.q_scale / den;
        } else {
          if (z != nullptr) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const uint32_t pair = u < 2 ? z4[i].x : z4[i].y;
              const float gate = p.vector ? ((u & 1) ? high_of(pair) : low_of(pair))
                                          : c + u < cols ? __bfloat162float(z[i * STEP * p.z_stride + u]) : 0.0f;
              y[u] *= gate / (1.0f + expf(-gate));
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) y[u] *= p.out_scale;
        }
        if (!has_state) y[0] = y[1] = y[2] = y[3] = 0.0f;
        float *to = dst + i * STEP * p.out_stride;
        if (p.vector) {
          *reinterpret_cast<float4 *>(to) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c + u < cols) to[u] = y[u];
        }
      }
    }
    if constexpr (SUMS) {
      if (c0 + CHUNK < tokens) fetch_v(c0 + CHUNK);
    }
    le::commit_copies();
    __syncthreads();                                       // everyone is done with this chunk
  }

  if (!SUMS && (piece != nullptr || !has_state)) return;   // (the starting states' kernel has moved the state row)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (c_row[h] >= cols) continue;
    float *to = SUMS ? piece + static_cast<int64_t>(e0 + c_row[h]) * D : p.state + column_at<MEMORY>(p, slot, head, e0 + c_row[h]);
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int d = 8 * i + 2 * t4;
      if (d < D) to[d] = S[i][2 * h];
      if (d + 1 < D) to[d + 1] = S[i][2 * h + 1];
    }
  }
  if (with_n && tid < D) {
    if (SUMS) {
      piece[static_cast<int64_t>(p.vdim) * D + tid] = n_mine;
    } else if (e0 == 0) {                                  // (no block reads n from the state row)
      for (int part = 0; part < p.vdim / p.part_rows; ++part) p.state[n_at(p, slot, head, part) + tid] = n_mine;
    }
  }
}

// From every segment's own sum: the state each segment starts from (in place of the sums) and the request's new state
// row.  A request's segments stand in the list in their order, other requests' between them; the blocks of its first one
// do its work, a thread for V neighbouring entries of a column of S (or of n; V = 4 where the columns are whole pieces),
// with the sums of eight segments asked for at a time.
constexpr int AHEAD = 8;
template <bool MEMORY, int V>
__global__ void __launch_bounds__(256)
decay_starts_kernel(DecayArgs p, int num_segments) {
  le::let_successor_start();
  const int seg = blockIdx.z, head = blockIdx.y;
  const int n = (p.vdim + (MEMORY ? 1 : 0)) * p.dim;
  const int i = (blockIdx.x * 256 + threadIdx.x) * V;
  if (p.tile_q0[seg] != 0 || i >= n) return;
  const int b = p.tile_request[seg];
  const int segments = (p.cu_q[b + 1] - p.cu_q[b] + SEGMENT - 1) / SEGMENT;
  const int slot = p.state_slots[b];
  const bool has_state = slot >= 0 && slot < p.num_state_rows;
  const int c = i / p.dim, d = i - c * p.dim;
  const bool is_n = MEMORY && c == p.vdim;
  float *part = p.scratch + static_cast<int64_t>(head) * n + i;       // of segment s of the list: + s * step
  const int64_t step = static_cast<int64_t>(p.heads) * n;
  auto load = [](float (&v)[V], const float *at) {
    if constexpr (V == 4) {
      const float4 r = *reinterpret_cast<const float4 *>(at);
      v[0] = r.x, v[1] = r.y, v[2] = r.z, v[3] = r.w;
    } else {
      v[0] = *at;
    }
  };
  auto store = [](float *at, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4 *>(at) = make_float4(v[0], v[1], v[2], v[3]);
    else *at = v[0];
  };
  le::wait_for_predecessor();
  float S[V] = {};
  if (is_n) load(S, p.starts_n + (static_cast<int64_t>(seg) * p.heads + head) * p.dim + d);
  else if (has_state) load(S, p.state + column_at<MEMORY>(p, slot, head, c) + d);
  int at = seg;                                   // the request's next segment in the list
  for (int s0 = 0; s0 < segments; s0 += AHEAD) {
    float sum[AHEAD][V], keep[AHEAD];
    int where[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      while (at < num_segments && p.tile_request[at] != b) ++at;
      where[u] = s0 + u < segments && at < num_segments ? at++ : -1;
      if (where[u] >= 0) {
        load(sum[u], part + where[u] * step);
        keep[u] = p.keeps[static_cast<int64_t>(where[u]) * p.heads + head];
      }
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (where[u] < 0) break;
      store(part + where[u] * step, S);
#pragma unroll
      for (int v = 0; v < V; ++v) S[v] = fmaf(keep[u], S[v], sum[u][v]);
    }
  }
  if (!has_state) return;
  if (is_n) {
    for (int q = 0; q < p.vdim / p.part_rows; ++q) store(p.state + n_at(p, slot, head, q) + d, S);
  } else {
    store(p.state + column_at<MEMORY>(p, slot, head, c) + d, S);
  }
}

bool aligned(const void *p, size_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

template <int DP, bool MEMORY, bool SUMS>
int launch_chunks(const DecayArgs &p, int segments, cudaStream_t stream) {
  constexpr size_t smem = decay_smem<DP, SUMS>();
  auto kernel = decay_chunk_kernel<DP, MEMORY, SUMS>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return le::invalid("le_decay_chunks: cannot get %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  }
  const dim3 grid(p.heads * ((p.vdim + COLS - 1) / COLS), segments);
  return le::launch_chained(kernel, grid, dim3(THREADS), smem, stream, p);
}

template <int DP, bool MEMORY>
int run_chunks(const DecayArgs &p, int segments, cudaStream_t stream) {
  if (p.scratch != nullptr) {
    int rc = launch_chunks<DP, MEMORY, true>(p, segments, stream);
    if (rc != 0) return rc;
    const bool quads = p.dim % 4 == 0 && aligned(p.scratch, 16) && aligned(p.state, 16) && aligned(p.starts_n, 16);
    const dim3 grid(((p.vdim + (MEMORY ? 1 : 0)) * p.dim / (quads ? 4 : 1) + 255) / 256, p.heads, segments);
    rc = quads ? le::launch_chained(decay_starts_kernel<MEMORY, 4>, grid, dim3(256), 0, stream, p, segments)
               : le::launch_chained(decay_starts_kernel<MEMORY, 1>, grid, dim3(256), 0, stream, p, segments);
    if (rc != 0) return rc;
  }
  return launch_chunks<DP, MEMORY, false>(p, segments, stream);
}

}  // namespace

LE_API int le_decay_segment() { return SEGMENT; }

// State-space duality over chunks: le_ssm_scan's form with one decay per head, for bfloat16 rows, float32 outputs and
// at most 128 numbers of state per channel.  tile_request / tile_q0 list num_segments segments of le_decay_segment()
// tokens: their requests and their first tokens within them, a request's segments in their order.  work: 4 heads
// num_tokens + num_segments heads (1 + n_state) floats, 16-byte aligned.  scratch: float32 [num_segments, rows, n_state] where a request has several segments, else null.
LE_API int le_duality_chunks(float *out, int64_t out_stride, const void *x, int64_t x_stride, const void *bc, int64_t bc_stride,
                             int b_col, int c_col, const void *dt, int64_t dt_stride, const void *z, int64_t z_stride,
                             const float *dt_bias, const float *a_log, const float *d_skip, float *state, int num_state_rows,
                             const int32_t *state_slots, const int32_t *cu_q, const int32_t *tile_request,
                             const int32_t *tile_q0, int num_segments, int num_tokens, int heads, int vdim, int n_state,
                             int heads_per_group, float out_scale, float *work, float *scratch, cudaStream_t stream) {
  if (num_segments <= 0) return 0;
  if (heads < 1 || heads > 65535 || n_state < 1 || n_state > 128 || vdim < 1 || heads_per_group < 1 || num_segments > 65535)
    return le::invalid("le_duality_chunks: %d heads of %d x %d in %d segments", heads, vdim, n_state, num_segments);
  if (!aligned(work, 16)) return le::invalid("le_duality_chunks: work has to start on 16 bytes");
  DecayArgs p = {};
  p.out = out, p.out_stride = out_stride;
  p.q = static_cast<const bf16 *>(bc) + c_col, p.k = static_cast<const bf16 *>(bc) + b_col, p.v = static_cast<const bf16 *>(x);
  p.q_stride = p.k_stride = bc_stride, p.v_stride = x_stride, p.heads_per_group = heads_per_group;
  p.gates = reinterpret_cast<float4 *>(work), p.tokens = num_tokens;
  p.keeps = work + 4 * static_cast<int64_t>(heads) * num_tokens;
  p.state = state, p.num_state_rows = num_state_rows, p.scratch = scratch;
  p.state_slots = state_slots, p.cu_q = cu_q, p.tile_request = tile_request, p.tile_q0 = tile_q0;
  p.heads = heads, p.dim = n_state, p.vdim = vdim, p.part_rows = 1;
  p.z = static_cast<const bf16 *>(z), p.z_stride = z_stride, p.d_skip = d_skip, p.out_scale = out_scale;
  p.vector = n_state % 8 == 0 && vdim % 8 == 0 && bc_stride % 8 == 0 && x_stride % 8 == 0 && aligned(p.q, 16) && aligned(p.k, 16) &&
             aligned(p.v, 16) && (z == nullptr || (z_stride % 4 == 0 && aligned(z, 8))) && out_stride % 4 == 0 && aligned(out, 16);
  int rc = le::launch_chained(duality_gates_kernel, dim3(num_segments, heads), dim3(SEGMENT), 0, stream, p,
                              static_cast<const bf16 *>(dt), dt_stride, dt_bias, a_log);
  if (rc != 0) return rc;
  return n_state <= 64 ? run_chunks<64, false>(p, num_segments, stream) : run_chunks<128, false>(p, num_segments, stream);
}

// The matrix memory over chunks: le_mlstm_scan for bfloat16 rows and heads of at most 128 entries.  part_rows:
// le_mlstm_rows(dim, vdim).  The lists and work (dim for n_state) as above; scratch: float32 [num_segments, heads, vdim + 1, dim].
LE_API int le_memory_chunks(float *out, int64_t out_stride, const void *rows, int64_t row_stride, int q_col, int k_col, int v_col,
                            int i_col, int f_col, const float *i_bias, const float *f_bias, float *state, int num_state_rows,
                            const int32_t *state_slots, const int32_t *cu_q, const int32_t *tile_request,
                            const int32_t *tile_q0, int num_segments, int num_tokens, int heads, int dim, int vdim,
                            int part_rows, float cap, float q_scale, float *work, float *scratch, cudaStream_t stream) {
  if (num_segments <= 0) return 0;
  if (heads < 1 || heads > 65535 || dim < 1 || dim > 128 || vdim < 1 || num_segments > 65535 || part_rows < 1 || vdim % part_rows)
    return le::invalid("le_memory_chunks: %d heads of %d x %d in %d segments", heads, dim, vdim, num_segments);
  if (!aligned(work, 16)) return le::invalid("le_memory_chunks: work has to start on 16 bytes");
  if (!(cap > 0.0f)) return le::invalid("le_memory_chunks: the gates' cap must be positive");
  DecayArgs p = {};
  const bf16 *base = static_cast<const bf16 *>(rows);
  p.out = out, p.out_stride = out_stride, p.q = base + q_col, p.k = base + k_col, p.v = base + v_col;
  p.q_stride = p.k_stride = p.v_stride = row_stride, p.heads_per_group = 1;
  p.gates = reinterpret_cast<float4 *>(work), p.tokens = num_tokens;
  p.keeps = work + 4 * static_cast<int64_t>(heads) * num_tokens, p.starts_n = p.keeps + static_cast<int64_t>(num_segments) * heads;
  p.state = state, p.num_state_rows = num_state_rows, p.scratch = scratch;
  p.state_slots = state_slots, p.cu_q = cu_q, p.tile_request = tile_request, p.tile_q0 = tile_q0;
  p.heads = heads, p.dim = dim, p.vdim = vdim, p.part_rows = part_rows, p.q_scale = q_scale, p.out_scale = 1.0f;
  p.vector = dim % 8 == 0 && vdim % 8 == 0 && row_stride % 8 == 0 && aligned(p.q, 16) && aligned(p.k, 16) && aligned(p.v, 16) &&
             out_stride % 4 == 0 && aligned(out, 16);
  int rc = le::launch_chained(memory_gates_kernel, dim3(num_segments, heads), dim3(SEGMENT), 0, stream, p, base, row_stride, i_col,
                              f_col, i_bias, f_bias, cap, num_segments);
  if (rc != 0) return rc;
  return dim <= 64 ? run_chunks<64, true>(p, num_segments, stream) : run_chunks<128, true>(p, num_segments, stream);
}
