// The gated delta rule: a linear recurrence over a matrix of state per head.
//
// Per head, with S the state [dim, vdim] (32-bit, carried from token to token
// for each request), k and q unit vectors of the head's key group (q also
// times dim^-1/2), v the head's values, and two numbers per token,
//   g    = exp(-exp(A_log) * softplus(a + dt_bias))     the decay, in (0, 1)
//   beta = sigmoid(b)                                   the step size,
// a token does, in this order,
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q.
// Every column of S (one entry of v, u and o) goes its own way: column j needs
// k, q, g, beta and v_j only.  With S0 the state before the token,
//   u_j = beta (v_j - g (S0[:, j] . k)),   o_j = g (S0[:, j] . q) + (k . q) u_j,
// so both dot products run over the old column, and the column is then
// brought up to date with one multiply-add per entry.
//
// gated_delta_prepare_kernel: what a token brings to the recurrence besides
// its vectors, made once for all columns: per key group the inverse lengths of
// k and q (q's times the query scale) and the unit vectors' product k . q, per
// head the decay and the step size; five 32-bit numbers a (token, head) in a
// row of 4 * groups + 2 * heads floats per token.
//
// gated_delta_scan_kernel: a block takes one request, one head and a slice of
// columns; a column belongs to LANES neighbouring lanes, each holding ROWS of
// its entries in registers, four at a time with LANES groups of four between
// them (LANES * ROWS >= dim; partial dot products meet by shuffles).  The
// request's tokens of the step are walked in order, in tiles of up to
// SCAN_MAX_TILE tokens held twice in shared memory: while the threads that
// hold the state run one tile, four more warps fetch the next one and make of
// it what the recurrence reads: k and q as 32-bit unit vectors (the projected
// entries times the token's inverse lengths), the column slice of v, and k . q,
// decay and step size.  So a token costs a holder two dot products over its
// rows, the shuffles, and one multiply-add and one multiply per entry.  The
// state is kept transposed, [vdim, dim] per head, so that a column is
// consecutive; it is read before the first token and written after the last.
// Rows that stand for no request (slot < 0) give zeros and keep nothing.  In a
// step of single tokens the block has no fetching warps.
//
// gated_delta_groups_kernel: the form for prompts in bfloat16 (see there).
//
// head_norm_gate_kernel: o of every (token, head) is divided by its root mean
// square over vdim, times a weight ([vdim], the same for every head, or [heads,
// vdim]), times silu(gate) or sigmoid(gate), times one number.
//
// Everything here is 32-bit except the inputs (projections and convolution
// outputs in the activations' type) and the gated result, which is rounded once.
#include <cstdlib>

#include "common.cuh"

namespace {

constexpr int SCAN_HOLDERS = 128;     // threads that hold state
constexpr int SCAN_FETCHERS = 128;    // threads that fetch the next tile
constexpr int SCAN_THREADS = SCAN_HOLDERS + SCAN_FETCHERS;
constexpr int SCAN_MAX_TILE = 32;
constexpr int SCAN_BATCH = 4;         // pieces a fetching thread has in flight
constexpr int SCAN_NUMBERS = 4;       // floats a token has in shared memory: k . q, decay, step size, -
constexpr int PREP_THREADS = 128;
constexpr int GROUP_PRODUCTS = 8;     // per token and key group: k . k of 1..3 tokens back, q . k of 0..3 back, -

__device__ __forceinline__ float softplus_f32(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float sigmoid_f32(float x) { return 1.0f / (1.0f + expf(-x)); }

template <typename T>
__global__ void __launch_bounds__(PREP_THREADS)
gated_delta_prepare_kernel(float *__restrict__ prep, int prep_stride, const T *__restrict__ qkv, int64_t qkv_stride, int q_col,
                           int k_col, const T *__restrict__ proj, int64_t proj_stride, int b_col, int a_col,
                           const float *__restrict__ a_log, const float *__restrict__ dt_bias, int heads, int kv_heads,
                           int dim, float unit_eps, float q_scale, int products) {
  le::let_successor_start();
  le::wait_for_predecessor();
  const int64_t t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = PREP_THREADS / 32;
  float *dst = prep + t * prep_stride;
  for (int g = blockIdx.y * warps + warp; g < kv_heads; g += gridDim.y * warps) {
    const T *kr = qkv + t * qkv_stride + k_col + g * dim;
    const T *qr = qkv + t * qkv_stride + q_col + g * dim;
    float kk = 0.0f, qq = 0.0f, kq = 0.0f;
    // products: with the keys of up to three tokens before (of whatever request: a group of tokens reads its own only)
    float nn[3] = {0.0f, 0.0f, 0.0f}, kb[3] = {0.0f, 0.0f, 0.0f}, qb[3] = {0.0f, 0.0f, 0.0f};
    for (int i = lane; i < dim; i += 32) {
      const float a = le::to_f32(kr[i]), c = le::to_f32(qr[i]);
      kk = fmaf(a, a, kk);
      qq = fmaf(c, c, qq);
      kq = fmaf(a, c, kq);
      if (products) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float e = t > d ? le::to_f32(kr[i - (d + 1) * qkv_stride]) : 0.0f;
          nn[d] = fmaf(e, e, nn[d]);
          kb[d] = fmaf(a, e, kb[d]);
          qb[d] = fmaf(c, e, qb[d]);
        }
      }
    }
    kk = le::warp_sum(kk);
    qq = le::warp_sum(qq);
    kq = le::warp_sum(kq);
    if (lane == 0) {
      const float k_inv = rsqrtf(kk + unit_eps), q_inv = rsqrtf(qq + unit_eps) * q_scale;
      dst[4 * g + 0] = k_inv;
      dst[4 * g + 1] = q_inv;
      dst[4 * g + 2] = kq * k_inv * q_inv;
      dst[4 * g + 3] = 0.0f;
    }
    if (products) {
      const float k_inv = rsqrtf(kk + unit_eps), q_inv = rsqrtf(qq + unit_eps) * q_scale;
      float *more = dst + 4 * kv_heads + 2 * heads + GROUP_PRODUCTS * g;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float e_inv = rsqrtf(le::warp_sum(nn[d]) + unit_eps);
        const float kx = le::warp_sum(kb[d]) * k_inv * e_inv, qx = le::warp_sum(qb[d]) * e_inv * q_inv;
        if (lane == 0) more[d] = kx, more[4 + d] = qx;
      }
      if (lane == 0) more[3] = kq * k_inv * q_inv;
    }
  }
  for (int h = blockIdx.y * PREP_THREADS + threadIdx.x; h < heads; h += gridDim.y * PREP_THREADS) {
    const float av = le::to_f32(proj[t * proj_stride + a_col + h]), bv = le::to_f32(proj[t * proj_stride + b_col + h]);
    dst[4 * kv_heads + 2 * h + 0] = expf(-expf(a_log[h]) * softplus_f32(av + dt_bias[h]));
    dst[4 * kv_heads + 2 * h + 1] = sigmoid_f32(bv);
  }
}

// A piece of a row as it is fetched: 16 bytes where the addresses allow it, else one entry.
template <typename T, int P>
struct RowPiece {
  using Raw = uint4;
  static __device__ __forceinline__ Raw zero() { return make_uint4(0u, 0u, 0u, 0u); }
  static __device__ __forceinline__ Raw load(const T *p) { return *reinterpret_cast<const uint4 *>(p); }
  // The piece as floats times `f`, to shared memory (16-byte aligned).
  static __device__ __forceinline__ void store(float *dst, const Raw &r, float f) {
    if constexpr (sizeof(T) == 2) {
      *reinterpret_cast<float4 *>(dst) = make_float4(__uint_as_float(r.x << 16) * f, __uint_as_float(r.x & 0xffff0000u) * f,
                                                     __uint_as_float(r.y << 16) * f, __uint_as_float(r.y & 0xffff0000u) * f);
      *reinterpret_cast<float4 *>(dst + 4) = make_float4(__uint_as_float(r.z << 16) * f, __uint_as_float(r.z & 0xffff0000u) * f,
                                                         __uint_as_float(r.w << 16) * f, __uint_as_float(r.w & 0xffff0000u) * f);
    } else {
      *reinterpret_cast<float4 *>(dst) = make_float4(__uint_as_float(r.x) * f, __uint_as_float(r.y) * f,
                                                     __uint_as_float(r.z) * f, __uint_as_float(r.w) * f);
    }
  }
};
template <typename T>
struct RowPiece<T, 1> {
  using Raw = float;
  static __device__ __forceinline__ Raw zero() { return 0.0f; }
  static __device__ __forceinline__ Raw load(const T *p) { return le::to_f32(*p); }
  static __device__ __forceinline__ void store(float *dst, const Raw &r, float f) { *dst = r * f; }
};

// n tokens' keys and queries of one group as 32-bit unit vectors (the query's times its scale) into kt and qt
// [n][dpad], zeros behind dim.  Every thread asks for SCAN_BATCH pieces before it waits for one.
template <typename T, int P>
__device__ __forceinline__ void fetch_unit_vectors(float *kt, float *qt, const T *src0, int64_t stride, int q_col, int k_col,
                                                   const float *prep0, int prep_stride, int group, int n, int dim, int dpad,
                                                   int tid, int nthreads) {
  using Piece = RowPiece<T, P>;
  const int pieces = dpad / P, per = n * pieces;
  for (int i0 = tid; i0 < 2 * per; i0 += SCAN_BATCH * nthreads) {
    typename Piece::Raw raw[SCAN_BATCH];
    float scale[SCAN_BATCH];
#pragma unroll
    for (int u = 0; u < SCAN_BATCH; ++u) {
      const int idx = i0 + u * nthreads;
      raw[u] = Piece::zero();
      scale[u] = 0.0f;
      if (idx < 2 * per) {
        const int which = idx >= per, r = idx - which * per, t = r / pieces, c = (r - t * pieces) * P;
        if (c < dim) {
          raw[u] = Piece::load(src0 + t * stride + (which ? q_col : k_col) + c);
          scale[u] = prep0[static_cast<int64_t>(t) * prep_stride + 4 * group + which];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < SCAN_BATCH; ++u) {
      const int idx = i0 + u * nthreads;
      if (idx < 2 * per) {
        const int which = idx >= per, r = idx - which * per;
        Piece::store((which ? qt : kt) + static_cast<int64_t>(r) * P, raw[u], scale[u]);
      }
    }
  }
}

template <typename T, int ROWS, int LANES>
__global__ void __launch_bounds__(SCAN_THREADS)
gated_delta_scan_kernel(float *__restrict__ out, int64_t out_stride, const T *__restrict__ qkv, int64_t qkv_stride, int q_col,
                        int k_col, int v_col, const float *__restrict__ prep, int prep_stride, float *__restrict__ state,
                        int num_state_rows, const int32_t *__restrict__ state_slots, const int32_t *__restrict__ cu_q,
                        int heads, int kv_heads, int dim, int vdim, int tile, int wide) {
  extern __shared__ __align__(16) unsigned char scan_smem[];
  constexpr int QUADS = ROWS / 4;                   // groups of four rows a thread holds
  constexpr int DPAD = ROWS * LANES;
  constexpr int COLS = SCAN_HOLDERS / LANES;        // columns of this block
  // One of the two buffers: k [tile][DPAD] | q [tile][DPAD] | v [tile][COLS] | numbers [tile][SCAN_NUMBERS], all float.
  const int vec_floats = tile * DPAD;
  const int buf_floats = 2 * vec_floats + tile * (COLS + SCAN_NUMBERS);
  float *smem = reinterpret_cast<float *>(scan_smem);
  le::let_successor_start();
  const int b = blockIdx.z, h = blockIdx.y;
  const int group = h / (heads / kv_heads);
  const int first = cu_q[b], q_len = cu_q[b + 1] - first;
  const int slot = state_slots[b];
  const bool kept = slot >= 0 && slot < num_state_rows;
  const bool holder = threadIdx.x < SCAN_HOLDERS;
  const int col = (threadIdx.x % SCAN_HOLDERS) / LANES, part = threadIdx.x % LANES;
  const int j = blockIdx.x * COLS + col;            // this thread's column of the state
  const bool col_ok = j < vdim;
  // Of its column a thread holds the rows 4 (i LANES + part) .. + 3, i < QUADS: neighbouring threads hold
  // neighbouring 16 bytes, of the state as of the tiles in shared memory.
  float S[ROWS];
  float *mine = nullptr;
  if (holder && kept && col_ok) mine = state + ((static_cast<int64_t>(slot) * heads + h) * vdim + j) * dim;
  const bool quads_whole = dim % 4 == 0;            // (every group of four then starts on 16 bytes and ends inside dim)
#pragma unroll
  for (int i = 0; i < QUADS; ++i) {
    const int r0 = 4 * (i * LANES + part);
    float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (mine != nullptr) {
      if (quads_whole) {
        if (r0 < dim) r = *reinterpret_cast<const float4 *>(mine + r0);
      } else {
        if (r0 < dim) r.x = mine[r0];
        if (r0 + 1 < dim) r.y = mine[r0 + 1];
        if (r0 + 2 < dim) r.z = mine[r0 + 2];
        if (r0 + 3 < dim) r.w = mine[r0 + 3];
      }
    }
    S[4 * i] = r.x, S[4 * i + 1] = r.y, S[4 * i + 2] = r.z, S[4 * i + 3] = r.w;
  }

  auto fetch = [&](int buf, int t0, int n, int tid, int nthreads) {
    float *kt = smem + buf * buf_floats, *qt = kt + vec_floats, *vt = qt + vec_floats, *nt = vt + tile * COLS;
    const T *src0 = qkv + static_cast<int64_t>(first + t0) * qkv_stride + group * dim;
    const float *prep0 = prep + static_cast<int64_t>(first + t0) * prep_stride;
    if (wide)
      fetch_unit_vectors<T, 16 / sizeof(T)>(kt, qt, src0, qkv_stride, q_col, k_col, prep0, prep_stride, group, n, dim, DPAD, tid, nthreads);
    else
      fetch_unit_vectors<T, 1>(kt, qt, src0, qkv_stride, q_col, k_col, prep0, prep_stride, group, n, dim, DPAD, tid, nthreads);
    // v's columns and three numbers a token: k . q, decay, step size
    constexpr int EACH = COLS + 3, SMALL = 4;
    const int small = n * EACH;
    for (int i0 = tid; i0 < small; i0 += SMALL * nthreads) {
      float val[SMALL];
#pragma unroll
      for (int u = 0; u < SMALL; ++u) {
        const int idx = i0 + u * nthreads;
        val[u] = 0.0f;
        if (idx < small) {
          const int t = idx / EACH, c = idx - t * EACH;
          if (c < COLS) {
            const int jj = blockIdx.x * COLS + c;
            if (jj < vdim) val[u] = le::to_f32(qkv[static_cast<int64_t>(first + t0 + t) * qkv_stride + v_col + h * vdim + jj]);
          } else {
            const float *row = prep0 + static_cast<int64_t>(t) * prep_stride;
            val[u] = c == COLS ? row[4 * group + 2] : row[4 * kv_heads + 2 * h + (c - COLS - 1)];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < SMALL; ++u) {
        const int idx = i0 + u * nthreads;
        if (idx < small) {
          const int t = idx / EACH, c = idx - t * EACH;
          if (c < COLS) vt[t * COLS + c] = val[u];
          else nt[t * SCAN_NUMBERS + (c - COLS)] = val[u];
        }
      }
    }
  };

  le::wait_for_predecessor();
  const int fetchers = static_cast<int>(blockDim.x) - SCAN_HOLDERS;    // (none in a step of single tokens)
  if (q_len > 0) fetch(0, 0, min(tile, q_len), threadIdx.x, blockDim.x);
  __syncthreads();
  const bool writer = holder && part == 0 && col_ok;
  int buf = 0;
  for (int t0 = 0; t0 < q_len; t0 += tile, buf ^= 1) {
    const int n = min(tile, q_len - t0);
    const bool more = t0 + tile < q_len;
    if (!holder) {
      if (more) fetch(buf ^ 1, t0 + tile, min(tile, q_len - t0 - tile), threadIdx.x - SCAN_HOLDERS, fetchers);
    } else {
      const float *kt = smem + buf * buf_floats + 4 * part, *qt = kt + vec_floats;
      const float *vt = smem + buf * buf_floats + 2 * vec_floats + col;
      const float *nt = smem + buf * buf_floats + 2 * vec_floats + tile * COLS;
      float *dst = out + static_cast<int64_t>(first + t0) * out_stride + h * vdim + j;
      for (int t = 0; t < n; ++t, kt += DPAD, qt += DPAD, vt += COLS, nt += SCAN_NUMBERS, dst += out_stride) {
        float kreg[ROWS], qreg[ROWS];
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
          const float4 k4 = *reinterpret_cast<const float4 *>(kt + 4 * i * LANES);
          const float4 q4 = *reinterpret_cast<const float4 *>(qt + 4 * i * LANES);
          kreg[4 * i] = k4.x, kreg[4 * i + 1] = k4.y, kreg[4 * i + 2] = k4.z, kreg[4 * i + 3] = k4.w;
          qreg[4 * i] = q4.x, qreg[4 * i + 1] = q4.y, qreg[4 * i + 2] = q4.z, qreg[4 * i + 3] = q4.w;
        }
        const float4 num = *reinterpret_cast<const float4 *>(nt);       // k . q, decay, step size
        const float v = *vt;
        float dk[4] = {0.0f, 0.0f, 0.0f, 0.0f}, dq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < ROWS; ++i) dk[i & 3] = fmaf(S[i], kreg[i], dk[i & 3]), dq[i & 3] = fmaf(S[i], qreg[i], dq[i & 3]);
        float sk = (dk[0] + dk[1]) + (dk[2] + dk[3]), sq = (dq[0] + dq[1]) + (dq[2] + dq[3]);
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) {
          sk += __shfl_xor_sync(0xffffffffu, sk, o);
          sq += __shfl_xor_sync(0xffffffffu, sq, o);
        }
        const float g = num.y;
        const float u = num.z * (v - g * sk);               // beta (v - (g S0)^T k)
#pragma unroll
        for (int i = 0; i < ROWS; ++i) S[i] = fmaf(kreg[i], u, g * S[i]);
        // o = (g S0 + k u^T)^T q = g (S0 . q) + (k . q) u
        if (writer) *dst = kept ? fmaf(g, sq, num.x * u) : 0.0f;
      }
    }
    __syncthreads();            // the next tile is there, and this one is done with
    if (fetchers <= 0 && more) {
      fetch(buf ^ 1, t0 + tile, min(tile, q_len - t0 - tile), threadIdx.x, blockDim.x);
      __syncthreads();
    }
  }
  if (mine != nullptr) {
#pragma unroll
    for (int i = 0; i < QUADS; ++i) {
      const int r0 = 4 * (i * LANES + part);
      if (quads_whole) {
        if (r0 < dim) *reinterpret_cast<float4 *>(mine + r0) = make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (r0 + e < dim) mine[r0 + e] = S[4 * i + e];
      }
    }
  }
}

// ---------------------------------------------------------------- four tokens at a time
// For heads of 65 to 128 entries and requests that bring several tokens.  With S0 the state before GROUP tokens,
// G_i = g_0 .. g_i, r_ij = g_(j+1) .. g_i, and k, q unit vectors (q times its scale):
//
//   u_i = beta_i (v_i - G_i (S0^T k_i) - sum_(j<i) r_ij (k_i . k_j) u_j)
//   o_i = G_i (S0^T q_i) + sum_(j<=i) r_ij (q_i . k_j) u_j
//   S  <- G_last S0 + sum_j r_(last,j) k_j u_j^T
//
// the same recurrence; gated_delta_factors_kernel makes its numbers beforehand, once per head and group, with the
// vectors' inverse lengths in them, so that the recurrence reads k, q and v as they lie in memory: exact bfloat16,
// by cp.async, GROUP_STAGES tiles ahead.
// What bounded the walk token by token (3,001 tokens, 16 heads of 128 x 128: 555 us, 0.18 us a token): the warps that
// fetch, which asked for a tile's pieces, prepared numbers and values one batch after the other and waited out the
// memory's latency for each (groups of four tokens behind the same fetching took as long).  Then the chain of a token:
// dots, shuffles and the update, each as long as its latencies.  In a group the dots of all four tokens with the old
// state depend on nothing of one another, their 16 sums (2 columns, 4 tokens, k and q) meet in 15 exchanges over the 16
// lanes that share a column instead of three per dot, and the state takes one multiplication for four tokens: the whole
// call 563 -> 437 us, error against 64 bits 2.30e-6 -> 2.23e-6.  What bounds it now: some 400 instructions a group and
// warp, one warp a scheduler, at 2.4 cycles each.
// A thread holds 8 entries of two columns, so that what it reads and widens of k and q serves both; with one column a
// thread and twice the warps the time was the same (438 us).
constexpr int GROUP = 4;
constexpr int GROUP_LANES = 16, GROUP_DIM = 128, GROUP_COLS = 16;     // lanes a column pair, entries, columns a block
constexpr int GROUP_THREADS = GROUP_LANES * GROUP_COLS / 2;
constexpr int GROUP_TILE = 8, GROUP_STAGES = 8;                       // tokens a stage holds
// Numbers of one head and group: beta [4] at 0, G_i / |k_i| [4] at 4, G_i / |q_i| [4] at 8, beta_i r_ij (k_i . k_j)
// [4][4] at 12 (zeros but j < i), r_ij (q_i . k_j) [4][4] at 28 (zeros but j <= i), r_(last,j) / |k_j| [4] at 44, G_last at 48.
constexpr int GROUP_FACTORS = 52;

// A request's first group in the list of all: groups of different requests never meet (request b has at most
// (its tokens) / 4 + 1 of them).  The list ends before tokens / 4 + requests.
__device__ __forceinline__ int64_t first_group(int first_token, int request) { return (first_token >> 2) + request; }

__global__ void __launch_bounds__(128)
gated_delta_factors_kernel(float *__restrict__ factors, const float *__restrict__ prep, int prep_stride,
                           const int32_t *__restrict__ cu_q, int heads, int kv_heads) {
  le::let_successor_start();
  const int b = blockIdx.y;
  const int first = cu_q[b], q_len = cu_q[b + 1] - first;
  const int64_t items = static_cast<int64_t>((q_len + GROUP - 1) / GROUP) * heads;
  le::wait_for_predecessor();
  for (int64_t item = static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x; item < items; item += static_cast<int64_t>(gridDim.x) * 128) {
    const int i = static_cast<int>(item / heads), h = static_cast<int>(item - static_cast<int64_t>(i) * heads);
    const int group = h / (heads / kv_heads);
    float g[GROUP], beta[GROUP], k_inv[GROUP], q_inv[GROUP], kk[GROUP][3], qk[GROUP][4];
#pragma unroll
    for (int a = 0; a < GROUP; ++a) {
      const bool in = i * GROUP + a < q_len;              // (behind the request's last token: u is zero, the state stays)
      const float *row = prep + static_cast<int64_t>(first + (in ? i * GROUP + a : 0)) * prep_stride;
      const float *p = row + 4 * kv_heads + 2 * heads + GROUP_PRODUCTS * group;
      k_inv[a] = in ? row[4 * group] : 0.0f;
      q_inv[a] = in ? row[4 * group + 1] : 0.0f;
      g[a] = in ? row[4 * kv_heads + 2 * h] : 1.0f;
      beta[a] = in ? row[4 * kv_heads + 2 * h + 1] : 0.0f;
#pragma unroll
      for (int d = 0; d < 3; ++d) kk[a][d] = in ? p[d] : 0.0f;
#pragma unroll
      for (int d = 0; d < 4; ++d) qk[a][d] = in ? p[3 + d] : 0.0f;
    }
    float f[GROUP_FACTORS];
#pragma unroll
    for (int e = 0; e < GROUP_FACTORS; ++e) f[e] = 0.0f;
    float G = 1.0f;
#pragma unroll
    for (int a = 0; a < GROUP; ++a) {
      G *= g[a];
      f[a] = beta[a], f[4 + a] = G * k_inv[a], f[8 + a] = G * q_inv[a];
      f[28 + 4 * a + a] = qk[a][0];
      float r = 1.0f;
#pragma unroll
      for (int j = GROUP - 1; j >= 0; --j) {
        if (j < a) {
          r *= g[j + 1];
          f[12 + 4 * a + j] = beta[a] * (r * kk[a][a - j - 1]);
          f[28 + 4 * a + j] = r * qk[a][a - j];
        }
      }
    }
    f[44] = g[1] * g[2] * g[3] * k_inv[0], f[45] = g[2] * g[3] * k_inv[1], f[46] = g[3] * k_inv[2], f[47] = k_inv[3], f[48] = G;
    float4 *dst = reinterpret_cast<float4 *>(factors + ((first_group(first, b) + i) * heads + h) * GROUP_FACTORS);
#pragma unroll
    for (int e = 0; e < GROUP_FACTORS / 4; ++e) dst[e] = make_float4(f[4 * e], f[4 * e + 1], f[4 * e + 2], f[4 * e + 3]);
  }
}

__device__ __forceinline__ void delta_cp16(void *smem, const void *gmem, bool valid) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(gmem), "r"(bytes));
}
// The eight bfloat16 of a 16-byte piece as pairs of floats.
__device__ __forceinline__ void piece_pairs(float2 (&v)[4], const uint4 &r) {
  v[0] = make_float2(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u));
  v[1] = make_float2(__uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
  v[2] = make_float2(__uint_as_float(r.z << 16), __uint_as_float(r.z & 0xffff0000u));
  v[3] = make_float2(__uint_as_float(r.w << 16), __uint_as_float(r.w & 0xffff0000u));
}

struct GroupStage {
  __nv_bfloat16 k[GROUP_TILE][GROUP_DIM], q[GROUP_TILE][GROUP_DIM], v[GROUP_TILE][GROUP_COLS];
  float factors[GROUP_TILE / GROUP][GROUP_FACTORS];
};
static_assert(sizeof(GroupStage) % 16 == 0, "stages start on 16 bytes");

__global__ void __launch_bounds__(GROUP_THREADS)
gated_delta_groups_kernel(float *__restrict__ out, int64_t out_stride, const __nv_bfloat16 *__restrict__ qkv, int64_t qkv_stride,
                          int q_col, int k_col, int v_col, const float *__restrict__ factors, float *__restrict__ state,
                          int num_state_rows, const int32_t *__restrict__ state_slots, const int32_t *__restrict__ cu_q,
                          int heads, int kv_heads, int dim, int vdim) {
  extern __shared__ __align__(16) unsigned char scan_smem[];
  GroupStage *ring = reinterpret_cast<GroupStage *>(scan_smem);
  le::let_successor_start();
  const int b = blockIdx.z, h = blockIdx.y;
  const int first = cu_q[b], q_len = cu_q[b + 1] - first;
  const int slot = state_slots[b];
  const bool kept = slot >= 0 && slot < num_state_rows;
  const int tid = threadIdx.x, part = tid % GROUP_LANES;
  const int c0 = tid / GROUP_LANES * 2;                              // this thread's columns of the block's: c0, c0 + 1
  const int j0 = blockIdx.x * GROUP_COLS + c0;
  auto mine = [&](int c) -> float * {                                // entries 8 part .. + 7 of column c
    return kept && j0 + c < vdim && 8 * part < dim ? state + ((static_cast<int64_t>(slot) * heads + h) * vdim + j0 + c) * dim + 8 * part : nullptr;
  };
  le::wait_for_predecessor();
  const __nv_bfloat16 *rows = qkv + static_cast<int64_t>(first) * qkv_stride;
  const int k_at = k_col + h / (heads / kv_heads) * dim, q_at = q_col + h / (heads / kv_heads) * dim;
  const int v_at = v_col + h * vdim + blockIdx.x * GROUP_COLS;
  const float *my_factors = factors + (first_group(first, b) * heads + h) * GROUP_FACTORS;
  const int groups = (q_len + GROUP - 1) / GROUP, tiles = (q_len + GROUP_TILE - 1) / GROUP_TILE;
  auto fetch = [&](int tile) {
    GroupStage &s = ring[tile % GROUP_STAGES];
    const int t0 = tile * GROUP_TILE;
    constexpr int PIECES = GROUP_DIM / 8;
#pragma unroll
    for (int i = 0; i < 2 * GROUP_TILE * PIECES / GROUP_THREADS; ++i) {
      const int c = tid + i * GROUP_THREADS;
      const int which = c / (GROUP_TILE * PIECES), t = c / PIECES % GROUP_TILE, e = c % PIECES * 8;
      const bool valid = t0 + t < q_len && e < dim;
      delta_cp16(which ? &s.q[t][e] : &s.k[t][e], rows + (valid ? static_cast<int64_t>(t0 + t) * qkv_stride + (which ? q_at : k_at) + e : 0), valid);
    }
    if (tid < GROUP_TILE * GROUP_COLS / 8) {
      const int t = tid / (GROUP_COLS / 8), e = tid % (GROUP_COLS / 8) * 8;
      const bool valid = t0 + t < q_len && blockIdx.x * GROUP_COLS + e < vdim;
      delta_cp16(&s.v[t][e], rows + (valid ? static_cast<int64_t>(t0 + t) * qkv_stride + v_at + e : 0), valid);
    } else if (tid >= 32 && tid < 32 + GROUP_TILE / GROUP * (GROUP_FACTORS / 4)) {
      const int g = (tid - 32) / (GROUP_FACTORS / 4), e = (tid - 32) % (GROUP_FACTORS / 4) * 4;
      const int at = tile * (GROUP_TILE / GROUP) + g;
      const bool valid = at < groups;
      delta_cp16(&s.factors[g][e], my_factors + (valid ? static_cast<int64_t>(at) * heads * GROUP_FACTORS + e : 0), valid);
    }
  };
#pragma unroll
  for (int s = 0; s < GROUP_STAGES - 2; ++s) {
    if (s < tiles) fetch(s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  float2 S[2][4];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const float *from = mine(c);
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f), y = x;
    if (from != nullptr) x = *reinterpret_cast<const float4 *>(from), y = *reinterpret_cast<const float4 *>(from + 4);
    S[c][0] = make_float2(x.x, x.y), S[c][1] = make_float2(x.z, x.w), S[c][2] = make_float2(y.x, y.y), S[c][3] = make_float2(y.z, y.w);
  }
  // the lane that ends with the sum of (column lane_c, k or q, token lane_i)
  const int lane_c = part >> 3, lane_i = part & 3;
  const bool writer = (part & 4) != 0 && j0 + lane_c < vdim;
  float *dst = out + static_cast<int64_t>(first + lane_i) * out_stride + static_cast<int64_t>(h) * vdim + j0 + lane_c;
  uint4 k_raw[GROUP], q_raw[GROUP];               // the next group's entries, read while the sums of this one meet
  auto arrive = [&](int tile) {                   // every thread's pieces of the tile are there, and the tile two before is done with
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GROUP_STAGES - 3));
    __syncthreads();
    if (tile + GROUP_STAGES - 2 < tiles) fetch(tile + GROUP_STAGES - 2);
    asm volatile("cp.async.commit_group;\n" ::);
  };
  auto read = [&](const GroupStage &s, int gi) {
#pragma unroll
    for (int a = 0; a < GROUP; ++a) {
      k_raw[a] = *reinterpret_cast<const uint4 *>(&s.k[gi * GROUP + a][8 * part]);
      q_raw[a] = *reinterpret_cast<const uint4 *>(&s.q[gi * GROUP + a][8 * part]);
    }
  };
  if (tiles > 0) {
    arrive(0);
    read(ring[0], 0);
  }
  for (int tile = 0; tile < tiles; ++tile) {
    const GroupStage &s = ring[tile % GROUP_STAGES];
#pragma unroll
    for (int gi = 0; gi < GROUP_TILE / GROUP; ++gi) {
      const int t0 = tile * GROUP_TILE + gi * GROUP;
      const float *f = s.factors[gi];
      float2 k[GROUP][4];
      float d[16];                                // column, k or q, token
#pragma unroll
      for (int a = 0; a < GROUP; ++a) {
        float2 q[4];
        piece_pairs(k[a], k_raw[a]);
        piece_pairs(q, q_raw[a]);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float2 sk = __fmul2_rn(S[c][0], k[a][0]), sq = __fmul2_rn(S[c][0], q[0]);
#pragma unroll
          for (int e = 1; e < 4; ++e) sk = __ffma2_rn(S[c][e], k[a][e], sk), sq = __ffma2_rn(S[c][e], q[e], sq);
          d[c * 8 + a] = sk.x + sk.y, d[c * 8 + 4 + a] = sq.x + sq.y;
        }
      }
      // what the sums below do not depend on is asked for before them
      const float4 beta = *reinterpret_cast<const float4 *>(f), G = *reinterpret_cast<const float4 *>(f + 4);
      const float4 a1 = *reinterpret_cast<const float4 *>(f + 16), a2 = *reinterpret_cast<const float4 *>(f + 20),
                   a3 = *reinterpret_cast<const float4 *>(f + 24);
      const float4 into = *reinterpret_cast<const float4 *>(f + 44);
      const float4 p = *reinterpret_cast<const float4 *>(f + 28 + 4 * lane_i);
      const float g_last = t0 < q_len ? f[48] : 1.0f;      // (a group behind the request's last: zeros, and the state stays)
      const float g_q = f[8 + lane_i];
      float2 v[GROUP];
#pragma unroll
      for (int a = 0; a < GROUP; ++a) v[a] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&s.v[gi * GROUP + a][c0]));
      if (gi + 1 < GROUP_TILE / GROUP) {
        read(s, gi + 1);
      } else if (tile + 1 < tiles) {
        arrive(tile + 1);
        read(ring[(tile + 1) % GROUP_STAGES], 0);
      }
      // lane `part` ends with the sum d[part] of the 16 lanes
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const bool up = (part & o) != 0;
#pragma unroll
        for (int e = 0; e < o; ++e) {
          const float send = up ? d[e] : d[e + o], keep = up ? d[e + o] : d[e];
          d[e] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      const float sum = d[0];
      float u[2][GROUP];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float sk[GROUP];
#pragma unroll
        for (int a = 0; a < GROUP; ++a) sk[a] = __shfl_sync(0xffffffffu, sum, c * 8 + a, GROUP_LANES);
        const float v0 = c ? v[0].y : v[0].x, v1 = c ? v[1].y : v[1].x, v2 = c ? v[2].y : v[2].x, v3 = c ? v[3].y : v[3].x;
        // beta (v - G S0 . k) of the four, then what the ones before take off
        u[c][0] = beta.x * fmaf(-G.x, sk[0], v0);
        u[c][1] = fmaf(-a1.x, u[c][0], beta.y * fmaf(-G.y, sk[1], v1));
        u[c][2] = fmaf(-a2.y, u[c][1], fmaf(-a2.x, u[c][0], beta.z * fmaf(-G.z, sk[2], v2)));
        u[c][3] = fmaf(-a3.z, u[c][2], fmaf(-a3.y, u[c][1], fmaf(-a3.x, u[c][0], beta.w * fmaf(-G.w, sk[3], v3))));
      }
      // S <- G_last S + sum of r_(last,j) u_j k_j
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float w[GROUP] = {into.x * u[c][0], into.y * u[c][1], into.z * u[c][2], into.w * u[c][3]};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float2 x = __fmul2_rn(make_float2(g_last, g_last), S[c][e]);
#pragma unroll
          for (int a = 0; a < GROUP; ++a) x = __ffma2_rn(make_float2(w[a], w[a]), k[a][e], x);
          S[c][e] = x;
        }
      }
      float o = g_q * sum;
      o = fmaf(p.x, lane_c ? u[1][0] : u[0][0], o);
      o = fmaf(p.y, lane_c ? u[1][1] : u[0][1], o);
      o = fmaf(p.z, lane_c ? u[1][2] : u[0][2], o);
      o = fmaf(p.w, lane_c ? u[1][3] : u[0][3], o);
      if (writer && t0 + lane_i < q_len) dst[t0 * out_stride] = kept ? o : 0.0f;
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float *to = mine(c);
    if (to == nullptr) continue;
    *reinterpret_cast<float4 *>(to) = make_float4(S[c][0].x, S[c][0].y, S[c][1].x, S[c][1].y);
    *reinterpret_cast<float4 *>(to + 4) = make_float4(S[c][2].x, S[c][2].y, S[c][3].x, S[c][3].y);
  }
}

template <typename T>
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(T *__restrict__ out, int64_t out_stride, const float *__restrict__ o, int64_t o_stride,
                      const T *__restrict__ gate, int64_t gate_stride, const float *__restrict__ weight, float eps,
                      int num_tokens, int heads, int vdim, int weight_per_head, int gate_kind, float out_scale) {
  le::let_successor_start();
  le::wait_for_predecessor();
  const int lane = threadIdx.x & 31;
  const int64_t item = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= static_cast<int64_t>(num_tokens) * heads) return;
  const int64_t t = item / heads;
  const int h = static_cast<int>(item - t * heads);
  const float *x = o + t * o_stride + h * vdim;
  float ss = 0.0f;
  for (int i = lane; i < vdim; i += 32) ss = fmaf(x[i], x[i], ss);
  ss = le::warp_sum(ss);
  const float inv = rsqrtf(ss / static_cast<float>(vdim) + eps);
  const T *gr = gate + t * gate_stride + h * vdim;
  T *dst = out + t * out_stride + h * vdim;
  if (weight_per_head) weight += h * vdim;
  if (gate_kind == 0 && out_scale == 1.0f) {
    for (int i = lane; i < vdim; i += 32) {
      const float z = le::to_f32(gr[i]);
      dst[i] = le::from_f32<T>(x[i] * inv * weight[i] * (z / (1.0f + expf(-z))));
    }
    return;
  }
  for (int i = lane; i < vdim; i += 32) {
    const float z = le::to_f32(gr[i]);
    const float g = gate_kind == 0 ? z / (1.0f + expf(-z)) : 1.0f / (1.0f + expf(-z));
    dst[i] = le::from_f32<T>(x[i] * inv * weight[i] * g * out_scale);
  }
}

}  // namespace

namespace {

// The same for few wide heads: a block per (token, head), four values a thread at a time, kept in registers between
// the sum of squares and the result (V groups of 1024 values; everything on 16-byte addresses for floats, 8 for bfloat16).
template <typename T, int V>
__global__ void __launch_bounds__(256)
head_norm_gate_wide_kernel(T *__restrict__ out, int64_t out_stride, const float *__restrict__ o, int64_t o_stride,
                           const T *__restrict__ gate, int64_t gate_stride, const float *__restrict__ weight, float eps,
                           int heads, int vdim, int weight_per_head, int gate_kind, float out_scale) {
  __shared__ float scratch[33];
  le::let_successor_start();
  le::wait_for_predecessor();
  const int64_t t = blockIdx.x / heads;
  const int h = static_cast<int>(blockIdx.x - t * heads);
  const float *x = o + t * o_stride + static_cast<int64_t>(h) * vdim;
  const T *gr = gate + t * gate_stride + static_cast<int64_t>(h) * vdim;
  T *dst = out + t * out_stride + static_cast<int64_t>(h) * vdim;
  if (weight_per_head) weight += static_cast<int64_t>(h) * vdim;
  float4 xv[V];
  float g[V][4];
  float ss = 0.0f;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int i = (threadIdx.x + v * 256) * 4;
    xv[v] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i < vdim) {
      xv[v] = *reinterpret_cast<const float4 *>(x + i);
      if constexpr (sizeof(T) == 2) {
        const uint2 r = *reinterpret_cast<const uint2 *>(gr + i);
        g[v][0] = __uint_as_float(r.x << 16), g[v][1] = __uint_as_float(r.x & 0xffff0000u);
        g[v][2] = __uint_as_float(r.y << 16), g[v][3] = __uint_as_float(r.y & 0xffff0000u);
      } else {
        const float4 r = *reinterpret_cast<const float4 *>(gr + i);
        g[v][0] = r.x, g[v][1] = r.y, g[v][2] = r.z, g[v][3] = r.w;
      }
    }
    ss = fmaf(xv[v].x, xv[v].x, fmaf(xv[v].y, xv[v].y, fmaf(xv[v].z, xv[v].z, fmaf(xv[v].w, xv[v].w, ss))));
  }
  const float inv = rsqrtf(le::block_sum(ss, scratch) / static_cast<float>(vdim) + eps) * out_scale;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int i = (threadIdx.x + v * 256) * 4;
    if (i >= vdim) continue;
    const float4 w = *reinterpret_cast<const float4 *>(weight + i);
    float y[4] = {xv[v].x * inv * w.x, xv[v].y * inv * w.y, xv[v].z * inv * w.z, xv[v].w * inv * w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float s = 1.0f / (1.0f + expf(-g[v][e]));
      y[e] *= gate_kind == 0 ? g[v][e] * s : s;
    }
    if constexpr (sizeof(T) == 2) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[1]), hi = __floats2bfloat162_rn(y[2], y[3]);
      uint2 r;
      r.x = *reinterpret_cast<const uint32_t *>(&lo), r.y = *reinterpret_cast<const uint32_t *>(&hi);
      *reinterpret_cast<uint2 *>(dst + i) = r;
    } else {
      *reinterpret_cast<float4 *>(dst + i) = make_float4(y[0], y[1], y[2], y[3]);
    }
  }
}

// How a column of the state is shared out for heads of `dim` entries: `rows` entries a thread, `lanes` threads a
// column (a power of two, rows * lanes >= dim); false: dim is too large.  Heads of 128 to 256 entries may be held 8 or
// 16 rows a thread (LYAPUNOV_DELTA_ROWS=8|16; the default is the one measured faster).
bool scan_shape(int dim, int &rows, int &lanes) {
  static const int preferred = [] {
    const char *v = std::getenv("LYAPUNOV_DELTA_ROWS");
    return v != nullptr && std::atoi(v) == 8 ? 8 : 16;
  }();
  if (dim < 1 || dim > 1024) return false;
  rows = dim <= 256 ? (dim >= 128 ? preferred : 8) : (dim <= 512 ? 16 : 32);
  lanes = 1;
  while (lanes * rows < dim) lanes <<= 1;
  return true;
}

}  // namespace

// The lanes that share a column of the state for heads of `dim` entries (a power of two; 0: dim is too large).
LE_API int le_gated_delta_lanes(int dim) {
  int rows = 0, lanes = 0;
  return scan_shape(dim, rows, lanes) ? lanes : 0;
}

// Floats of one token's numbers (gated_delta_prepare_kernel).
static int delta_numbers(int heads, int kv_heads) { return (4 + GROUP_PRODUCTS) * kv_heads + 2 * heads; }
// Floats per token of the scratch that le_gated_delta_scan needs: the token's numbers, and its part of the groups'
// numbers per head (tokens / 4 + requests groups at most, and no more requests than tokens).
LE_API int le_gated_delta_scratch(int heads, int kv_heads) {
  return delta_numbers(heads, kv_heads) + GROUP_FACTORS * heads * (GROUP + 1) / GROUP + 4;
}

// out [tokens, heads * vdim] float32.  qkv: rows holding the convolved, activated queries and keys [kv_heads, dim]
// at columns q_col and k_col and values [heads, vdim] at v_col.  proj: rows holding one number per head at b_col
// (step size before its sigmoid) and at a_col (decay before its softplus).  state: [rows, heads, vdim, dim] float32.
// scratch: [tokens, le_gated_delta_scratch()] float32, rewritten here.
LE_API int le_gated_delta_scan(float *out, int64_t out_stride, const void *qkv, int64_t qkv_stride, int q_col, int k_col,
                               int v_col, const void *proj, int64_t proj_stride, int b_col, int a_col, int dtype,
                               const float *a_log, const float *dt_bias, float *state, int num_state_rows,
                               const int32_t *state_slots, const int32_t *cu_q, int num_requests, int num_tokens, int heads,
                               int kv_heads, int dim, int vdim, float unit_eps, float q_scale, float *scratch,
                               cudaStream_t stream) {
  if (num_requests <= 0 || num_tokens <= 0) return 0;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads) return le::invalid("le_gated_delta_scan: %d heads, %d groups", heads, kv_heads);
  int rows = 0, lanes = 0;
  if (!scan_shape(dim, rows, lanes)) return le::invalid("le_gated_delta_scan: heads of %d entries (at most 1024)", dim);
  if (dtype != LE_BF16 && dtype != LE_F32) return le::invalid("le_gated_delta_scan: unknown dtype code %d", dtype);
  const int cols = SCAN_HOLDERS / lanes;
  const int prep_stride = delta_numbers(heads, kv_heads);
  const size_t elem = dtype == LE_BF16 ? 2 : 4;
  const int vec = static_cast<int>(16 / elem);
  const int wide = dim % vec == 0 && qkv_stride % vec == 0 && q_col % vec == 0 && k_col % vec == 0 &&
                   reinterpret_cast<uintptr_t>(qkv) % 16 == 0;
  const size_t per_token = sizeof(float) * (2 * static_cast<size_t>(lanes) * rows + cols + SCAN_NUMBERS);
  int tile = static_cast<int>((36 * 1024) / per_token);
  tile = tile < 1 ? 1 : (tile > SCAN_MAX_TILE ? SCAN_MAX_TILE : tile);
  const bool single = num_tokens == num_requests;      // a step of single tokens: one tile of one token, nobody fetches ahead
  if (single) tile = 1;
  const int threads = single ? SCAN_HOLDERS : SCAN_THREADS;
  const size_t smem = 2 * tile * per_token;
  const dim3 prep_grid(num_tokens, (kv_heads + PREP_THREADS / 32 - 1) / (PREP_THREADS / 32));
  const dim3 grid((vdim + cols - 1) / cols, heads, num_requests);
  // Four tokens at a time (see gated_delta_groups_kernel): heads whose entries its 16 lanes of 8 fill to more than a half,
  // in the activations' 16-bit type (the 32-bit engine keeps the order of the walk token by token), whose rows are whole
  // 16-byte pieces.
  const bool grouped = !single && dtype == LE_BF16 && dim > GROUP_DIM / 2 && dim <= GROUP_DIM && wide && vdim % 8 == 0 &&
                       v_col % 8 == 0 && (reinterpret_cast<uintptr_t>(scratch) | reinterpret_cast<uintptr_t>(state)) % 16 == 0;
  if (grid.y > 65535 || grid.z > 65535 || prep_grid.y > 65535)
    return le::invalid("le_gated_delta_scan: too many heads or requests for one launch");
#define LE_GO(T, R, L)                                                                                                  \
  do {                                                                                                                  \
    int rc = le::launch_chained(gated_delta_prepare_kernel<T>, prep_grid, dim3(PREP_THREADS), 0, stream, scratch,       \
                                prep_stride, static_cast<const T *>(qkv), qkv_stride, q_col, k_col,                     \
                                static_cast<const T *>(proj), proj_stride, b_col, a_col, a_log, dt_bias, heads, kv_heads, \
                                dim, unit_eps, q_scale, 0);                                                             \
    if (rc != 0) return rc;                                                                                             \
    if (smem > 48 * 1024)                                                                                               \
      cudaFuncSetAttribute(gated_delta_scan_kernel<T, R, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    return le::launch_chained(gated_delta_scan_kernel<T, R, L>, grid, dim3(threads), smem, stream, out, out_stride,     \
                              static_cast<const T *>(qkv), qkv_stride, q_col, k_col, v_col,                             \
                              static_cast<const float *>(scratch), prep_stride, state, num_state_rows, state_slots, cu_q, \
                              heads, kv_heads, dim, vdim, tile, wide);                                                  \
  } while (0)
#define LE_SHAPE(T, R, L) \
  if (rows == R && lanes == L) LE_GO(T, R, L)
#define LE_SHAPES(T)                                                                                                    \
  LE_SHAPE(T, 8, 1); LE_SHAPE(T, 8, 2); LE_SHAPE(T, 8, 4); LE_SHAPE(T, 8, 8); LE_SHAPE(T, 8, 16); LE_SHAPE(T, 8, 32);   \
  LE_SHAPE(T, 16, 8); LE_SHAPE(T, 16, 16); LE_SHAPE(T, 16, 32); LE_SHAPE(T, 32, 32)
  if (grouped) {
    const auto *rows16 = static_cast<const __nv_bfloat16 *>(qkv);
    int rc = le::launch_chained(gated_delta_prepare_kernel<__nv_bfloat16>, prep_grid, dim3(PREP_THREADS), 0, stream, scratch,
                                prep_stride, rows16, qkv_stride, q_col, k_col, static_cast<const __nv_bfloat16 *>(proj),
                                proj_stride, b_col, a_col, a_log, dt_bias, heads, kv_heads, dim, unit_eps, q_scale, 1);
    if (rc != 0) return rc;
    float *factors = scratch + (static_cast<int64_t>(num_tokens) * prep_stride + 3) / 4 * 4;
    const int64_t most = static_cast<int64_t>((num_tokens + GROUP - 1) / GROUP) * heads;      // one request's, if it has all the tokens
    const dim3 factor_grid(static_cast<unsigned>(most / 128 + 1 < 128 ? most / 128 + 1 : 128), num_requests);
    rc = le::launch_chained(gated_delta_factors_kernel, factor_grid, dim3(128), 0, stream, factors, static_cast<const float *>(scratch),
                            prep_stride, cu_q, heads, kv_heads);
    if (rc != 0) return rc;
    // Its blocks may come while the kernels before it still hold multiprocessors, and would then share the others while
    // those stay idle (four to one: 1,040 us instead of 380).  Where every block
    // can have a multiprocessor of its own it asks for more than half of the shared memory, so that each gets one.
    constexpr int ALONE = 116 * 1024;
    const dim3 group_grid((vdim + GROUP_COLS - 1) / GROUP_COLS, heads, num_requests);
    const size_t bytes = static_cast<int64_t>(group_grid.x) * heads * num_requests <= 148 ? ALONE : GROUP_STAGES * sizeof(GroupStage);
    cudaError_t e = cudaFuncSetAttribute(gated_delta_groups_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ALONE);
    if (e != cudaSuccess) return le::invalid("le_gated_delta_scan: cannot get %d bytes of shared memory: %s", ALONE, cudaGetErrorString(e));
    return le::launch_chained(gated_delta_groups_kernel, group_grid, dim3(GROUP_THREADS), bytes, stream, out, out_stride, rows16,
                              qkv_stride, q_col, k_col, v_col, static_cast<const float *>(factors), state, num_state_rows,
                              state_slots, cu_q, heads, kv_heads, dim, vdim);
  }
  if (dtype == LE_BF16) { LE_SHAPES(__nv_bfloat16); }
  else { LE_SHAPES(float); }
#undef LE_SHAPES
#undef LE_SHAPE
#undef LE_GO
  return le::invalid("le_gated_delta_scan: no kernel for %d rows a thread and %d threads a column", rows, lanes);
}

// out[t, h, :] = o[t, h, :] / sqrt(mean(o[t, h, :]^2) + eps) * weight * act(gate[t, h, :]) * out_scale; weight is
// [vdim], or [heads, vdim] with weight_per_head; act is silu (gate_kind 0) or the sigmoid (1).
LE_API int le_head_norm_gate(void *out, int64_t out_stride, const float *o, int64_t o_stride, const void *gate,
                             int64_t gate_stride, int dtype, const float *weight, float eps, int num_tokens, int heads,
                             int vdim, int weight_per_head, int gate_kind, float out_scale, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  const int64_t items = static_cast<int64_t>(num_tokens) * heads;
  const auto on16 = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (vdim >= 512 && vdim <= 8192 && vdim % 4 == 0 && out_stride % 4 == 0 && o_stride % 4 == 0 && gate_stride % 4 == 0 &&
      on16(o) && on16(weight) && (reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(out)) % (dtype == LE_BF16 ? 8 : 16) == 0) {
#define LE_WIDE(V)                                                                                                        \
  LE_DISPATCH_DTYPE(dtype, T,                                                                                             \
                    return le::launch_chained(head_norm_gate_wide_kernel<T, V>, dim3(static_cast<unsigned>(items)),       \
                                              dim3(256), 0, stream, static_cast<T *>(out), out_stride, o, o_stride,       \
                                              static_cast<const T *>(gate), gate_stride, weight, eps, heads, vdim,        \
                                              weight_per_head, gate_kind, out_scale))
    if (vdim <= 1024) LE_WIDE(1);
    if (vdim <= 2048) LE_WIDE(2);
    if (vdim <= 4096) LE_WIDE(4);
    LE_WIDE(8);
#undef LE_WIDE
  }
  const dim3 grid(static_cast<unsigned>((items + 3) / 4));
  LE_DISPATCH_DTYPE(dtype, T,
                    return le::launch_chained(head_norm_gate_kernel<T>, grid, dim3(128), 0, stream, static_cast<T *>(out),
                                              out_stride, o, o_stride, static_cast<const T *>(gate), gate_stride, weight,
                                              eps, num_tokens, heads, vdim, weight_per_head, gate_kind, out_scale));
}
