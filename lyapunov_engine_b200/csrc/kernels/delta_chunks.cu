// The gated delta rule over chunks of 16 tokens on the tensor cores: the form
// of the recurrence in delta_rule.cu for requests that bring several tokens in
// bfloat16, heads of 65 to 128 entries, from each request's state row and back
// into it.
//
// With S0 the state before a chunk, G_i = g_0 .. g_i, r_ij = g_(j+1) .. g_i, and
// k, q unit vectors (q times its scale), the chunk's updates solve
//
//   u_i + sum_(j<i) beta_i r_ij (k_i . k_j) u_j = beta_i (v_i - G_i S0^T k_i)
//
// whose matrix depends on the tokens alone, and
//
//   o_i = G_i S0^T q_i + sum_(j<=i) r_ij (q_i . k_j) u_j
//   S  <- G_last S0 + sum_j r_(last,j) k_j u_j^T.
//
// delta_chunk_numbers_kernel makes a chunk's numbers beforehand, all chunks side
// by side: per head the inverse of that unit triangular matrix (by substitution,
// times beta_j), the products r_ij (q_i . k_j) times it, and the vectors' inverse
// lengths in the factors around them, so that the chunks' walk reads k, q and v as
// they lie in memory, and u and o follow from the same right sides.
//
// delta_chunk_kernel walks a request's chunks in order: a block is one head and
// 16 columns of S, and each of its eight warps keeps 16 entries of dim of those
// columns in the accumulators of its update, whose layout is that of the left
// operand of the next product.  S0^T [k q] (S in three bfloat16 parts that keep
// all its 24 bits, k and q exact) is summed over the warps through shared memory;
// the two small products with the right sides are 32-bit multiply-adds; the update multiplies
// u in three parts with exact k.  All sums are 32-bit.
//
// What bounds it: token by token (3,001 tokens, 16 heads of 128 x 128) a prompt is
// 3,001 steps of dots, shuffles and updates, each as long as its latencies, behind
// warps that fetch one batch after the other (539 us; four tokens at a time in
// 32-bit multiply-adds it was 437).  A chunk is four meetings of the block instead:
// 227 us, of which the numbers take 30 (u and o one after the other 248).  Error
// against 64 bits over 1,024 tokens 2.7e-7 to 6.0e-7, the scan's 2.8e-7 to 6.6e-7.
#include "chunk_mma.cuh"

namespace {

using bf16 = __nv_bfloat16;
using le::ldsm4, le::ldsm4_trans, le::mma, le::mma_first, le::mma_split3, le::split_pair3, le::split_state3;

constexpr int CHUNK = 16;
constexpr int DIM = 128;                    // entries of a head, padded
constexpr int COLS = 16;                    // columns of S a block takes
constexpr int THREADS = 256;                // a warp for 16 entries of dim; a thread for (token, column)
constexpr int LD = DIM + 8;                 // rows of k and q in shared memory: eight rows' pieces in different banks
constexpr int LDP = COLS + 4;               // rows of the sums and of u
// Numbers of one head and chunk: the inverse times beta_j [16][16], r_ij (q_i . k_j) times it [16][16], G_i / |k_i| [16], G_i / |q_i| [16], r_(last,j) / |k_j| [16], G_last.
constexpr int AT_P = 256, AT_GK = 512, AT_GQ = 528, AT_INTO = 544, AT_LAST = 560, NUMBERS = 564;

__device__ __forceinline__ float softplus_f32(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
// A request's first chunk in the list of all: requests never meet (request b has at most (its tokens) / 16 + 1).
__device__ __forceinline__ int64_t first_chunk(int first_token, int request) { return first_token / CHUNK + request; }

struct DeltaArgs {
  float *out; int64_t out_stride;
  const bf16 *qkv; int64_t qkv_stride; int q_col, k_col, v_col;
  const bf16 *proj; int64_t proj_stride; int b_col, a_col;
  const float *a_log, *dt_bias;
  float *state; int num_state_rows;
  const int32_t *state_slots, *cu_q;
  const int32_t *requests;                  // the requests this launch takes, or null: all in order
  int heads, kv_heads, dim, vdim;
  float unit_eps, q_scale;
  float *numbers;                           // [tokens / 16 + requests, heads, NUMBERS]
};

// One block per chunk and key group (blocks take the chunks of a request in turn).
__global__ void __launch_bounds__(THREADS)
delta_chunk_numbers_kernel(DeltaArgs p) {
  constexpr int LDF = DIM + 4;
  __shared__ __align__(16) float s_k[CHUNK][LDF], s_q[CHUNK][LDF];
  __shared__ float s_inv[2][CHUNK], s_g[CHUNK], s_beta[CHUNK], s_a[CHUNK][CHUNK + 1], s_x[CHUNK][CHUNK + 1], s_p[CHUNK][CHUNK + 1];
  le::let_successor_start();
  const int group = blockIdx.y, b = p.requests != nullptr ? p.requests[blockIdx.z] : blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int i = tid / CHUNK, j = tid % CHUNK;
  const int first = p.cu_q[b], q_len = p.cu_q[b + 1] - first;
  const int per_group = p.heads / p.kv_heads;
  le::wait_for_predecessor();
  for (int t0 = blockIdx.x * CHUNK; t0 < q_len; t0 += gridDim.x * CHUNK) {
    const int len = min(CHUNK, q_len - t0);
    // a thread fetches 8 entries of k and of q of token i
    {
      const int e = j * 8;
      float kv[8] = {}, qv[8] = {};
      if (i < len && e < p.dim) {
        const bf16 *row = p.qkv + static_cast<int64_t>(first + t0 + i) * p.qkv_stride + group * p.dim + e;
        le::load_piece16<bf16>(kv, row + p.k_col);
        le::load_piece16<bf16>(qv, row + p.q_col);
      }
      float kk = 0.0f, qq = 0.0f;
#pragma unroll
      for (int u = 0; u < 8; ++u) kk = fmaf(kv[u], kv[u], kk), qq = fmaf(qv[u], qv[u], qq);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) kk += __shfl_xor_sync(0xffffffffu, kk, o), qq += __shfl_xor_sync(0xffffffffu, qq, o);
      if (j == 0) {
        s_inv[0][i] = i < len ? rsqrtf(kk + p.unit_eps) : 0.0f;
        s_inv[1][i] = i < len ? rsqrtf(qq + p.unit_eps) * p.q_scale : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; u += 4) {
        *reinterpret_cast<float4 *>(&s_k[i][e + u]) = make_float4(kv[u], kv[u + 1], kv[u + 2], kv[u + 3]);
        *reinterpret_cast<float4 *>(&s_q[i][e + u]) = make_float4(qv[u], qv[u + 1], qv[u + 2], qv[u + 3]);
      }
    }
    __syncthreads();
    float kk[4] = {}, qk[4] = {};
    if (j <= i) {
#pragma unroll 4
      for (int e = 0; e < DIM; e += 4) {
        const float4 ki = *reinterpret_cast<const float4 *>(&s_k[i][e]), kj = *reinterpret_cast<const float4 *>(&s_k[j][e]);
        const float4 qi = *reinterpret_cast<const float4 *>(&s_q[i][e]);
        kk[0] = fmaf(ki.x, kj.x, kk[0]), kk[1] = fmaf(ki.y, kj.y, kk[1]), kk[2] = fmaf(ki.z, kj.z, kk[2]), kk[3] = fmaf(ki.w, kj.w, kk[3]);
        qk[0] = fmaf(qi.x, kj.x, qk[0]), qk[1] = fmaf(qi.y, kj.y, qk[1]), qk[2] = fmaf(qi.z, kj.z, qk[2]), qk[3] = fmaf(qi.w, kj.w, qk[3]);
      }
    }
    const float kk_ij = ((kk[0] + kk[1]) + (kk[2] + kk[3])) * s_inv[0][i] * s_inv[0][j];
    const float qk_ij = ((qk[0] + qk[1]) + (qk[2] + qk[3])) * s_inv[1][i] * s_inv[0][j];
    for (int h = group * per_group; h < (group + 1) * per_group; ++h) {
      if (tid < CHUNK) {
        float g = 1.0f, beta = 0.0f;                    // (behind the request's last token: u is zero, the state stays)
        if (tid < len) {
          const bf16 *row = p.proj + static_cast<int64_t>(first + t0 + tid) * p.proj_stride;
          const float av = __bfloat162float(row[p.a_col + h]), bv = __bfloat162float(row[p.b_col + h]);
          g = expf(-expf(p.a_log[h]) * softplus_f32(av + p.dt_bias[h]));
          beta = 1.0f / (1.0f + expf(-bv));
        }
        s_g[tid] = g, s_beta[tid] = beta;
      }
      __syncthreads();
      float r = 1.0f, G = 1.0f;                         // r_ij; and G_i (threads j = 0)
      for (int t = j + 1; t <= i; ++t) r *= s_g[t];
      for (int t = 0; t <= i; ++t) G *= s_g[t];
      s_a[i][j] = j < i ? s_beta[i] * (r * kk_ij) : 0.0f;
      float *dst = p.numbers + ((first_chunk(first, b) + t0 / CHUNK) * p.heads + h) * NUMBERS;
      s_p[i][j] = j <= i ? r * qk_ij : 0.0f;
      if (j == 0) dst[AT_GK + i] = G * s_inv[0][i], dst[AT_GQ + i] = G * s_inv[1][i];
      if (i == CHUNK - 1) dst[AT_INTO + j] = r * s_inv[0][j];
      if (tid == THREADS - 1) dst[AT_LAST] = G;
      __syncthreads();
      // column j of the inverse: x_jj = 1, x_ij = -sum_(j <= m < i) a_im x_mj
      if (warp == 0 && lane < CHUNK) {
        float x[CHUNK];
#pragma unroll
        for (int a = 0; a < CHUNK; ++a) {
          float sum = 0.0f;
#pragma unroll
          for (int m = 0; m < a; ++m) sum = fmaf(s_a[a][m], x[m], sum);
          x[a] = a < lane ? 0.0f : (a == lane ? 1.0f : -sum);
          s_x[a][lane] = x[a];
        }
      }
      __syncthreads();
      dst[tid] = s_x[i][j] * s_beta[j];
      float px = 0.0f;
#pragma unroll
      for (int m = 0; m < CHUNK; ++m) px = m <= i ? fmaf(s_p[i][m], s_x[m][j], px) : px;
      dst[AT_P + tid] = px * s_beta[j];
      __syncthreads();                                  // s_g, s_beta, s_a, s_x and s_p are read
    }
  }
}

struct Stage {
  bf16 k[CHUNK][LD], q[CHUNK][LD], v[CHUNK][COLS];
  float numbers[NUMBERS];
};
static_assert(sizeof(Stage) % 16 == 0 && NUMBERS % 4 == 0, "stages start on 16 bytes");
struct Meeting {
  float part[THREADS / 32][2 * CHUNK][LDP];             // S0^T k of 16 tokens, S0^T q of 16: every warp's share of dim
  float rhs[CHUNK][LDP], u[CHUNK][LDP];
};

template <int STAGES>
__global__ void __launch_bounds__(THREADS)
delta_chunk_kernel(DeltaArgs p) {
  extern __shared__ __align__(16) unsigned char delta_smem[];
  Meeting &meet = *reinterpret_cast<Meeting *>(delta_smem);
  Stage *ring = reinterpret_cast<Stage *>(delta_smem + sizeof(Meeting));
  le::let_successor_start();
  const int b = p.requests != nullptr ? p.requests[blockIdx.z] : blockIdx.z, h = blockIdx.y, e0 = blockIdx.x * COLS;
  const int first = p.cu_q[b], q_len = p.cu_q[b + 1] - first;
  const int slot = p.state_slots[b];
  const bool kept = slot >= 0 && slot < p.num_state_rows;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3, j8 = lane >> 3, r8 = lane & 7;
  const int i = tid / COLS, c = tid % COLS;             // this thread's token of a chunk and column of the block
  const int chunks = (q_len + CHUNK - 1) / CHUNK;
  const int group = h / (p.heads / p.kv_heads);
  const float *numbers = p.numbers + (first_chunk(first, b) * p.heads + h) * NUMBERS;
  const bf16 *rows = p.qkv + static_cast<int64_t>(first) * p.qkv_stride;
  const int k_at = p.k_col + group * p.dim, q_at = p.q_col + group * p.dim, v_at = p.v_col + h * p.vdim + e0;
  le::wait_for_predecessor();

  auto fetch = [&](int chunk) {
    Stage &s = ring[chunk % STAGES];
    const int t0 = chunk * CHUNK;
    constexpr int PIECES = DIM / 8;
#pragma unroll
    for (int u = 0; u < 2; ++u) {                       // k, then q: a thread's piece of a token
      const int t = tid / PIECES, e = tid % PIECES * 8;
      const bool live = t0 + t < q_len && e < p.dim;
      le::copy16_async(u ? &s.q[t][e] : &s.k[t][e], rows + (live ? static_cast<int64_t>(t0 + t) * p.qkv_stride + (u ? q_at : k_at) + e : 0), live);
    }
    if (tid < CHUNK * COLS / 8) {
      const int t = tid / (COLS / 8), e = tid % (COLS / 8) * 8;
      const bool live = t0 + t < q_len && e0 + e < p.vdim;
      le::copy16_async(&s.v[t][e], rows + (live ? static_cast<int64_t>(t0 + t) * p.qkv_stride + v_at + e : 0), live);
    } else if (tid >= 64 && tid < 64 + NUMBERS / 4) {
      const int e = (tid - 64) * 4;
      le::copy16_async(&s.numbers[e], numbers + static_cast<int64_t>(chunk) * p.heads * NUMBERS + e, true);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < chunks) fetch(s);
    le::commit_copies();
  }
  // S^T: tile d holds columns e0 + g (entries 0, 1) and + 8 (2, 3), entries 16 warp + 8 d + 2 t4 and the next of dim
  float S[2][4];
  float *mine[2] = {nullptr, nullptr};
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int col = e0 + g + 8 * x;
    if (kept && col < p.vdim) mine[x] = p.state + ((static_cast<int64_t>(slot) * p.heads + h) * p.vdim + col) * p.dim;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const int at = 16 * warp + 8 * d + 2 * t4;        // (dim is a multiple of 8: a pair is inside or outside)
      const float2 v = mine[x] != nullptr && at < p.dim ? *reinterpret_cast<const float2 *>(mine[x] + at) : make_float2(0.0f, 0.0f);
      S[d][2 * x] = v.x, S[d][2 * x + 1] = v.y;
    }
  }
  float *dst = p.out + static_cast<int64_t>(first + i) * p.out_stride + static_cast<int64_t>(h) * p.vdim + e0 + c;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                    // the chunk is there, and the one before is done with
    if (chunk + STAGES - 1 < chunks) fetch(chunk + STAGES - 1);
    le::commit_copies();
    const Stage &s = ring[chunk % STAGES];
    const float *f = s.numbers;
    // S0^T [k q] of this warp's entries
    {
      uint32_t a[3][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) split_state3(S[u >> 1][2 * (u & 1)], S[u >> 1][2 * (u & 1) + 1], a[0][u], a[1][u], a[2][u]);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t vec[4];
        ldsm4(vec, (x ? &s.q[0][0] : &s.k[0][0]) + ((j8 >> 1) * 8 + r8) * LD + warp * 16 + (j8 & 1) * 8);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          float d[4];
          mma_first(d, a[2], vec[2 * nt], vec[2 * nt + 1]);
          mma(d, a[1], vec[2 * nt], vec[2 * nt + 1]);
          mma(d, a[0], vec[2 * nt], vec[2 * nt + 1]);
          float(*to)[LDP] = &meet.part[warp][x * CHUNK + nt * 8 + 2 * t4];
          to[0][g] = d[0], to[1][g] = d[1], to[0][g + 8] = d[2], to[1][g + 8] = d[3];
        }
      }
    }
    __syncthreads();
    float sk[2] = {0.0f, 0.0f}, sq[2] = {0.0f, 0.0f};
#pragma unroll
    for (int w = 0; w < THREADS / 32; w += 2) {
      sk[0] += meet.part[w][i][c], sk[1] += meet.part[w + 1][i][c];
      sq[0] += meet.part[w][CHUNK + i][c], sq[1] += meet.part[w + 1][CHUNK + i][c];
    }
    meet.rhs[i][c] = fmaf(-f[AT_GK + i], sk[0] + sk[1], __bfloat162float(s.v[i][c]));
    const float of_state = sq[0] + sq[1];
    float o;
    __syncthreads();
    {
      float u[4] = {0.0f, 0.0f, 0.0f, 0.0f}, more[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int j = 0; j < CHUNK; j += 4) {
        const float4 m = *reinterpret_cast<const float4 *>(f + CHUNK * i + j), n = *reinterpret_cast<const float4 *>(f + AT_P + CHUNK * i + j);
        // (both matrices are zero above the diagonal, or what a NaN made of it: later tokens stay out)
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] = meet.rhs[j + e][c];
        const float to_u[4] = {m.x, m.y, m.z, m.w}, to_o[4] = {n.x, n.y, n.z, n.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (j + e > i) continue;
          u[e] = fmaf(to_u[e], r[e], u[e]);
          more[e] = fmaf(to_o[e], r[e], more[e]);
        }
      }
      meet.u[i][c] = (u[0] + u[1]) + (u[2] + u[3]);
      o = fmaf(f[AT_GQ + i], of_state, (more[0] + more[1]) + (more[2] + more[3]));
    }
    if (chunk * CHUNK + i < q_len && e0 + c < p.vdim) dst[static_cast<int64_t>(chunk) * CHUNK * p.out_stride] = kept ? o : 0.0f;
    __syncthreads();
    // the state behind the chunk
    {
      uint32_t a[3][4], kf[4];
      ldsm4_trans(kf, &s.k[0][0] + ((j8 & 1) * 8 + r8) * LD + warp * 16 + (j8 >> 1) * 8);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = 2 * t4 + 8 * (u >> 1), col = g + 8 * (u & 1);
        const float2 into = *reinterpret_cast<const float2 *>(f + AT_INTO + t);
        split_pair3(into.x * meet.u[t][col], into.y * meet.u[t + 1][col], a[0][u], a[1][u], a[2][u]);
      }
      const float last = f[AT_LAST];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
#pragma unroll
        for (int x = 0; x < 4; ++x) S[d][x] *= last;
        mma_split3(S[d], a, kf[2 * d], kf[2 * d + 1]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    if (mine[x] == nullptr) continue;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const int at = 16 * warp + 8 * d + 2 * t4;
      if (at < p.dim) *reinterpret_cast<float2 *>(mine[x] + at) = make_float2(S[d][2 * x], S[d][2 * x + 1]);
    }
  }
}

template <int STAGES>
int launch_walk(const DeltaArgs &p, dim3 grid, size_t least, cudaStream_t stream) {
  const size_t need = sizeof(Meeting) + STAGES * sizeof(Stage), bytes = need > least ? need : least;
  cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e != cudaSuccess) return le::invalid("le_gated_delta_chunks: cannot get %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
  return le::launch_chained(delta_chunk_kernel<STAGES>, grid, dim3(THREADS), bytes, stream, p);
}

}  // namespace

// The scratch of le_gated_delta_chunks: tokens / le_gated_delta_chunk() + requests rows of le_gated_delta_chunk_width()
// floats (the step's tokens and requests, those that are not listed too).
LE_API int le_gated_delta_chunk() { return CHUNK; }
LE_API int le_gated_delta_chunk_width(int heads) { return heads * NUMBERS; }

// Whether the form applies: bfloat16 rows in whole 16-byte pieces, heads of more than 64 and at most 128 entries (its
// eight warps hold 16 each).
LE_API int le_gated_delta_chunks_apply(const void *qkv, int64_t qkv_stride, int q_col, int k_col, int v_col, int dtype, int dim,
                                       int vdim) {
  return dtype == LE_BF16 && dim > DIM / 2 && dim <= DIM && dim % 8 == 0 && vdim % 8 == 0 && qkv_stride % 8 == 0 && q_col % 8 == 0 &&
                 k_col % 8 == 0 && v_col % 8 == 0 && reinterpret_cast<uintptr_t>(qkv) % 16 == 0
             ? 1
             : 0;
}

// le_gated_delta_scan's recurrence over chunks, where le_gated_delta_chunks_apply.  requests: the indices of the
// num_requests requests to run, or null: requests 0 .. num_requests - 1; num_tokens: their tokens in all (it only
// chooses the launch's shape).  scratch: see le_gated_delta_chunk_width, 16-byte aligned.
LE_API int le_gated_delta_chunks(float *out, int64_t out_stride, const void *qkv, int64_t qkv_stride, int q_col, int k_col,
                                 int v_col, const void *proj, int64_t proj_stride, int b_col, int a_col, const float *a_log,
                                 const float *dt_bias, float *state, int num_state_rows, const int32_t *state_slots,
                                 const int32_t *cu_q, const int32_t *requests, int num_requests, int num_tokens, int heads,
                                 int kv_heads, int dim, int vdim, float unit_eps, float q_scale, float *scratch,
                                 cudaStream_t stream) {
  if (num_requests <= 0 || num_tokens <= 0) return 0;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads) return le::invalid("le_gated_delta_chunks: %d heads, %d groups", heads, kv_heads);
  if (!le_gated_delta_chunks_apply(qkv, qkv_stride, q_col, k_col, v_col, LE_BF16, dim, vdim) ||
      (reinterpret_cast<uintptr_t>(scratch) & 15) || (reinterpret_cast<uintptr_t>(state) & 15))
    return le::invalid("le_gated_delta_chunks: heads of %d x %d entries, or rows that are not whole 16-byte pieces", dim, vdim);
  DeltaArgs p{};
  p.out = out, p.out_stride = out_stride, p.qkv = static_cast<const bf16 *>(qkv), p.qkv_stride = qkv_stride;
  p.q_col = q_col, p.k_col = k_col, p.v_col = v_col, p.proj = static_cast<const bf16 *>(proj), p.proj_stride = proj_stride;
  p.b_col = b_col, p.a_col = a_col, p.a_log = a_log, p.dt_bias = dt_bias, p.state = state, p.num_state_rows = num_state_rows;
  p.state_slots = state_slots, p.cu_q = cu_q, p.requests = requests, p.heads = heads, p.kv_heads = kv_heads, p.dim = dim, p.vdim = vdim;
  p.unit_eps = unit_eps, p.q_scale = q_scale, p.numbers = scratch;
  const int most = (num_tokens + CHUNK - 1) / CHUNK;    // chunks of one request, if it has all the tokens
  const dim3 grid((vdim + COLS - 1) / COLS, heads, num_requests);
  if (heads > 65535 || num_requests > 65535) return le::invalid("le_gated_delta_chunks: too many heads or requests for one launch");
  // (with many requests the chunks of a long one are shared out over 16 blocks a group, so that the others' blocks, most of
  // which find nothing to do, stay few)
  const int share = num_requests == 1 ? most : (most < 16 ? most : (2 * most / num_requests > 16 ? 2 * most / num_requests : 16));
  int rc = le::launch_chained(delta_chunk_numbers_kernel, dim3(share, kv_heads, num_requests), dim3(THREADS), 0, stream, p);
  if (rc != 0) return rc;
  // Its blocks may come while the kernel before it still holds multiprocessors, and would then share the others while
  // those stay idle (blocks of the form with four tokens, four to a multiprocessor: 1,040 us instead of 380).  Where every
  // block can have a multiprocessor of its own it asks for more than half of the shared memory, so that each gets one.
  if (static_cast<int64_t>(grid.x) * grid.y * grid.z <= le::multiprocessors()) return launch_walk<8>(p, grid, 116 * 1024, stream);
  return launch_walk<4>(p, grid, 0, stream);
}
