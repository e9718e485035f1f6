// Gated linear attention: a recurrence over a 32-bit state per (sequence, head) whose decay is a number per KEY CHANNEL and
// token:
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T        (S: dim x vdim, a_t: dim numbers in (0, 1])
//     o_t = S_t^T (q_t * q_scale)
//
// with a_t = exp(log_scale * dt_t), dt the caller's 32-bit rows [tokens][heads dim] (log_scale < 0 <= dt: a softplus of the
// negated gate's pre-activation, for instance).  q, k, v are channels of the step's projections, taken as they are.
// The state lives in `state[slot][head][dim][vdim]`; a sequence that starts finds zeros there.
//
// Token by token (gla_scan_kernel): a block owns value channels of one (sequence, head) and keeps its part of the state in
// registers for all tokens of the step; a value channel belongs to SPLIT adjacent lanes with DPT key channels each.
// A block that holds a whole head also divides the head's o by its root mean square, multiplies by a weight and by
// g * sigmoid(g), and writes the row that the output projection reads.
//
// Long runs go by chunks, further below.
#include "chunk_mma.cuh"
#include "common.cuh"

namespace bt {

constexpr int GS_TOKENS = 16;  // tokens staged in shared memory at a time

// exp for decays: the special-function unit's form beside bfloat16 rows, the library's beside 32-bit rows
template <typename T> __device__ __forceinline__ float gla_exp(float x) { return __expf(x); }
template <> __device__ __forceinline__ float gla_exp<float>(float x) { return expf(x); }

struct GlaNorm {               // weight null: the block leaves o in `out`
  const float* weight;         // [vdim], shared by the heads
  float eps;
  int g_off;
  void* mixed;
  long long mixed_row_stride;
};

template <typename T, int DPT, int SPLIT>
__global__ void __launch_bounds__(512)
gla_scan_kernel(const T* __restrict__ proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale,
                const float* __restrict__ dt, float log_scale, float* __restrict__ state, const int* __restrict__ slots,
                const int* __restrict__ seq_start, float* __restrict__ out, long long out_row_stride, int n_heads, int dim,
                int vdim, int cols, GlaNorm norm) {
  extern __shared__ float sm[];
  float* q_s = sm;                          // [GS_TOKENS][dim]
  float* k_s = q_s + GS_TOKENS * dim;       // [GS_TOKENS][dim]
  float* a_s = k_s + GS_TOKENS * dim;       // [GS_TOKENS][dim]
  float* v_s = a_s + GS_TOKENS * dim;       // [GS_TOKENS][cols]; with a norm, o takes its place
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * cols;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  const int part = threadIdx.x % SPLIT, col_local = threadIdx.x / SPLIT;
  const int col = col0 + col_local;
  const bool owns = col_local < cols && col < vdim;
  const int d0 = part * DPT;
  float* s_base = state + (((long long)slots[seq] * n_heads + head) * dim) * vdim;
  float s[DPT];
#pragma unroll
  for (int i = 0; i < DPT; ++i) s[i] = owns && d0 + i < dim ? s_base[(long long)(d0 + i) * vdim + col] : 0.f;
  for (int t0 = 0; t0 < n_new; t0 += GS_TOKENS) {
    const int nt = min(GS_TOKENS, n_new - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < nt * dim; i += blockDim.x) {
      const int t = i / dim, d = i - t * dim;
      const long long row = first + t0 + t;
      const T* src = proj + row * row_stride + (long long)head * dim + d;
      q_s[i] = to_float(src[q_off]) * q_scale;
      k_s[i] = to_float(src[k_off]);
      a_s[i] = gla_exp<T>(dt[(row * n_heads + head) * dim + d] * log_scale);
    }
    for (int i = threadIdx.x; i < nt * cols; i += blockDim.x) {
      const int t = i / cols, c = i - t * cols;
      v_s[i] = col0 + c < vdim
                   ? to_float(proj[(long long)(first + t0 + t) * row_stride + v_off + (long long)head * vdim + col0 + c]) : 0.f;
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      const float v = col_local < cols ? v_s[t * cols + col_local] : 0.f;
      const float* kt = k_s + t * dim + d0;
      const float* qt = q_s + t * dim + d0;
      const float* at = a_s + t * dim + d0;
      float o = 0.f;
#pragma unroll
      for (int i = 0; i < DPT; ++i) {
        if (d0 + i < dim) {
          s[i] = fmaf(at[i], s[i], kt[i] * v);
          o = fmaf(s[i], qt[i], o);
        }
      }
#pragma unroll
      for (int x = 1; x < SPLIT; x <<= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
      if (owns && part == 0) {
        // (a column's v of this token was read by its own lanes above, before the shuffles)
        if (norm.weight != nullptr) v_s[t * cols + col_local] = o;
        else out[(long long)(first + t0 + t) * out_row_stride + (long long)head * vdim + col] = o;
      }
    }
    if (norm.weight != nullptr) {
      __syncthreads();
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
      for (int t = warp; t < nt; t += n_warps) {
        const float* o_s = v_s + t * cols;
        float ss = 0.f;
        for (int c = lane; c < vdim; c += 32) ss = fmaf(o_s[c], o_s[c], ss);
        const float inv = 1.f / sqrtf(warp_sum(ss) / (float)vdim + norm.eps);
        const long long row = first + t0 + t;
        const T* g = proj + row * row_stride + norm.g_off + (long long)head * vdim;
        T* dst = reinterpret_cast<T*>(norm.mixed) + row * norm.mixed_row_stride + (long long)head * vdim;
        for (int c = lane; c < vdim; c += 32) {
          const float gate = to_float(g[c]);
          dst[c] = from_float<T>(o_s[c] * inv * norm.weight[c] * (gate / (1.f + expf(-gate))));
        }
      }
    }
  }
  if (owns) {
#pragma unroll
    for (int i = 0; i < DPT; ++i)
      if (d0 + i < dim) s_base[(long long)(d0 + i) * vdim + col] = s[i];
  }
}

// lanes a value channel is spread over
static inline int gla_split(int dim) { return dim <= 128 ? 4 : 8; }
static inline bool gla_holds_head(int dim, int vdim) { return gla_split(dim) * vdim <= 512; }

template <typename T>
static int launch_gla_scan(const T* proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale, const float* dt,
                           float log_scale, float* state, const int* slots, const int* seq_start, float* out,
                           long long out_row_stride, int n_seqs, int n_heads, int dim, int vdim, const GlaNorm& norm,
                           cudaStream_t stream) {
  const int split = gla_split(dim);
  int cols = vdim;
  if (!gla_holds_head(dim, vdim)) cols = 512 / split;
  else if (norm.weight == nullptr && cols > 64) cols = 64;        // (more blocks where nothing asks for a whole head)
  const int threads = (split * cols + 31) / 32 * 32;
  const dim3 grid((vdim + cols - 1) / cols, n_heads, n_seqs), block(threads);
  const size_t smem = (size_t)GS_TOKENS * (3 * dim + cols) * sizeof(float);
#define BT_GS(DPT, SPLIT)                                                                                              \
  do {                                                                                                                 \
    auto kernel = gla_scan_kernel<T, DPT, SPLIT>;                                                                      \
    if (smem > 48 * 1024)                                                                                              \
      BT_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess,    \
               "gla_scan: cannot reserve %zu bytes of shared memory", smem);                                           \
    BT_PDL_OK("gla_scan", launch_pdl(kernel, grid, block, smem, stream, 1, proj, row_stride, q_off, k_off, v_off, q_scale, \
                                     dt, log_scale, state, slots, seq_start, out, out_row_stride, n_heads, dim, vdim, cols, \
                                     norm));                                                                           \
  } while (0)
  if (dim <= 32) BT_GS(8, 4);
  else if (dim <= 64) BT_GS(16, 4);
  else if (dim <= 128) BT_GS(32, 4);
  else BT_GS(32, 8);
#undef BT_GS
  return 0;
}

// ---- long runs of new tokens: the same recurrence by chunks ------------------------------------------------------
//
// Let b_t be the sum of the log decays up to token t since the chunk's first token (a number per key channel, falling).
// Unrolled over a chunk that starts from S_in,
//
//     o_t   = (q_t e^{b_t})^T S_in + sum_{s <= t} (sum_d q_t[d] k_s[d] e^{b_t[d] - b_s[d]}) v_s
//     S_out = diag(e^{b_end}) S_in + sum_s (k_s e^{b_end - b_s}) v_s^T
//
// e^{-b_s} alone may overflow, so no weight is formed as a quotient: the chunk's 64 tokens lie in 16 groups of four, B_g is
// b at the start of group g, and a weight between groups is the product of three factors that are each at most one,
// e^{b_t - B_g(t)} (kept with q), e^{B_g(t) - B_(g(s)+1)} (formed per pair of groups and channel) and e^{B_(g(s)+1) - b_s}
// (kept with k); inside a group the weights are products of one to three decays.  gla_chunk_kernel forms, per chunk, the
// sums over s, the chunk's own contribution to the state, e^{b_end}, and q_t e^{b_t}; gla_prefix_kernel walks a sequence's
// chunks; gla_carry_kernel adds the incoming state's part.  All 32-bit multiply-adds.  What bounds these kernels is the way
// into and out of shared memory: rows are read and results written 16 bytes a lane where they lie on such boundaries (`vec`),
// the state's product reads four tokens of a channel at once, B's rows have an odd length (with rows of 64, eight groups'
// numbers of a channel lay in one bank).  2 x 1,024 tokens of 16 heads of 64 x 64 in a recorded layer: 63 + 8 + 20 us before,
// 42 + 8 + 15 now.

constexpr int GC = 64;     // tokens a chunk
constexpr int GCP = 68;    // row length of the transposed tiles ([channel][token])
constexpr int GG = GC / 4; // groups of four tokens

// grid (chunks, heads * column blocks, sequences); 256 threads; a block owns 64 value channels.
template <typename T>
__global__ void __launch_bounds__(256)
gla_chunk_kernel(const T* __restrict__ proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale,
                 const float* __restrict__ dt, float log_scale, const int* __restrict__ seq_start, float* __restrict__ out,
                 long long out_row_stride, float* __restrict__ states, float* __restrict__ ends, float* __restrict__ aged_q,
                 int max_chunks, int n_heads, int dim, int vdim, int col_blocks, int vec) {
  extern __shared__ __align__(16) float sm[];
  float* q_t = sm;                       // [dim][GCP]   q_t e^{b_t - B_g(t)}
  float* k_t = q_t + dim * GCP;          // [dim][GCP]   k_s e^{B_(g(s)+1) - b_s}; then k_s e^{b_end - b_s}
  float* v_s = k_t + dim * GCP;          // [GC][64]
  float* a_t = v_s + GC * 64;            // [GC][GCP]    a_t[s][t]: token t's weight on token s
  float* bs = a_t + GC * GCP;            // [GG + 1][bsp]  B_0 .. B_16
  const int bsp = dim | 1;               // (an odd row length: a channel's numbers of several groups lie in several banks)
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col_block = blockIdx.y - head * col_blocks, col0 = col_block * 64;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * GC >= n_new) return;
  const int len = min(GC, n_new - chunk * GC);
  const long long row0 = first + (long long)chunk * GC;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, warp = tid >> 5, lane = tid & 31;
  constexpr int V = 16 / (int)sizeof(T);
  if (vec) {
#pragma unroll 2
    for (int i = tid; i < GC * 64 / V; i += 256) {
      const int t = i / (64 / V), c = i % (64 / V) * V;
      float x[V];
      unpack16(t < len && col0 + c < vdim
                   ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * row_stride + v_off + (long long)head * vdim + col0 + c))
                   : make_uint4(0u, 0u, 0u, 0u), x);
#pragma unroll
      for (int u = 0; u < V; u += 4) *reinterpret_cast<float4*>(v_s + t * 64 + c + u) = make_float4(x[u], x[u + 1], x[u + 2], x[u + 3]);
    }
  } else {
    for (int i = tid; i < GC * 64; i += 256) {
      const int t = i >> 6, c = i & 63;
      v_s[i] = (t < len && col0 + c < vdim)
                   ? to_float(proj[(row0 + t) * row_stride + v_off + (long long)head * vdim + col0 + c]) : 0.f;
    }
  }
  // a warp takes two groups, a lane a channel: the groups' q, k and decays, and the weights inside a group (both groups'
  // numbers are asked for before either's are used)
  {
    float w[2][10] = {};
    for (int d = lane; d < dim; d += 32) {
      float q[2][4], k[2][4], la[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = 4 * (2 * warp + h) + i;
          q[h][i] = k[h][i] = la[h][i] = 0.f;
          if (t < len) {
            const T* src = proj + (row0 + t) * row_stride + (long long)head * dim + d;
            q[h][i] = to_float(src[q_off]);
            k[h][i] = to_float(src[k_off]);
            la[h][i] = dt[((row0 + t) * n_heads + head) * dim + d];
          }
        }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int g = 2 * warp + h;
        float a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          q[h][i] *= q_scale;
          la[h][i] *= log_scale;
          a[i] = gla_exp<T>(la[h][i]);
        }
        bs[(g + 1) * bsp + d] = (la[h][0] + la[h][1]) + (la[h][2] + la[h][3]);
        const float a12 = a[1] * a[2], a23 = a[2] * a[3], a123 = a12 * a[3];
        const float(&qh)[4] = q[h];
        const float(&kh)[4] = k[h];
        w[h][0] = fmaf(qh[0], kh[0], w[h][0]);
        w[h][1] = fmaf(qh[1], kh[1], w[h][1]);
        w[h][2] = fmaf(qh[2], kh[2], w[h][2]);
        w[h][3] = fmaf(qh[3], kh[3], w[h][3]);
        w[h][4] = fmaf(qh[1], kh[0] * a[1], w[h][4]);
        w[h][5] = fmaf(qh[2], kh[1] * a[2], w[h][5]);
        w[h][6] = fmaf(qh[3], kh[2] * a[3], w[h][6]);
        w[h][7] = fmaf(qh[2], kh[0] * a12, w[h][7]);
        w[h][8] = fmaf(qh[3], kh[1] * a23, w[h][8]);
        w[h][9] = fmaf(qh[3], kh[0] * a123, w[h][9]);
        const float p1 = a[0] * a[1], p2 = p1 * a[2], p3 = p2 * a[3];
        *reinterpret_cast<float4*>(q_t + d * GCP + 4 * g) = make_float4(qh[0] * a[0], qh[1] * p1, qh[2] * p2, qh[3] * p3);
        *reinterpret_cast<float4*>(k_t + d * GCP + 4 * g) = make_float4(kh[0] * a123, kh[1] * a23, kh[2] * a[3], kh[3]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 0; i < 10; ++i) w[h][i] = warp_sum(w[h][i]);
      if (lane == 0) {
        float* cell = a_t + 4 * (2 * warp + h) * GCP + 4 * (2 * warp + h);      // [s][t]
        *reinterpret_cast<float4*>(cell) = make_float4(w[h][0], w[h][4], w[h][7], w[h][9]);
        *reinterpret_cast<float4*>(cell + GCP) = make_float4(0.f, w[h][1], w[h][5], w[h][8]);
        *reinterpret_cast<float4*>(cell + 2 * GCP) = make_float4(0.f, 0.f, w[h][2], w[h][6]);
        *reinterpret_cast<float4*>(cell + 3 * GCP) = make_float4(0.f, 0.f, 0.f, w[h][3]);
      }
    }
  }
  __syncthreads();
  for (int d = tid; d < dim; d += 256) {
    float sum = 0.f;
    bs[d] = 0.f;
    for (int g = 1; g <= GG; ++g) {
      sum += bs[g * bsp + d];
      bs[g * bsp + d] = sum;
    }
    if (col_block == 0) ends[(((long long)seq * max_chunks + chunk) * n_heads + head) * dim + d] = gla_exp<T>(sum);
  }
  __syncthreads();
  if (col_block == 0)
    for (int i = tid; i < len * dim; i += 256) {
      const int t = i / dim, d = i - t * dim;
      aged_q[((row0 + t) * n_heads + head) * dim + d] = q_t[d * GCP + t] * gla_exp<T>(bs[(t >> 2) * bsp + d]);
    }
  // weights between groups: 120 pairs (later group gt, earlier group gs), each shared by two threads with half of the channels
  {
    const int pair = tid & 127, half = tid >> 7;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    int gt = 1;
    while (gt < GG - 1 && (gt + 1) * gt / 2 <= pair) ++gt;
    const int gs = pair - gt * (gt - 1) / 2;
    const bool live = pair < GG * (GG - 1) / 2 && 4 * gt < len;
    float* cell = a_t + 4 * gs * GCP + 4 * gt;
    if (live) {
      const int d_mid = (dim + 1) / 2, d_end = half ? dim : d_mid;
      const float* bt_ = bs + gt * bsp;
      const float* bq = bs + (gs + 1) * bsp;
      for (int d = half ? d_mid : 0; d < d_end; ++d) {
        const float f = gla_exp<T>(bt_[d] - bq[d]);
        const float4 qv = *reinterpret_cast<const float4*>(q_t + d * GCP + gt * 4);
        const float4 kv = *reinterpret_cast<const float4*>(k_t + d * GCP + gs * 4);
        const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ka[4] = {kv.x * f, kv.y * f, kv.z * f, kv.w * f};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(qa[i], ka[j], acc[i][j]);
      }
      if (half)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<float4*>(cell + j * GCP) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
    }
    __syncthreads();
    if (live && !half) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float4* at = reinterpret_cast<float4*>(cell + j * GCP);
        const float4 o = *at;
        *at = make_float4(acc[0][j] + o.x, acc[1][j] + o.y, acc[2][j] + o.z, acc[3][j] + o.w);
      }
    }
  }
  __syncthreads();
  // k_s e^{b_end - b_s}
  for (int i = tid; i < GG * dim; i += 256) {
    const int g = i / dim, d = i - g * dim;
    const float f = gla_exp<T>(bs[GG * bsp + d] - bs[(g + 1) * bsp + d]);
    float4* at = reinterpret_cast<float4*>(k_t + d * GCP + 4 * g);
    const float4 kv = *at;
    *at = make_float4(kv.x * f, kv.y * f, kv.z * f, kv.w * f);
  }
  // the part of o_t that needs no earlier chunk: tokens 4 ty .., channels 4 tx ..
  {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int s_end = ty * 4 < len ? min(len, ty * 4 + 4) : 0;
    for (int sx = 0; sx < s_end; ++sx) {
      const float4 av = *reinterpret_cast<const float4*>(a_t + sx * GCP + ty * 4);
      const float4 vv = *reinterpret_cast<const float4*>(v_s + sx * 64 + tx * 4);
      const float aa[4] = {av.x, av.y, av.z, av.w}, va[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(aa[i], va[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ty * 4 + i;
      if (t >= len) break;
      float* o = out + (row0 + t) * out_row_stride + (long long)head * vdim + col0 + tx * 4;
      if (vec) {
        if (col0 + tx * 4 < vdim) *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col0 + tx * 4 + j < vdim) o[j] = acc[i][j];
    }
  }
  __syncthreads();
  // the chunk's contribution to the state, key channels 4 ty .. (+ 64, ...)
  float* dst = states + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim;
  for (int i0 = ty * 4; i0 < dim; i0 += 64) {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int sx = 0; sx < len; sx += 4) {
      // (tokens past the chunk's last one are zeros in both tiles)
      float kw[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 kv = i0 + i < dim ? *reinterpret_cast<const float4*>(k_t + (i0 + i) * GCP + sx) : make_float4(0.f, 0.f, 0.f, 0.f);
        kw[i][0] = kv.x; kw[i][1] = kv.y; kw[i][2] = kv.z; kw[i][3] = kv.w;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 vv = *reinterpret_cast<const float4*>(v_s + (sx + u) * 64 + tx * 4);
        const float va[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(kw[i][u], va[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i0 + i >= dim) break;
      float* o = dst + (long long)(i0 + i) * vdim + col0 + tx * 4;
      if (vec) {
        if (col0 + tx * 4 < vdim) *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col0 + tx * 4 + j < vdim) o[j] = acc[i][j];
    }
  }
}

// One thread per (sequence, head, state element): walks the sequence's chunks in order; leaves in states[chunk] the state
// that chunk STARTS from and in `state` the state after the last one.  Four chunks are asked for at a time.
__global__ void __launch_bounds__(256)
gla_prefix_kernel(float* states, const float* __restrict__ ends, float* __restrict__ state, const int* __restrict__ slots,
                  const int* __restrict__ seq_start, int max_chunks, int n_heads, int dim, int vdim) {
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y;
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e >= dim * vdim) return;
  const int n_new = seq_start[seq + 1] - seq_start[seq];
  const int n_chunks = (n_new + GC - 1) / GC;
  float* st = state + (((long long)slots[seq] * n_heads + head) * dim) * vdim + e;
  const long long stride = (long long)n_heads * dim * vdim, end_stride = (long long)n_heads * dim;
  float* cell = states + (((long long)seq * max_chunks) * n_heads + head) * (long long)dim * vdim + e;
  const float* end = ends + ((long long)seq * max_chunks * n_heads + head) * dim + e / vdim;
  float s = *st;
  for (int c = 0; c < n_chunks; c += 4) {
    float kv[4], decay[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      kv[u] = c + u < n_chunks ? __ldcg(cell + (c + u) * stride) : 0.f;
      decay[u] = c + u < n_chunks ? end[(c + u) * end_stride] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c + u < n_chunks) {
        cell[(c + u) * stride] = s;
        s = fmaf(decay[u], s, kv[u]);
      }
    }
  }
  *st = s;
}

// out[t] += (q_t e^{b_t})^T S_in for the tokens of a chunk; grid and blocks as gla_chunk_kernel.
__global__ void __launch_bounds__(256)
gla_carry_kernel(const float* __restrict__ aged_q, const int* __restrict__ seq_start, float* __restrict__ out,
                 long long out_row_stride, const float* __restrict__ states, int max_chunks, int n_heads, int dim, int vdim,
                 int col_blocks, int vec) {
  extern __shared__ __align__(16) float sm[];
  float* q_t = sm;                 // [dim][GCP]
  float* s_s = q_t + dim * GCP;    // [dim][64]
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col0 = (blockIdx.y - head * col_blocks) * 64;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * GC >= n_new) return;
  const int len = min(GC, n_new - chunk * GC);
  const long long row0 = first + (long long)chunk * GC;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const float* src = states + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim + col0;
  if (vec) {      // (a warp's lanes are 32 tokens, whose numbers meet all banks when they are written channel by channel)
#pragma unroll 4
    for (int i = tid; i < dim / 4 * GC; i += 256) {
      const int t = i % GC, d = i / GC * 4;
      const float4 x = t < len ? *reinterpret_cast<const float4*>(aged_q + ((row0 + t) * n_heads + head) * dim + d) : make_float4(0.f, 0.f, 0.f, 0.f);
      q_t[d * GCP + t] = x.x;
      q_t[(d + 1) * GCP + t] = x.y;
      q_t[(d + 2) * GCP + t] = x.z;
      q_t[(d + 3) * GCP + t] = x.w;
    }
#pragma unroll 4
    for (int i = tid; i < dim * 16; i += 256) {
      const int d = i >> 4, c = (i & 15) * 4;
      *reinterpret_cast<float4*>(s_s + d * 64 + c) =
          col0 + c < vdim ? *reinterpret_cast<const float4*>(src + (long long)d * vdim + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
    for (int i = tid; i < GC * dim; i += 256) {
      const int t = i / dim, d = i - t * dim;
      q_t[d * GCP + t] = t < len ? aged_q[((row0 + t) * n_heads + head) * dim + d] : 0.f;
    }
    for (int i = tid; i < dim * 64; i += 256) {
      const int d = i >> 6, c = i & 63;
      s_s[i] = col0 + c < vdim ? src[(long long)d * vdim + c] : 0.f;
    }
  }
  __syncthreads();
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int d = 0; d < dim; ++d) {
    const float4 qv = *reinterpret_cast<const float4*>(q_t + d * GCP + ty * 4);
    const float4 sv = *reinterpret_cast<const float4*>(s_s + d * 64 + tx * 4);
    const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, sa[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(qa[i], sa[j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty * 4 + i;
    if (t >= len) break;
    float* o = out + (row0 + t) * out_row_stride + (long long)head * vdim + col0 + tx * 4;
    if (vec) {
      if (col0 + tx * 4 < vdim) {
        const float4 before = *reinterpret_cast<const float4*>(o);
        *reinterpret_cast<float4*>(o) = make_float4(before.x + acc[i][0], before.y + acc[i][1], before.z + acc[i][2], before.w + acc[i][3]);
      }
      continue;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (col0 + tx * 4 + j < vdim) o[j] += acc[i][j];
  }
}

// The chunks on tensor cores (chunk_mma.cuh), for heads of whole operand tiles up to 64 channels: first every chunk's contribution to the
// state (gla_state_kernel), then gla_prefix_vec_kernel, then all of o at once (gla_out_kernel), written once; no aged q in memory.
// The weights are products of factors of at most one as above, with sub-blocks of 16 tokens between the chunk and the groups of four:
// q_t e^{b_t - B} k_s e^{B - b_s}, B at the end of s's sub-block, is a product of matrices for every later sub-block; inside a
// sub-block the groups' weights are multiply-adds.  The kernels above are bound by shared memory; these by forming factors and parts.
// The kernels above / here, us, all three: 2 x 1,024 tokens of 16 heads of 64 x 64 73 / 44, one prompt of 700 of 12 heads 49 / 31; 32-bit rows
// 72 / 49 and 48 / 31; errors against 64 bits 1.6e-7 / 1.4e-7.  Heads of 128 channels leave two blocks a multiprocessor
// and took 121 where the kernels above take 104, 32-bit heads of 16 15.4 against 13.7.

// The numbers of a chunk's contribution to the state that are not finite, by multiply-adds (a call of its own: inside, it costs the kernel registers).
template <typename T>
__device__ __noinline__ void gla_plain_state(const T* k, const T* v, long long stride, const float* dt, long long dt_stride, float log_scale, int len,
                                             int dim, int cols, float* dst, int vdim) {
  for (int i = threadIdx.x; i < dim * cols; i += CM_THREADS) {
    const int d = i / cols, c = i - d * cols;
    float* at = dst + (long long)d * vdim + c;
    if (isfinite(*at)) continue;
    float x = 0.f, after = 0.f;
#pragma unroll 8
    for (int t = len - 1; t >= 0; --t) {
      x = fmaf(to_float(k[t * stride + d]) * gla_exp<T>(log_scale * after), to_float(v[t * stride + c]), x);
      after += dt[t * dt_stride + d];
    }
    *at = x;
  }
}

// A chunk's contribution to the state: sum_s (k_s e^{b_end - b_s}) v_s^T.  A thread takes two key channels of 16 tokens and adds the log
// decays up from the end.
template <typename T, int PARTS>
__global__ void __launch_bounds__(CM_THREADS, 4)
gla_state_kernel(const T* __restrict__ proj, long long row_stride, int k_off, int v_off, const float* __restrict__ dt, float log_scale,
                 const int* __restrict__ seq_start, float* __restrict__ states, float* __restrict__ ends, int max_chunks, int n_heads,
                 int dim, int vdim, int col_blocks) {
  extern __shared__ __align__(16) unsigned char cm_smem[];
  const int k_stride = dim + 8, k_part = CM_CHUNK * k_stride, v_part = CM_CHUNK * CM_ROW;
  __nv_bfloat16* k_s = reinterpret_cast<__nv_bfloat16*>(cm_smem);      // [3][64][dim + 8]
  __nv_bfloat16* v_s = k_s + 3 * k_part;                               // [PARTS][64][72]
  float2* sums = reinterpret_cast<float2*>(v_s + PARTS * v_part);      // [4][dim / 2] of 16 tokens each
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col_block = blockIdx.y - head * col_blocks, col0 = col_block * CM_COLS;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * CM_CHUNK >= n_new) return;
  const int len = min(CM_CHUNK, n_new - chunk * CM_CHUNK), pairs = dim / 2;
  const long long row0 = first + (long long)chunk * CM_CHUNK;
  const T* rows = proj + row0 * row_stride;
  const float* dt_rows = dt + (row0 * n_heads + head) * dim;
  const long long dt_stride = (long long)n_heads * dim;
  // (at most 64 channels: a pair of channels and a quarter of the tokens a thread.  A token past the last one: the last one's
  // numbers, so that all reads are asked for together)
  const int quarter = threadIdx.x / pairs, d = (threadIdx.x - quarter * pairs) * 2;
  float2 x[16], k[16];
  if (quarter < 4) {
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const long long t = min(quarter * 16 + i, len - 1);
      x[i] = *reinterpret_cast<const float2*>(dt_rows + t * dt_stride + d);
      k[i] = cm_load2(rows + t * row_stride + k_off + head * dim + d);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (quarter * 16 + i >= len) x[i] = k[i] = make_float2(0.f, 0.f);
      sum.x += x[i].x;
      sum.y += x[i].y;
    }
    sums[threadIdx.x] = sum;
  }
  cm_fill<PARTS>(v_s, CM_CHUNK, CM_COLS, CM_ROW, v_part, [&](int t, int c, float (&y)[8]) {
    const bool in = t < len && col0 + c < vdim;
    if (in) cm_load8(rows + t * row_stride + v_off + head * vdim + col0 + c, y);
#pragma unroll
    for (int u = 0; u < 8; ++u) y[u] = in ? y[u] : 0.f;
  });
  __syncthreads();
  if (quarter < 4) {
    float2 after = make_float2(0.f, 0.f);      // of the tokens behind the one in hand
    for (int h = quarter + 1; h < 4; ++h) {
      const float2 y = sums[h * pairs + d / 2];
      after.x += y.x;
      after.y += y.y;
    }
    if (quarter == 0 && col_block == 0) {
      const float2 y = sums[d / 2];
      *reinterpret_cast<float2*>(ends + (((long long)seq * max_chunks + chunk) * n_heads + head) * dim + d) =
          make_float2(gla_exp<T>(log_scale * (y.x + after.x)), gla_exp<T>(log_scale * (y.y + after.y)));
    }
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      unsigned part[3];
      cm_split<3>(k[i].x * gla_exp<T>(log_scale * after.x), k[i].y * gla_exp<T>(log_scale * after.y), part);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<unsigned*>(k_s + q * k_part + (quarter * 16 + i) * k_stride + d) = part[q];
      after.x += x[i].x;
      after.y += x[i].y;
    }
  }
  __syncthreads();
  float* dst = states + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim + col0;
  const bool bad = cm_state<3, PARTS>(k_s, k_stride, k_part, v_s, v_part, dim, [&](int c, int at, float a, float b) {
    if (col0 + at < vdim) *reinterpret_cast<float2*>(dst + (long long)c * vdim + at) = make_float2(a, b);
  });
  if (__syncthreads_or(bad))
    gla_plain_state<T>(rows + k_off + head * dim, rows + v_off + head * vdim + col0, row_stride, dt_rows, dt_stride, log_scale, len, dim,
                       min(CM_COLS, vdim - col0), dst, vdim);
}

// gla_prefix_kernel with four value channels a thread and eight chunks asked for at a time.
__global__ void __launch_bounds__(128)
gla_prefix_vec_kernel(float* states, const float* __restrict__ ends, float* __restrict__ state, const int* __restrict__ slots,
                      const int* __restrict__ seq_start, int max_chunks, int n_heads, int dim, int vdim) {
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y, e = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (e >= dim * vdim) return;
  const int n_chunks = (seq_start[seq + 1] - seq_start[seq] + GC - 1) / GC;
  float4* st = reinterpret_cast<float4*>(state + (((long long)slots[seq] * n_heads + head) * dim) * vdim + e);
  const long long stride = (long long)n_heads * dim * vdim / 4, end_stride = (long long)n_heads * dim;
  float4* cell = reinterpret_cast<float4*>(states + (((long long)seq * max_chunks) * n_heads + head) * (long long)dim * vdim + e);
  const float* end = ends + ((long long)seq * max_chunks * n_heads + head) * dim + e / vdim;
  float4 s = *st;
  for (int c = 0; c < n_chunks; c += 8) {
    float4 kv[8];
    float decay[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      kv[u] = c + u < n_chunks ? __ldcg(cell + (c + u) * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
      decay[u] = c + u < n_chunks ? end[(c + u) * end_stride] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (c + u >= n_chunks) break;
      cell[(c + u) * stride] = s;
      s = make_float4(fmaf(decay[u], s.x, kv[u].x), fmaf(decay[u], s.y, kv[u].y), fmaf(decay[u], s.z, kv[u].z), fmaf(decay[u], s.w, kv[u].w));
    }
  }
  *st = s;
}

// N sums over lanes at once: lanes `from` apart and then nearer ones, down to `to` apart, hand each other half of their numbers; once a
// lane is left with one, x[0], the rest of the distances add it up.
template <int N>
__device__ __forceinline__ void gla_lane_sums(float (&x)[N], int from, int to) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = from, n = N / 2; o >= to; o >>= 1, n >>= 1) {
    const bool high = (lane & o) != 0;
    if (n == 0) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float give = high ? x[i] : x[i + n], keep = high ? x[i + n] : x[i];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
}

// The results of a chunk's tokens (bits of `redo`, from token `first_token` on) that are no finite numbers, by multiply-adds, a warp together, a lane
// two of the (at most 64) key channels: token by token back from a row's own, then the incoming state.  qk, v and dt are the chunk's rows
// from the head's channels on, v's and out's the block's.
template <typename T>
__device__ __noinline__ void gla_plain_rows(unsigned redo, const T* qk, const T* v, long long stride, int q_off, int k_off, float q_scale,
                                            const float* dt, long long dt_stride, float log_scale, const float* state, int vdim,
                                            int first_token, int dim, int cols, float* out, long long out_stride) {
  const int lane = threadIdx.x & 31;
  bool nan[2];
  cm_nan_columns(dim, cols, [&](int d, int c) { return state[(long long)d * vdim + c]; }, nan);
  for (; redo; redo &= redo - 1) {
    const int t = first_token + __ffs(redo) - 1;
    float* at = out + t * out_stride + lane;
    const bool need[2] = {!nan[0] && !isfinite(at[0]), !nan[1] && !isfinite(at[32])};
    if (!__any_sync(0xffffffffu, need[0] || need[1])) continue;
    float x[2] = {0.f, 0.f}, q[2], sum[2] = {0.f, 0.f};      // q, and what lies of dt between the token in hand and t
#pragma unroll
    for (int i = 0; i < 2; ++i) q[i] = lane + 32 * i < dim ? to_float(qk[t * stride + q_off + lane + 32 * i]) * q_scale : 0.f;
#pragma unroll 1
    for (int s = t; s >= 0; s -= 8) {      // (eight tokens', and eight channels', numbers are asked for at once)
      float k[8][2], a[8][2], y[8][2];
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int token = max(s - u, 0), c = lane + 32 * i;
          k[u][i] = c < dim ? to_float(qk[token * stride + k_off + c]) : 0.f;
          a[u][i] = c < dim ? dt[token * dt_stride + c] : 0.f;
          y[u][i] = c < cols ? to_float(v[token * stride + c]) : 0.f;
        }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float w = 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (lane + 32 * i < dim) w = fmaf(q[i] * gla_exp<T>(log_scale * sum[i]), k[u][i], w);
          sum[i] += s - u >= 0 ? a[u][i] : 0.f;
        }
        w = warp_sum(w);
        if (s - u < 0) break;
        x[0] = fmaf(w, y[u][0], x[0]);
        x[1] = fmaf(w, y[u][1], x[1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      q[i] *= gla_exp<T>(log_scale * sum[i]);
#pragma unroll 1
      for (int d = 32 * i; d < min(dim, 32 * i + 32); d += 8) {
        float y[8][2];
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) y[u][h] = lane + 32 * h < cols ? state[(long long)(d + u) * vdim + lane + 32 * h] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float z = __shfl_sync(0xffffffffu, q[i], (d + u) & 31);
          x[0] = fmaf(z, y[u][0], x[0]);
          x[1] = fmaf(z, y[u][1], x[1]);
        }
      }
    }
    if (need[0]) at[0] = x[0];
    if (need[1]) at[32] = x[1];
  }
}

constexpr int GD = 20;      // row length of a sub-block's weights ([token s][token t])
template <typename T, int PARTS>
__global__ void __launch_bounds__(CM_THREADS, 4)
gla_out_kernel(const T* __restrict__ proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale, const float* __restrict__ dt,
               float log_scale, const int* __restrict__ seq_start, float* __restrict__ out, long long out_row_stride,
               const float* __restrict__ states, int max_chunks, int n_heads, int dim, int vdim, int col_blocks, int held) {
  extern __shared__ __align__(16) unsigned char cm_smem[];
  float* q_t = reinterpret_cast<float*>(cm_smem);                      // [dim][GCP]   q_t e^{b_t - B_g(t)}
  float* k_t = q_t + dim * GCP;                                        // [dim][GCP]   k_s e^{B_(g(s)+1) - b_s}; in its place then
  const int k_stride = dim + 8, k_part = CM_CHUNK * k_stride, s_part = CM_CHUNK * CM_ROW;
  __nv_bfloat16* parts = reinterpret_cast<__nv_bfloat16*>(k_t);        // [3][64][dim + 8] k; [3][dim][72] the state; [PARTS][64][72] v
  float* bs = reinterpret_cast<float*>(cm_smem + held);                // [GG + 1][bsp]  B_0 .. B_16
  const int bsp = dim | 1;
  float* a_t = bs + (((GG + 1) * bsp + 3) & ~3);                       // [4][16][GD]  a sub-block's weights on itself
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col0 = (blockIdx.y - head * col_blocks) * CM_COLS;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * CM_CHUNK >= n_new) return;
  const int len = min(CM_CHUNK, n_new - chunk * CM_CHUNK);
  const long long row0 = first + (long long)chunk * CM_CHUNK;
  const T* rows = proj + row0 * row_stride;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // two groups of a warp at a time, a lane two channels: the groups' q, k and decays, and the weights inside a group
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    float w[2][16] = {};
    const int d = 2 * lane;
    if (d < dim) {
      float2 q[2][4], k[2][4], la[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // (a token past the last one: the last one's numbers, so that all reads are asked for together)
          const long long t = min(4 * (4 * warp + 2 * pass + h) + i, len - 1);
          const T* src = rows + t * row_stride + head * dim + d;
          q[h][i] = cm_load2(src + q_off);
          k[h][i] = cm_load2(src + k_off);
          la[h][i] = *reinterpret_cast<const float2*>(dt + ((row0 + t) * n_heads + head) * dim + d);
        }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int g = 4 * warp + 2 * pass + h;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (4 * g + i >= len) q[h][i] = k[h][i] = la[h][i] = make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float qh[4], kh[4], a[4], log_a[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            qh[i] = (u ? q[h][i].y : q[h][i].x) * q_scale;
            kh[i] = u ? k[h][i].y : k[h][i].x;
            log_a[i] = (u ? la[h][i].y : la[h][i].x) * log_scale;
            a[i] = gla_exp<T>(log_a[i]);
          }
          bs[(g + 1) * bsp + d + u] = (log_a[0] + log_a[1]) + (log_a[2] + log_a[3]);
          const float a12 = a[1] * a[2], a23 = a[2] * a[3], a123 = a12 * a[3];
          // (numbers 4 s + t of a cell of 4 x 4)
          w[h][0] = fmaf(qh[0], kh[0], w[h][0]);
          w[h][5] = fmaf(qh[1], kh[1], w[h][5]);
          w[h][10] = fmaf(qh[2], kh[2], w[h][10]);
          w[h][15] = fmaf(qh[3], kh[3], w[h][15]);
          w[h][1] = fmaf(qh[1], kh[0] * a[1], w[h][1]);
          w[h][6] = fmaf(qh[2], kh[1] * a[2], w[h][6]);
          w[h][11] = fmaf(qh[3], kh[2] * a[3], w[h][11]);
          w[h][2] = fmaf(qh[2], kh[0] * a12, w[h][2]);
          w[h][7] = fmaf(qh[3], kh[1] * a23, w[h][7]);
          w[h][3] = fmaf(qh[3], kh[0] * a123, w[h][3]);
          const float p1 = a[0] * a[1], p2 = p1 * a[2], p3 = p2 * a[3];
          *reinterpret_cast<float4*>(q_t + (d + u) * GCP + 4 * g) = make_float4(qh[0] * a[0], qh[1] * p1, qh[2] * p2, qh[3] * p3);
          *reinterpret_cast<float4*>(k_t + (d + u) * GCP + 4 * g) = make_float4(kh[0] * a123, kh[1] * a23, kh[2] * a[3], kh[3]);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      gla_lane_sums(w[h], 16, 1);      // (a lane pair's number: lane / 2)
      const int g = 2 * pass + h, number = lane >> 1;
      if ((lane & 1) == 0) a_t[(warp * 16 + 4 * g + number / 4) * GD + 4 * g + number % 4] = w[h][0];
    }
  }
  __syncthreads();
  if (tid < dim) {
    float sum = 0.f;
    bs[tid] = 0.f;
#pragma unroll
    for (int g = 1; g <= GG; ++g) {
      sum += bs[g * bsp + tid];
      bs[g * bsp + tid] = sum;
    }
  }
  __syncthreads();
  {
    // weights between the groups of a sub-block: 24 pairs (later group gt, earlier group gs), four lanes each with a quarter of the channels
    const int pair = min(tid >> 2, 23), block = pair / 6, r = pair - block * 6;
    const int later = r < 1 ? 1 : r < 3 ? 2 : 3, earlier = r - later * (later - 1) / 2, gt = 4 * block + later, gs = 4 * block + earlier;
    float acc[16] = {};
    const float* bt_ = bs + gt * bsp;
    const float* bq = bs + (gs + 1) * bsp;
#pragma unroll 4
    for (int d = tid & 3; d < dim; d += 4) {
      const float f = gla_exp<T>(bt_[d] - bq[d]);
      const float4 qv = *reinterpret_cast<const float4*>(q_t + d * GCP + gt * 4);
      const float4 kv = *reinterpret_cast<const float4*>(k_t + d * GCP + gs * 4);
      const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ka[4] = {kv.x * f, kv.y * f, kv.z * f, kv.w * f};
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[4 * j + i] = fmaf(qa[i], ka[j], acc[4 * j + i]);
    }
    gla_lane_sums(acc, 2, 1);      // (a lane's four numbers: those of token s = 4 gs + its place among the four)
    if (tid < 96)
      *reinterpret_cast<float4*>(a_t + (block * 16 + 4 * earlier + (tid & 3)) * GD + 4 * later) = make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
  {
    // k_s e^{B - b_s} with B at the end of s's sub-block, in parts (a thread's numbers wait in registers until k_t has been read)
    const int t = tid & 63, c0 = (tid >> 6) * 32, g = t >> 2, end = (t >> 4) * 4 + 4;
    const bool there = t < 48 && c0 < dim;      // (the last sub-block's weights on itself are all there is of it)
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int d = c0 + i;
      x[i] = there && d < dim ? k_t[d * GCP + t] * gla_exp<T>(bs[end * bsp + d] - bs[(g + 1) * bsp + d]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
      if (!there || c0 + i >= dim) break;
      unsigned part[4][3];
#pragma unroll
      for (int u = 0; u < 4; ++u) cm_split<3>(x[i + 2 * u], x[i + 2 * u + 1], part[u]);
#pragma unroll
      for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(parts + p * k_part + t * k_stride + c0 + i) = make_uint4(part[0][p], part[1][p], part[2][p], part[3][p]);
    }
  }
  __syncthreads();
  const int g = lane >> 2, t2 = (lane & 3) * 2, ta = warp * 16 + g, tb = ta + 8;      // this thread's rows
  // the operand of 16 channels from d on of q_t e^{b_t - B_ref}
  auto query = [&](int d, int ref, unsigned (&a)[3][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = i & 1 ? tb : ta, c = d + t2 + 8 * (i >> 1);
      const float* b = bs + (t >> 2) * bsp + c;
      const float* r = bs + ref * bsp + c;
      unsigned part[3];
      cm_split<3>(q_t[c * GCP + t] * gla_exp<T>(b[0] - r[0]), q_t[(c + 1) * GCP + t] * gla_exp<T>(b[1] - r[1]), part);
#pragma unroll
      for (int p = 0; p < 3; ++p) a[p][i] = part[p];
    }
  };
  float sc[8][4];      // the weights of this warp's tokens on those up to its last one
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float small[2][4] = {};
#pragma unroll
    for (int i = 0; i < 4; ++i) sc[2 * j][i] = sc[2 * j + 1][i] = 0.f;
    if (j < warp) {
      for (int d = 0; d < dim; d += 16) {
        unsigned a[3][4], b[3][4];
        query(d, 4 * j + 4, a);
        // (matrices: tokens 16 j.. of channels d.., of channels d + 8.., then tokens 16 j + 8..)
        const __nv_bfloat16* at = parts + (16 * j + (lane & 7) + (lane >> 4) * 8) * k_stride + d + (lane >> 3 & 1) * 8;
#pragma unroll
        for (int p = 0; p < 3; ++p) cm_ldmatrix(b[p], at + p * k_part);
        cm_products<3, 3>(sc[2 * j], small[0], sc[2 * j + 1], small[1], a, b);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sc[2 * j][i] += small[0][i];
        sc[2 * j + 1][i] += small[1][i];
      }
    } else if (j == warp) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = g + 8 * (i >> 1), at = 8 * h + t2 + (i & 1);
          sc[2 * j + h][i] = at <= t ? a_t[(warp * 16 + at) * GD + t] : 0.f;
        }
    }
  }
  __syncthreads();      // k has been read
  const float* src = states + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim + col0;
  cm_fill<3>(parts, dim, CM_COLS, CM_ROW, s_part, [&](int d, int c, float (&x)[8]) {
    if (col0 + c < vdim) cm_load8(src + (long long)d * vdim + c, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = col0 + c < vdim ? x[u] : 0.f;
  });
  __syncthreads();
  float o[8][4], o_small[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] = o_small[j][i] = 0.f;
  for (int d = 0; d < dim; d += 16) {
    unsigned a[3][4];
    query(d, 0, a);
    cm_step_rows<3, 3, 8>(o, o_small, a, parts, d, s_part);
  }
  __syncthreads();      // the state has been read
  cm_fill<PARTS>(parts, CM_CHUNK, CM_COLS, CM_ROW, s_part, [&](int t, int c, float (&x)[8]) {
    const bool in = t < len && col0 + c < vdim;
    if (in) cm_load8(rows + t * row_stride + v_off + head * vdim + col0 + c, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = in ? x[u] : 0.f;
  });
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {      // 16 tokens s at a time
    if (j > warp) break;
    unsigned a[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      unsigned part[3];
      cm_split<3>(sc[2 * j + (i >> 1)][2 * (i & 1)], sc[2 * j + (i >> 1)][2 * (i & 1) + 1], part);
#pragma unroll
      for (int p = 0; p < 3; ++p) a[p][i] = part[p];
    }
    cm_step_rows<3, PARTS, 8>(o, o_small, a, parts, 16 * j, s_part);
  }
  float zeros[2] = {0.f, 0.f};      // (zero times a row's numbers)
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 8 * j + t2;
    if (col0 + c >= vdim) break;
    float* at = out + row0 * out_row_stride + (long long)head * vdim + col0 + c;
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] += o_small[j][i];
    zeros[0] = fmaf(o[j][0] + o[j][1], 0.f, zeros[0]);
    zeros[1] = fmaf(o[j][2] + o[j][3], 0.f, zeros[1]);
    if (ta < len) *reinterpret_cast<float2*>(at + ta * out_row_stride) = make_float2(o[j][0], o[j][1]);
    if (tb < len) *reinterpret_cast<float2*>(at + tb * out_row_stride) = make_float2(o[j][2], o[j][3]);
  }
  const unsigned redo = cm_bad_rows(ta < len && zeros[0] != 0.f, tb < len && zeros[1] != 0.f);
  if (redo == 0) return;
  __syncwarp();
  gla_plain_rows<T>(redo, rows + head * dim, rows + v_off + head * vdim + col0, row_stride, q_off, k_off, q_scale, dt + (row0 * n_heads + head) * dim,
                    (long long)n_heads * dim, log_scale, src, vdim, warp * 16, dim, min(CM_COLS, vdim - col0),
                    out + row0 * out_row_stride + (long long)head * vdim + col0, out_row_stride);
}

// Scratch of the chunked form: [states | ends | aged_q].  (The kernels in parts leave aged_q as it is; which kernels take a call is known
// with its addresses only.)
static inline long long gla_state_floats(int n_seqs, int max_new, int n_heads, int dim, int vdim) {
  return (long long)n_seqs * ((max_new + GC - 1) / GC) * n_heads * dim * vdim;
}
static inline long long gla_end_floats(int n_seqs, int max_new, int n_heads, int dim) {
  return (long long)n_seqs * ((max_new + GC - 1) / GC) * n_heads * dim;
}

template <typename T, int PARTS>
static int launch_gla_mma(const T* proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale, const float* dt,
                          float log_scale, float* state, const int* slots, const int* seq_start, float* out, long long out_row_stride,
                          float* states, float* ends, int max_chunks, int n_seqs, int n_heads, int dim, int vdim, int col_blocks,
                          cudaStream_t stream) {
  const dim3 grid(max_chunks, n_heads * col_blocks, n_seqs), block(CM_THREADS);
  const size_t rows_k = 2 * 3 * (size_t)CM_CHUNK * (dim + 8), rows_v = 2 * (size_t)PARTS * CM_CHUNK * CM_ROW;
  const size_t smem_s = rows_k + rows_v + (size_t)2 * dim * sizeof(float2);
  // (k_t, the parts of k, of the state and of v lie in one place in turn; the state's are the longest)
  const size_t held = (size_t)dim * GCP * sizeof(float) + 2 * 3 * (size_t)CM_CHUNK * CM_ROW;
  const size_t smem_o = held + ((((size_t)(GG + 1) * (dim | 1) + 3) & ~(size_t)3) + 4 * 16 * GD) * sizeof(float);
  static SharedMemoryAllowance allowed_s, allowed_o;
  BT_CHECK(allow_shared_memory(allowed_s, gla_state_kernel<T, PARTS>, smem_s) && allow_shared_memory(allowed_o, gla_out_kernel<T, PARTS>, smem_o),
           "gla: cannot reserve %zu bytes of shared memory", smem_s > smem_o ? smem_s : smem_o);
  BT_PDL_OK("gla_state", launch_pdl(gla_state_kernel<T, PARTS>, grid, block, smem_s, stream, 1, proj, row_stride, k_off, v_off, dt,
                                    log_scale, seq_start, states, ends, max_chunks, n_heads, dim, vdim, col_blocks));
  if ((unsigned long long)state % 16 == 0)
    BT_PDL_OK("gla_prefix", launch_pdl(gla_prefix_vec_kernel, dim3((dim * vdim + 511) / 512, n_heads, n_seqs), dim3(128), 0, stream, 1, states,
                                       (const float*)ends, state, slots, seq_start, max_chunks, n_heads, dim, vdim));
  else
    BT_PDL_OK("gla_prefix", launch_pdl(gla_prefix_kernel, dim3((dim * vdim + 255) / 256, n_heads, n_seqs), dim3(256), 0, stream, 1, states,
                                       (const float*)ends, state, slots, seq_start, max_chunks, n_heads, dim, vdim));
  BT_PDL_OK("gla_out", launch_pdl(gla_out_kernel<T, PARTS>, grid, block, smem_o, stream, 1, proj, row_stride, q_off, k_off, v_off, q_scale,
                                  dt, log_scale, seq_start, out, out_row_stride, (const float*)states, max_chunks, n_heads, dim, vdim,
                                  col_blocks, (int)held));
  return 0;
}

template <typename T>
static int launch_gla_chunked(const T* proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale,
                              const float* dt, float log_scale, float* state, const int* slots, const int* seq_start,
                              float* out, long long out_row_stride, float* scratch, int max_new, int n_seqs, int n_heads,
                              int dim, int vdim, cudaStream_t stream) {
  const int col_blocks = (vdim + 63) / 64, max_chunks = (max_new + GC - 1) / GC;
  BT_CHECK((long long)n_heads * col_blocks <= 65535, "gla: %d heads x %d column blocks are too many", n_heads, col_blocks);
  const dim3 grid(max_chunks, n_heads * col_blocks, n_seqs), block(256);
  const size_t smem_a = ((size_t)2 * dim * GCP + (size_t)GC * 64 + (size_t)GC * GCP + (size_t)(GG + 1) * (dim | 1)) * sizeof(float);
  const size_t smem_c = ((size_t)dim * GCP + (size_t)dim * 64) * sizeof(float);
  auto chunk_kernel = gla_chunk_kernel<T>;
  if (smem_a > 48 * 1024)
    BT_CHECK(cudaFuncSetAttribute(chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_a) == cudaSuccess,
             "gla: cannot reserve %zu bytes of shared memory", smem_a);
  if (smem_c > 48 * 1024)
    BT_CHECK(cudaFuncSetAttribute(gla_carry_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_c) == cudaSuccess,
             "gla: cannot reserve %zu bytes of shared memory", smem_c);
  float* states = scratch;
  float* ends = states + gla_state_floats(n_seqs, max_new, n_heads, dim, vdim);
  float* aged_q = ends + gla_end_floats(n_seqs, max_new, n_heads, dim);
  // 16-byte accesses: every head of every row, of the results and of the scratch on such a boundary
  constexpr int V = 16 / (int)sizeof(T);
  const int vec = dim % 4 == 0 && vdim % V == 0 && v_off % V == 0 && row_stride % V == 0 && out_row_stride % 4 == 0 &&
                  ((unsigned long long)proj | (unsigned long long)out | (unsigned long long)states | (unsigned long long)aged_q) % 16 == 0;
  if (vec && dim % 16 == 0 && dim >= (sizeof(T) == 4 ? 32 : 16) && dim <= 64 && vdim % 8 == 0 && v_off % 8 == 0 && q_off % 2 == 0 &&
      k_off % 2 == 0 && row_stride % 8 == 0 && (unsigned long long)dt % 8 == 0 && (unsigned long long)ends % 8 == 0)
    return launch_gla_mma<T, sizeof(T) == 2 ? 1 : 3>(proj, row_stride, q_off, k_off, v_off, q_scale, dt, log_scale, state, slots, seq_start,
                                                     out, out_row_stride, states, ends, max_chunks, n_seqs, n_heads, dim, vdim, col_blocks,
                                                     stream);
  BT_PDL_OK("gla_chunk", launch_pdl(chunk_kernel, grid, block, smem_a, stream, 1, proj, row_stride, q_off, k_off, v_off, q_scale,
                                    dt, log_scale, seq_start, out, out_row_stride, states, ends, aged_q, max_chunks, n_heads,
                                    dim, vdim, col_blocks, vec));
  BT_PDL_OK("gla_prefix", launch_pdl(gla_prefix_kernel, dim3((dim * vdim + 255) / 256, n_heads, n_seqs), block, 0, stream, 1,
                                     states, (const float*)ends, state, slots, seq_start, max_chunks, n_heads, dim, vdim));
  BT_PDL_OK("gla_carry", launch_pdl(gla_carry_kernel, grid, block, smem_c, stream, 1, (const float*)aged_q, seq_start, out,
                                    out_row_stride, (const float*)states, max_chunks, n_heads, dim, vdim, col_blocks, vec));
  return 0;
}

}  // namespace bt

// Whether the token-by-token kernel holds a whole head of this size in one block (and can norm and gate it).
extern "C" int bt_gla_scan_fuses(int dim, int vdim) { return bt::gla_holds_head(dim, vdim) ? 1 : 0; }

// norm_weight (null: none): see GlaNorm; the read-out then goes to `mixed` (rows of proj's type) and `out` is not written.
extern "C" int bt_gla_scan(const void* proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale,
                           const float* dt, float log_scale, float* state, const int* slots, const int* seq_start, float* out,
                           long long out_row_stride, int n_seqs, int n_heads, int dim, int vdim, const float* norm_weight,
                           float eps, int g_off, void* mixed, long long mixed_row_stride, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && dim > 0 && dim <= 256 && vdim > 0 && n_seqs >= 0 && n_seqs <= 65535 && n_heads <= 65535,
           "gla_scan: bad sizes seqs=%d heads=%d dim=%d vdim=%d", n_seqs, n_heads, dim, vdim);
  BT_CHECK(norm_weight == nullptr || gla_holds_head(dim, vdim), "gla_scan: no block holds a head of %d x %d", dim, vdim);
  BT_CHECK(norm_weight != nullptr ? mixed != nullptr : out != nullptr, "gla_scan: nowhere to leave the result");
  if (n_seqs == 0) return 0;
  const GlaNorm norm{norm_weight, eps, g_off, mixed, mixed_row_stride};
  if (dtype == kF32)
    return launch_gla_scan<float>((const float*)proj, row_stride, q_off, k_off, v_off, q_scale, dt, log_scale, state, slots,
                                  seq_start, out, out_row_stride, n_seqs, n_heads, dim, vdim, norm, stream);
  if (dtype == kBF16)
    return launch_gla_scan<__nv_bfloat16>((const __nv_bfloat16*)proj, row_stride, q_off, k_off, v_off, q_scale, dt, log_scale,
                                          state, slots, seq_start, out, out_row_stride, n_seqs, n_heads, dim, vdim, norm, stream);
  return fail("gla_scan: unknown dtype %d", dtype);
}

// The same results as bt_gla_scan (beyond rounding), the chunks of a run worked side by side; `out` [tokens][heads vdim].
// scratch: (n_seqs * chunks of max_new) * n_heads * dim * (vdim + 1) + n_tokens * n_heads * dim floats.
extern "C" int bt_gla_chunked(const void* proj, long long row_stride, int q_off, int k_off, int v_off, float q_scale,
                              const float* dt, float log_scale, float* state, const int* slots, const int* seq_start,
                              float* out, long long out_row_stride, float* scratch, int max_new, int n_seqs, int n_heads,
                              int dim, int vdim, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && dim > 0 && dim <= 256 && vdim > 0 && n_seqs >= 0 && n_seqs <= 65535 && max_new > 0 && scratch,
           "gla_chunked: bad sizes seqs=%d heads=%d dim=%d vdim=%d max_new=%d", n_seqs, n_heads, dim, vdim, max_new);
  if (n_seqs == 0) return 0;
  if (dtype == kF32)
    return launch_gla_chunked<float>((const float*)proj, row_stride, q_off, k_off, v_off, q_scale, dt, log_scale, state, slots,
                                     seq_start, out, out_row_stride, scratch, max_new, n_seqs, n_heads, dim, vdim, stream);
  if (dtype == kBF16)
    return launch_gla_chunked<__nv_bfloat16>((const __nv_bfloat16*)proj, row_stride, q_off, k_off, v_off, q_scale, dt, log_scale,
                                             state, slots, seq_start, out, out_row_stride, scratch, max_new, n_seqs, n_heads, dim,
                                             vdim, stream);
  return fail("gla_chunked: unknown dtype %d", dtype);
}
