// A matrix memory with exponential gates, as a recurrence over a 32-bit state per (sequence, head):
//
//     a_t = cap tanh((x_i,t + bias_i) / cap)                      log of the input gate
//     b_t = log sigmoid(cap tanh((x_f,t + bias_f) / cap))         log of the forget gate
//     m_t = max(b_t + m_(t-1), a_t)                               running maximum (0 before the first token)
//     S_t = exp(b_t + m_(t-1) - m_t) S_(t-1) + exp(a_t - m_t) k_t v_t^T       (S: dim x vdim)
//     n_t = the same with k_t alone                                            (n: dim)
//     o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6)
//
// x_i, x_f, q, k, v are columns of the step's projections; q is scaled here (dim^-1/2 is handed in).  Everything
// from the gates on is 32-bit.  Columns of S (value channels) never mix, so a block owns a group of value channels of
// one (sequence, head) and keeps its part of S in registers for all tokens of the step; n and m are small and every
// block keeps its own copy (the block of the first channel group writes them back).  A value channel belongs to SPLIT
// adjacent lanes, each with DPT of the head's key channels; partial sums meet by shuffles.
// State: s[slot][head][dim][vdim], n[slot][head][dim], m[slot][head]; a sequence that starts finds zeros there.
#include "chunk_mma.cuh"
#include "common.cuh"

namespace bt {

constexpr int ML_TOKENS = 16;  // tokens staged in shared memory at a time

__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

struct MlstmArgs {
  long long row_stride;
  int q_off, k_off, v_off, i_off, f_off;
  const float* i_bias;
  const float* f_bias;
  float cap, q_scale;
  float* s;
  float* n;
  float* m;
  const int* slots;
  const int* seq_start;
  float* out;
  long long out_row_stride;
  int n_heads, dim, vdim, cols;
  // with `mixed`: a block holds all value channels of its head, and instead of o the kernel leaves
  // o / rms(o) * norm_w * sigmoid(gate) (the gate's channels at g_off of the rows of proj) in `mixed`, in proj's type
  const float* norm_w;
  float eps;
  int g_off;
  void* mixed;
  long long mixed_row_stride;
};

template <typename T, int DPT, int SPLIT>
__global__ void __launch_bounds__(256) mlstm_scan_kernel(const T* __restrict__ proj, MlstmArgs p) {
  extern __shared__ float sm[];
  const int dim = p.dim, vdim = p.vdim, cols = p.cols;
  float* q_s = sm;                            // [ML_TOKENS][dim]
  float* k_s = q_s + ML_TOKENS * dim;         // [ML_TOKENS][dim]
  float* v_s = k_s + ML_TOKENS * dim;         // [ML_TOKENS][cols]
  float* keep_s = v_s + ML_TOKENS * cols;     // [ML_TOKENS] exp(b + m_old - m_new)
  float* take_s = keep_s + ML_TOKENS;         // [ML_TOKENS] exp(a - m_new)
  float* floor_s = take_s + ML_TOKENS;        // [ML_TOKENS] exp(-m_new)
  float* red_s = floor_s + ML_TOKENS;         // [33] for sums over the block
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * cols;
  const int first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - first;
  const int part = threadIdx.x % SPLIT, col_local = threadIdx.x / SPLIT;
  const int col = col0 + col_local;
  const bool owns = col_local < cols && col < vdim;
  const int d0 = part * DPT;
  const long long slot_head = (long long)p.slots[seq] * p.n_heads + head;
  float* s_base = p.s + slot_head * dim * vdim;
  float* n_base = p.n + slot_head * dim;
  float s[DPT], nn[DPT];
#pragma unroll
  for (int i = 0; i < DPT; ++i) {
    s[i] = owns && d0 + i < dim ? s_base[(long long)(d0 + i) * vdim + col] : 0.f;
    nn[i] = d0 + i < dim ? n_base[d0 + i] : 0.f;
  }
  float m = p.m[slot_head];                   // (only thread 0's copy is advanced)
  const float bias_i = p.i_bias[head], bias_f = p.f_bias[head];
  for (int t0 = 0; t0 < n_new; t0 += ML_TOKENS) {
    const int nt = min(ML_TOKENS, n_new - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < nt * dim; i += blockDim.x) {
      const int t = i / dim, d = i - t * dim;
      const T* row = proj + (long long)(first + t0 + t) * p.row_stride + (long long)head * dim + d;
      q_s[i] = to_float(row[p.q_off]) * p.q_scale;
      k_s[i] = to_float(row[p.k_off]);
    }
    for (int i = threadIdx.x; i < nt * cols; i += blockDim.x) {
      const int t = i / cols, c = i - t * cols;
      v_s[i] = col0 + c < vdim
                   ? to_float(proj[(long long)(first + t0 + t) * p.row_stride + p.v_off + (long long)head * vdim + col0 + c])
                   : 0.f;
    }
    // the gates' nonlinearities side by side, then the running maximum token after token
    if (threadIdx.x < nt) {
      const T* row = proj + (long long)(first + t0 + threadIdx.x) * p.row_stride + head;
      keep_s[threadIdx.x] = log_sigmoid(p.cap * tanhf((to_float(row[p.f_off]) + bias_f) / p.cap));
      take_s[threadIdx.x] = p.cap * tanhf((to_float(row[p.i_off]) + bias_i) / p.cap);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int t = 0; t < nt; ++t) {
        const float b = keep_s[t], a = take_s[t];
        const float m_new = fmaxf(b + m, a);
        keep_s[t] = expf(b + m - m_new);
        take_s[t] = expf(a - m_new);
        floor_s[t] = expf(-m_new);
        m = m_new;
      }
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      const float v = col_local < cols ? v_s[t * cols + col_local] : 0.f;
      const float keep = keep_s[t], take = take_s[t];
      const float* kt = k_s + t * dim + d0;
      const float* qt = q_s + t * dim + d0;
      float o = 0.f, nq = 0.f;
#pragma unroll
      for (int i = 0; i < DPT; ++i) {
        if (d0 + i < dim) {
          const float tk = take * kt[i];
          s[i] = fmaf(keep, s[i], tk * v);
          nn[i] = fmaf(keep, nn[i], tk);
          o = fmaf(s[i], qt[i], o);
          nq = fmaf(nn[i], qt[i], nq);
        }
      }
#pragma unroll
      for (int x = 1; x < SPLIT; x <<= 1) {
        o += __shfl_xor_sync(0xffffffffu, o, x);
        nq += __shfl_xor_sync(0xffffffffu, nq, x);
      }
      const float read = o / (fmaxf(fabsf(nq), floor_s[t]) + 1e-6f);
      if (p.mixed) {
        const float ss = block_sum(owns && part == 0 ? read * read : 0.f, red_s);
        if (owns && part == 0) {
          const long long row = first + t0 + t;
          const int ch = head * vdim + col;
          const float gate = to_float(proj[row * p.row_stride + p.g_off + ch]);
          const float y = read / sqrtf(ss / (float)vdim + p.eps) * p.norm_w[ch] / (1.f + expf(-gate));
          reinterpret_cast<T*>(p.mixed)[row * p.mixed_row_stride + ch] = from_float<T>(y);
        }
      } else if (owns && part == 0) {
        p.out[(long long)(first + t0 + t) * p.out_row_stride + (long long)head * vdim + col] = read;
      }
    }
  }
  if (owns) {
#pragma unroll
    for (int i = 0; i < DPT; ++i)
      if (d0 + i < dim) s_base[(long long)(d0 + i) * vdim + col] = s[i];
  }
  if (blockIdx.x == 0 && col_local == 0) {
#pragma unroll
    for (int i = 0; i < DPT; ++i)
      if (d0 + i < dim) n_base[d0 + i] = nn[i];
    if (threadIdx.x == 0) p.m[slot_head] = m;
  }
}

template <typename T>
static int launch_mlstm(const T* proj, MlstmArgs p, int n_seqs, cudaStream_t stream) {
  // DPT key channels per lane, SPLIT lanes per value channel: SPLIT * DPT >= dim
  int dpt, split;
  if (p.dim <= 32) { dpt = 8; split = 4; }
  else if (p.dim <= 64) { dpt = 8; split = 8; }
  else if (p.dim <= 128) { dpt = 16; split = 8; }
  else { dpt = 32; split = 8; }
  if (p.mixed && p.vdim > 256 / split) {      // a whole head a block: 64 value channels, more key channels a lane
    split = 4;
    dpt = p.dim <= 64 ? 16 : 32;
  }
  p.cols = 256 / split < p.vdim ? 256 / split : p.vdim;   // value channels per block
  const dim3 grid((p.vdim + p.cols - 1) / p.cols, p.n_heads, n_seqs), block(256);
  BT_CHECK(!p.mixed || grid.x == 1, "mlstm_scan: a head of %d x %d does not fit one block, the norm cannot be fused", p.dim,
           p.vdim);
  const size_t smem = (size_t)(ML_TOKENS * (2 * p.dim + p.cols + 3) + 33) * sizeof(float);
#define BT_ML(DPT, SPLIT) \
  BT_PDL_OK("mlstm_scan", launch_pdl(mlstm_scan_kernel<T, DPT, SPLIT>, grid, block, smem, stream, 1, proj, p))
  if (dpt == 8 && split == 4) BT_ML(8, 4);
  else if (dpt == 8) BT_ML(8, 8);
  else if (dpt == 16 && split == 4) BT_ML(16, 4);
  else if (dpt == 32 && split == 4) BT_ML(32, 4);
  else if (dpt == 16) BT_ML(16, 8);
  else BT_ML(32, 8);
#undef BT_ML
  return 0;
}


// ---- long runs of new tokens: the same recurrence by chunks ------------------------------------------------------
//
// With c_t the sum of the forget gates' logs b from the chunk's first token to t, a chunk that starts from
// (S_in, n_in, m_in) has, for its tokens t and s <= t,
//
//     m_t   = max(c_t + m_in, max_s (c_t - c_s + a_s))                                 (the same m_t as token by token)
//     num_t = exp(c_t + m_in - m_t) S_in^T q_t + sum_s exp(c_t - c_s + a_s - m_t) (q_t . k_s) v_s
//     den_t = exp(c_t + m_in - m_t) n_in . q_t + sum_s exp(c_t - c_s + a_s - m_t) (q_t . k_s)
//     o_t   = num_t / (max(|den_t|, exp(-m_t)) + 1e-6)
//     S_out = exp(c_L + m_in - m_L) S_in + sum_s exp(c_L - c_s + a_s - m_L) k_s v_s^T      (L: the chunk's last token)
//
// and no exponent is above zero.  mlstm_gates_kernel forms a, c and m for every token (a warp scans the running maximum:
// the maps m -> max(m + b, a) compose); mlstm_chunk_kernel the sums over s per chunk, side by side; mlstm_prefix_kernel
// walks a sequence's chunks in order and leaves each the state it starts from; mlstm_carry_kernel adds the parts with
// S_in and n_in and divides.
constexpr int MC = 64;    // tokens per chunk
constexpr int MCP = 68;   // row length of the transposed tiles

struct MlstmChunked {
  // rows, results and cells lie on 16-byte boundaries, head by head: they are then read and written 16 bytes a lane, which is
  // what bounds these kernels (2 x 1,024 tokens of 16 heads of 64 x 64, beside other work: chunk 75 to 48 us, carry 37 to 29)
  int vec;
  MlstmArgs a;
  float* ga;       // [rows][heads] log input gate
  float* gc;       // [rows][heads] sum of the log forget gates since the chunk's first token
  float* gm;       // [rows][heads] running maximum
  float* den;      // [rows][heads] the chunk's own part of n . q
  float* m_start;  // [seqs][chunks][heads] maximum the chunk starts from
  float* carry;    // [seqs][chunks][heads] exp(c_L + m_in - m_L)
  float* ds;       // [seqs][chunks][heads][dim][vdim] contribution, then the state the chunk starts from
  float* dn;       // [seqs][chunks][heads][dim]
  int max_chunks, col_blocks;
};

constexpr int MG_TOKENS = 2048;   // tokens whose gates lie in shared memory at a time (a multiple of the chunk)

template <typename T>
__global__ void __launch_bounds__(256) mlstm_gates_kernel(const T* __restrict__ proj, MlstmChunked c) {
  __shared__ float a_s[MG_TOKENS], b_s[MG_TOKENS];
  const MlstmArgs& p = c.a;
  pdl_trigger();
  pdl_wait();
  const int head = blockIdx.x, seq = blockIdx.y, H = p.n_heads;
  const int first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - first;
  const float bias_i = p.i_bias[head], bias_f = p.f_bias[head];
  const int lane = threadIdx.x & 31;
  const long long slot_head = (long long)p.slots[seq] * H + head;
  float m = p.m[slot_head], m_in = m, sum = 0.f;       // (warp 0's copies are the ones that count)
  for (int base = 0; base < n_new; base += MG_TOKENS) {
    const int count = min(MG_TOKENS, n_new - base);
    __syncthreads();
    for (int t = threadIdx.x; t < count; t += blockDim.x) {
      const T* row = proj + (long long)(first + base + t) * p.row_stride + head;
      const float a = p.cap * tanhf((to_float(row[p.i_off]) + bias_i) / p.cap);
      a_s[t] = a;
      b_s[t] = log_sigmoid(p.cap * tanhf((to_float(row[p.f_off]) + bias_f) / p.cap));
      c.ga[(long long)(first + base + t) * H + head] = a;
    }
    __syncthreads();
    if (threadIdx.x >= 32) continue;
    for (int t0 = 0; t0 < count; t0 += 32) {
      const int chunk = (base + t0) / MC;
      const long long at = ((long long)seq * c.max_chunks + chunk) * H + head;
      if ((base + t0) % MC == 0) {
        sum = 0.f;
        m_in = m;
        if (lane == 0) c.m_start[at] = m;
      }
      const int t = t0 + lane;
      const bool valid = t < count;
      // the map of token t is m -> max(m + B, A); lanes past the run hold the identity
      float B = valid ? b_s[t] : 0.f, A = valid ? a_s[t] : -INFINITY;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float Bp = __shfl_up_sync(0xffffffffu, B, o), Ap = __shfl_up_sync(0xffffffffu, A, o);
        if (lane >= o) {
          A = fmaxf(Ap + B, A);
          B = Bp + B;
        }
      }
      const float m_t = fmaxf(m + B, A);
      if (valid) {
        const long long g = (long long)(first + base + t) * H + head;
        c.gc[g] = sum + B;
        c.gm[g] = m_t;
      }
      const int last = min(31, count - 1 - t0);
      m = __shfl_sync(0xffffffffu, m_t, last);
      sum += __shfl_sync(0xffffffffu, B, last);
      if (lane == 0 && ((base + t0 + 32) % MC == 0 || base + t0 + 32 >= n_new)) c.carry[at] = expf(sum + m_in - m);
    }
  }
  if (threadIdx.x == 0) p.m[slot_head] = m;
}

// grid (chunks, heads * column blocks, sequences); 256 threads as a 16 x 16 grid, thread (ty, tx) owns a 4 x 4 patch of
// every product; a block owns 64 value channels.  Tiles hold their 64 tokens along the fast axis.
template <typename T>
__global__ void __launch_bounds__(256) mlstm_chunk_kernel(const T* __restrict__ proj, MlstmChunked c) {
  const MlstmArgs& p = c.a;
  const int dim = p.dim, vdim = p.vdim, H = p.n_heads;
  extern __shared__ __align__(16) float sm[];
  float* q_t = sm;                       // [dim][MCP]   q_t[d][t]
  float* k_t = q_t + dim * MCP;          // [dim][MCP]   k_t[d][s]
  float* v_s = k_t + dim * MCP;          // [MC][64]     v_s[s][j]
  float* a_t = v_s + MC * 64;            // [MC][MCP]    a_t[s][t] = exp(c_t - c_s + a_s - m_t) (q_t . k_s), zero for s > t
  float* g_a = a_t + MC * MCP;           // [MC] a_s - c_s
  float* g_c = g_a + MC;                 // [MC] c_t - m_t
  float* w_end = g_c + MC;               // [MC] exp(c_L - c_s + a_s - m_L)
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / c.col_blocks, col_block = blockIdx.y - head * c.col_blocks, col0 = col_block * 64;
  const int first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - first;
  if (chunk * MC >= n_new) return;
  const int len = min(MC, n_new - chunk * MC);
  const long long row0 = first + (long long)chunk * MC;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  if (tid < MC) {
    float ga = 0.f, gc = 0.f, gm = 0.f;
    if (tid < len) {
      const long long g = (row0 + tid) * H + head;
      ga = c.ga[g]; gc = c.gc[g]; gm = c.gm[g];
    }
    const long long gl = (row0 + len - 1) * H + head;
    g_a[tid] = ga - gc;
    g_c[tid] = gc - gm;
    w_end[tid] = tid < len ? expf(c.gc[gl] - c.gm[gl] + ga - gc) : 0.f;
  }
  constexpr int V = 16 / (int)sizeof(T);
  if (c.vec) {      // (a warp's lanes are 32 tokens, whose numbers meet all banks when they are written channel by channel)
    const int groups = dim / V;
#pragma unroll 4
    for (int i = tid; i < 2 * groups * MC; i += 256) {
      const int t = i % MC, g = i / MC;                    // (q's groups of channels, then k's)
      const bool key = g >= groups;
      const int d = (key ? g - groups : g) * V;
      float x[V];
      unpack16(t < len ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * p.row_stride + (key ? p.k_off : p.q_off) + (long long)head * dim + d))
                       : make_uint4(0u, 0u, 0u, 0u), x);
      float* dst = (key ? k_t : q_t) + d * MCP + t;
      const float scale = key ? 1.f : p.q_scale;
#pragma unroll
      for (int u = 0; u < V; ++u) dst[u * MCP] = x[u] * scale;
    }
#pragma unroll 2
    for (int i = tid; i < MC * 64 / V; i += 256) {
      const int t = i / (64 / V), cc = i % (64 / V) * V;
      float x[V];
      unpack16(t < len && col0 + cc < vdim
                   ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * p.row_stride + p.v_off + (long long)head * vdim + col0 + cc))
                   : make_uint4(0u, 0u, 0u, 0u), x);
#pragma unroll
      for (int u = 0; u < V; u += 4) *reinterpret_cast<float4*>(v_s + t * 64 + cc + u) = make_float4(x[u], x[u + 1], x[u + 2], x[u + 3]);
    }
  } else {
    for (int i = tid; i < MC * dim; i += 256) {
      const int t = i / dim, d = i - t * dim;
      float qv = 0.f, kv = 0.f;
      if (t < len) {
        const T* row = proj + (row0 + t) * p.row_stride + (long long)head * dim + d;
        qv = to_float(row[p.q_off]) * p.q_scale;
        kv = to_float(row[p.k_off]);
      }
      q_t[d * MCP + t] = qv;
      k_t[d * MCP + t] = kv;
    }
    for (int i = tid; i < MC * 64; i += 256) {
      const int t = i >> 6, cc = i & 63;
      v_s[i] = (t < len && col0 + cc < vdim)
                   ? to_float(proj[(row0 + t) * p.row_stride + p.v_off + (long long)head * vdim + col0 + cc]) : 0.f;
    }
  }
  __syncthreads();
  // weighted scores of the chunk: tokens t = 4 ty .. and s = 4 tx ..
  {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    if (tx <= ty) {                      // (patches above the diagonal are zeros)
      for (int d = 0; d < dim; ++d) {
        const float4 qv = *reinterpret_cast<const float4*>(q_t + d * MCP + ty * 4);
        const float4 kv = *reinterpret_cast<const float4*>(k_t + d * MCP + tx * 4);
        const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ka[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(qa[i], ka[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int sx = tx * 4 + j;
      float4 o;
      float* oa = reinterpret_cast<float*>(&o);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = ty * 4 + i;
        oa[i] = (sx <= t && t < len) ? acc[i][j] * expf(g_c[t] + g_a[sx]) : 0.f;
      }
      *reinterpret_cast<float4*>(a_t + sx * MCP + ty * 4) = o;
    }
  }
  __syncthreads();
  // the parts of num_t and den_t that need no earlier chunk: tokens 4 ty .., channels 4 tx ..
  {
    float acc[4][4], den[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int s_end = min(len, ty * 4 + 4);
    for (int sx = 0; sx < s_end; ++sx) {
      const float4 av = *reinterpret_cast<const float4*>(a_t + sx * MCP + ty * 4);
      const float4 vv = *reinterpret_cast<const float4*>(v_s + sx * 64 + tx * 4);
      const float aa[4] = {av.x, av.y, av.z, av.w}, va[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        den[i] += aa[i];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(aa[i], va[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ty * 4 + i;
      if (t >= len) break;
      if (tx == 0 && col_block == 0) c.den[(row0 + t) * H + head] = den[i];
      float* o = p.out + (row0 + t) * p.out_row_stride + (long long)head * vdim + col0 + tx * 4;
      if (c.vec) {
        if (col0 + tx * 4 < vdim) *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col0 + tx * 4 + j < vdim) o[j] = acc[i][j];
    }
  }
  // the chunk's contribution to the state: key channels 4 ty .. (+ 64, ...)
  const long long cell = ((long long)seq * c.max_chunks + chunk) * H + head;
  float* dst = c.ds + cell * dim * vdim;
  for (int i0 = ty * 4; i0 < dim; i0 += 64) {
    float acc[4][4], nacc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int sx = 0; sx < len; sx += 4) {
      // (four tokens of a channel at once; tokens past the chunk's last one have the weight 0)
      const float4 wv = *reinterpret_cast<const float4*>(w_end + sx);
      float kw[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 kv = i0 + i < dim ? *reinterpret_cast<const float4*>(k_t + (i0 + i) * MCP + sx) : make_float4(0.f, 0.f, 0.f, 0.f);
        kw[i][0] = kv.x * wv.x; kw[i][1] = kv.y * wv.y; kw[i][2] = kv.z * wv.z; kw[i][3] = kv.w * wv.w;
        nacc[i] = fmaf(kv.w, wv.w, fmaf(kv.z, wv.z, fmaf(kv.y, wv.y, fmaf(kv.x, wv.x, nacc[i]))));      // (each product and sum rounded once)
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
      if (tx == 0 && col_block == 0) c.dn[cell * dim + i0 + i] = nacc[i];
      float* o = dst + (long long)(i0 + i) * vdim + col0 + tx * 4;
      if (c.vec) {
        if (col0 + tx * 4 < vdim) *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (col0 + tx * 4 + j < vdim) o[j] = acc[i][j];
    }
  }
}

// One thread per (sequence, head, element of S or of n): walks the sequence's chunks in order; leaves in the chunk's
// cell the state that chunk STARTS from, and in the state what the last chunk leaves.
__global__ void __launch_bounds__(256) mlstm_prefix_kernel(MlstmChunked c) {
  const MlstmArgs& p = c.a;
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y, H = p.n_heads, dim = p.dim, vdim = p.vdim;
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e >= dim * (vdim + 1)) return;
  const int n_new = p.seq_start[seq + 1] - p.seq_start[seq];
  const int n_chunks = (n_new + MC - 1) / MC;
  const long long slot_head = (long long)p.slots[seq] * H + head;
  const bool is_s = e < dim * vdim;
  float* st = is_s ? p.s + slot_head * dim * vdim + e : p.n + slot_head * dim + (e - dim * vdim);
  const long long base = ((long long)seq * c.max_chunks) * H + head;
  float* cell = is_s ? c.ds + base * dim * vdim + e : c.dn + base * dim + (e - dim * vdim);
  const long long stride = (long long)H * (is_s ? dim * vdim : dim);
  float s = *st;
  for (int k = 0; k < n_chunks; k += 4) {
    float kv[4], f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      kv[u] = k + u < n_chunks ? __ldcg(cell + (k + u) * stride) : 0.f;
      f[u] = k + u < n_chunks ? c.carry[base + (long long)(k + u) * H] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k + u < n_chunks) {
        cell[(k + u) * stride] = s;
        s = fmaf(f[u], s, kv[u]);
      }
    }
  }
  *st = s;
}

// The same, four neighbouring elements a thread and eight chunks asked for at a time, where rows of S and n are whole pieces of 16
// bytes on such boundaries (12 to 6 us beside other work at 2 x 1,024 tokens).
__global__ void __launch_bounds__(128) mlstm_prefix_vec_kernel(MlstmChunked c) {
  const MlstmArgs& p = c.a;
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y, H = p.n_heads, dim = p.dim, vdim = p.vdim;
  const int e = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (e >= dim * (vdim + 1)) return;
  const int n_new = p.seq_start[seq + 1] - p.seq_start[seq];
  const int n_chunks = (n_new + MC - 1) / MC;
  const long long slot_head = (long long)p.slots[seq] * H + head;
  const bool is_s = e < dim * vdim;
  float* st = is_s ? p.s + slot_head * dim * vdim + e : p.n + slot_head * dim + (e - dim * vdim);
  const long long base = ((long long)seq * c.max_chunks) * H + head;
  float* cell = is_s ? c.ds + base * dim * vdim + e : c.dn + base * dim + (e - dim * vdim);
  const long long stride = (long long)H * (is_s ? dim * vdim : dim);
  float4 s = *reinterpret_cast<float4*>(st);
  for (int k = 0; k < n_chunks; k += 8) {
    float4 kv[8];
    float f[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      kv[u] = k + u < n_chunks ? __ldcg(reinterpret_cast<const float4*>(cell + (k + u) * stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
      f[u] = k + u < n_chunks ? c.carry[base + (long long)(k + u) * H] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (k + u < n_chunks) {
        *reinterpret_cast<float4*>(cell + (k + u) * stride) = s;
        s = make_float4(fmaf(f[u], s.x, kv[u].x), fmaf(f[u], s.y, kv[u].y), fmaf(f[u], s.z, kv[u].z), fmaf(f[u], s.w, kv[u].w));
      }
    }
  }
  *reinterpret_cast<float4*>(st) = s;
}

// out[t] = (out[t] + f_t S_in^T q_t) / (max(|den_t + f_t n_in . q_t|, exp(-m_t)) + 1e-6), f_t = exp(c_t + m_in - m_t);
// grid and blocks as mlstm_chunk_kernel.
template <typename T>
__global__ void __launch_bounds__(256) mlstm_carry_kernel(const T* __restrict__ proj, MlstmChunked c) {
  const MlstmArgs& p = c.a;
  const int dim = p.dim, vdim = p.vdim, H = p.n_heads;
  extern __shared__ __align__(16) float sm[];
  float* q_t = sm;                 // [dim][MCP], q_t[d][t] already times f_t
  float* s_s = q_t + dim * MCP;    // [dim][64]
  float* n_s = s_s + dim * 64;     // [dim]
  float* f_s = n_s + dim;          // [MC]
  float* div_s = f_s + MC;         // [MC] the divisor of token t
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / c.col_blocks, col0 = (blockIdx.y - head * c.col_blocks) * 64;
  const int first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - first;
  if (chunk * MC >= n_new) return;
  const int len = min(MC, n_new - chunk * MC);
  const long long row0 = first + (long long)chunk * MC;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const long long cell = ((long long)seq * c.max_chunks + chunk) * H + head;
  if (tid < MC) {
    const long long g = (row0 + tid) * H + head;
    f_s[tid] = tid < len ? expf(c.gc[g] + c.m_start[cell] - c.gm[g]) : 0.f;
  }
  for (int d = tid; d < dim; d += 256) n_s[d] = c.dn[cell * dim + d];
  __syncthreads();
  const float* src = c.ds + cell * dim * vdim + col0;
  constexpr int V = 16 / (int)sizeof(T);
  if (c.vec) {
#pragma unroll 2
    for (int i = tid; i < dim / V * MC; i += 256) {
      const int t = i % MC, d = i / MC * V;
      float x[V];
      unpack16(t < len ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * p.row_stride + p.q_off + (long long)head * dim + d))
                       : make_uint4(0u, 0u, 0u, 0u), x);
#pragma unroll
      for (int u = 0; u < V; ++u) q_t[(d + u) * MCP + t] = x[u] * p.q_scale * f_s[t];
    }
#pragma unroll 4
    for (int i = tid; i < dim * 16; i += 256) {
      const int d = i >> 4, cc = (i & 15) * 4;
      *reinterpret_cast<float4*>(s_s + d * 64 + cc) =
          col0 + cc < vdim ? *reinterpret_cast<const float4*>(src + (long long)d * vdim + cc) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
    for (int i = tid; i < MC * dim; i += 256) {
      const int t = i / dim, d = i - t * dim;
      q_t[d * MCP + t] = t < len ? to_float(proj[(row0 + t) * p.row_stride + p.q_off + (long long)head * dim + d]) *
                                       p.q_scale * f_s[t] : 0.f;
    }
    for (int i = tid; i < dim * 64; i += 256) {
      const int d = i >> 6, cc = i & 63;
      s_s[i] = col0 + cc < vdim ? src[(long long)d * vdim + cc] : 0.f;
    }
  }
  __syncthreads();
  if (tid < len) {
    float nq = 0.f;
    for (int d = 0; d < dim; ++d) nq = fmaf(q_t[d * MCP + tid], n_s[d], nq);
    const long long g = (row0 + tid) * H + head;
    div_s[tid] = fmaxf(fabsf(c.den[g] + nq), expf(-c.gm[g])) + 1e-6f;
  }
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int d = 0; d < dim; ++d) {
    const float4 qv = *reinterpret_cast<const float4*>(q_t + d * MCP + ty * 4);
    const float4 sv = *reinterpret_cast<const float4*>(s_s + d * 64 + tx * 4);
    const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, sa[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(qa[i], sa[j], acc[i][j]);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty * 4 + i;
    if (t >= len) break;
    float* o = p.out + (row0 + t) * p.out_row_stride + (long long)head * vdim + col0 + tx * 4;
    const float by = div_s[t];
    if (c.vec) {
      if (col0 + tx * 4 < vdim) {
        const float4 x = *reinterpret_cast<const float4*>(o);
        *reinterpret_cast<float4*>(o) =
            make_float4((x.x + acc[i][0]) / by, (x.y + acc[i][1]) / by, (x.z + acc[i][2]) / by, (x.w + acc[i][3]) / by);
      }
      continue;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (col0 + tx * 4 + j < vdim) o[j] = (o[j] + acc[i][j]) / by;
  }
}

// The numbers of a chunk's contribution to S that are not finite, by multiply-adds (a call of its own: inside, it costs the kernel registers).
template <typename T>
__device__ __noinline__ void mlstm_plain_state(const T* k, const T* v, long long stride, const float* w_end, int len, int dim, int cols, float* dst,
                                               int vdim) {
  for (int i = threadIdx.x; i < dim * cols; i += CM_THREADS) {
    const int d = i / cols, c = i - d * cols;
    float* at = dst + (long long)d * vdim + c;
    if (isfinite(*at)) continue;
    float x = 0.f;
#pragma unroll 8
    for (int t = 0; t < len; ++t) x = fmaf(to_float(k[t * stride + d]) * w_end[t], to_float(v[t * stride + c]), x);
    *at = x;
  }
}

// The chunks on tensor cores (chunk_mma.cuh), for rows on 16-byte boundaries with channels in whole operand tiles: first every
// chunk's contribution to S and n, then mlstm_prefix_kernel, then all of o at once, which is written once.  bfloat16 q, k and v go
// in as they are; the weights, the state and n in three parts.  The whole chain (gates, the
// three kernels) at 2 x 1,024 tokens of 16 heads of 64 x 64 takes 80 us with the kernels above and 46 so, 32-bit rows 85 and 62,
// 6 x 1,000 of 12 heads 123 and 76, one run of 700 45 and 36, of 400 29 and 31.  n is summed by multiply-adds (see there).
template <typename T>
__global__ void __launch_bounds__(CM_THREADS, 4) mlstm_state_kernel(const T* __restrict__ proj, MlstmChunked c) {
  constexpr int PARTS = sizeof(T) == 2 ? 1 : 3;
  const MlstmArgs& p = c.a;
  const int dim = p.dim, vdim = p.vdim, H = p.n_heads;
  extern __shared__ __align__(16) unsigned char cm_smem[];
  __nv_bfloat16* k_s = reinterpret_cast<__nv_bfloat16*>(cm_smem);      // [3][64][dim + 8]: exp(c_L - c_s + a_s - m_L) k_s
  const int k_stride = dim + 8, k_part = CM_CHUNK * k_stride, v_part = CM_CHUNK * CM_ROW;
  __nv_bfloat16* v_s = k_s + 3 * k_part;                               // [PARTS][64][72]
  __shared__ float w_end[CM_CHUNK];
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / c.col_blocks, col_block = blockIdx.y - head * c.col_blocks, col0 = col_block * CM_COLS;
  const int first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - first;
  if (chunk * MC >= n_new) return;
  const int len = min(MC, n_new - chunk * MC);
  const long long row0 = first + (long long)chunk * MC;
  const T* rows = proj + row0 * p.row_stride;
  if (threadIdx.x < MC) {
    const long long g = (row0 + threadIdx.x) * H + head, gl = (row0 + len - 1) * H + head;
    w_end[threadIdx.x] = threadIdx.x < len ? expf(c.gc[gl] - c.gm[gl] + c.ga[g] - c.gc[g]) : 0.f;
  }
  __syncthreads();
  // Keys times their weights, in parts; and n in multiply-adds, each product and sum rounded once: a thread's tokens of eight channels here,
  // the threads of a channel in order further below.  (As a product of the parts with ones, n was cut twelve times a chunk: 1.3e-7 of it
  // on average, where the multiply-adds' errors of 8e-8 have no sign.)
  const int pieces = dim / 8, at_once = CM_THREADS / pieces, k_first = threadIdx.x / pieces, k_ch = (threadIdx.x - k_first * pieces) * 8;
  float n[8] = {};
  if (k_first < at_once) {
#pragma unroll 2
    for (int t = k_first; t < MC; t += at_once) {
      float x[8] = {};
      if (t < len) cm_load8(rows + t * p.row_stride + p.k_off + head * dim + k_ch, x);
      const float w = w_end[t];
      unsigned part[4][3];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        n[u] = fmaf(x[u], w, n[u]);
        x[u] *= w;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) cm_split<3>(x[2 * u], x[2 * u + 1], part[u]);
#pragma unroll
      for (int q = 0; q < 3; ++q)
        *reinterpret_cast<uint4*>(k_s + q * k_part + t * k_stride + k_ch) = make_uint4(part[0][q], part[1][q], part[2][q], part[3][q]);
    }
  }
  cm_fill<PARTS>(v_s, MC, CM_COLS, CM_ROW, v_part, [&](int t, int ch, float (&x)[8]) {
    const bool in = t < len && col0 + ch < vdim;
    if (in) cm_load8(rows + t * p.row_stride + p.v_off + head * vdim + col0 + ch, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = in ? x[u] : 0.f;
  });
  __syncthreads();
  const long long cell = ((long long)seq * c.max_chunks + chunk) * H + head;
  float* dst = c.ds + cell * dim * vdim + col0;
  const bool bad = cm_state<3, PARTS>(k_s, k_stride, k_part, v_s, v_part, dim, [&](int d, int ch, float x, float y) {
    if (col0 + ch < vdim) *reinterpret_cast<float2*>(dst + (long long)d * vdim + ch) = make_float2(x, y);
  });
  if (__syncthreads_or(bad))      // (and the keys have been read)
    mlstm_plain_state<T>(rows + p.k_off + head * dim, rows + p.v_off + head * vdim + col0, p.row_stride, w_end, len, dim, min(CM_COLS, vdim - col0), dst, vdim);
  if (col_block != 0) return;
  float* n_s = reinterpret_cast<float*>(cm_smem);      // [at_once][dim]
  if (k_first < at_once)
#pragma unroll
    for (int u = 0; u < 8; u += 4) *reinterpret_cast<float4*>(n_s + k_first * dim + k_ch + u) = make_float4(n[u], n[u + 1], n[u + 2], n[u + 3]);
  __syncthreads();
  for (int d = threadIdx.x; d < dim; d += CM_THREADS) {
    float sum = n_s[d];
    for (int i = 1; i < at_once; ++i) sum += n_s[i * dim + d];
    c.dn[cell * dim + d] = sum;
  }
}

// A chunk's tokens (bits of `redo`, from token `first` on; of `den` those whose divisor is in doubt) by multiply-adds, a warp together, whole rows
// (the divisor is every channel's): qk and v are the chunk's rows from the head's channels on, v's and out's the block's; n the incoming
// normaliser.  (A call of its own: inside, it costs the kernel registers.)
template <typename T>
__device__ __noinline__ void mlstm_plain_rows(unsigned redo, unsigned den, const T* qk, const T* v, long long stride, int q_off, int k_off,
                                              float q_scale, const float* state, int vdim, const float* n, const float* f_s,
                                              const float* floor_s, const float* g_c, const float* g_a, int first, int dim, int cols, float* out,
                                              long long out_stride) {
  const int lane = threadIdx.x & 31;
  auto in = [&](int d, int c) { return state[(long long)d * vdim + c]; };
  bool nan[2];
  cm_nan_columns(dim, cols, in, nan);
  for (; redo; redo &= redo - 1) {
    const int t = first + __ffs(redo) - 1;
    float* at = out + t * out_stride + lane;
    const bool doubt = (den & redo & (0u - redo)) != 0;
    if (!__any_sync(0xffffffffu, (!nan[0] && (doubt || !isfinite(at[0]))) || (!nan[1] && (doubt || !isfinite(at[32]))))) continue;
    auto query = [&](int d) { return to_float(qk[t * stride + q_off + d]) * q_scale; };
    float x[2], nq = 0.f;
#pragma unroll 1
    for (int d = lane; d < dim; d += 32) nq = fmaf(query(d), n[d], nq);
    nq = warp_sum(nq) * f_s[t];
    const float sum = cm_plain_row(t, dim, cols, f_s[t], query, [&](int s, int d) { return to_float(qk[s * stride + k_off + d]); },
                                   [&](int s, int c) { return to_float(v[s * stride + c]); }, in,
                                   [&](int s, float w) { return w * expf(g_c[t] + g_a[s]); }, x);
    const float by = fmaxf(fabsf(sum + nq), floor_s[t]) + 1e-6f;
    if (!nan[0]) at[0] = x[0] / by;
    if (!nan[1]) at[32] = x[1] / by;
  }
}

template <typename T>
__global__ void __launch_bounds__(CM_THREADS, 4) mlstm_out_kernel(const T* __restrict__ proj, MlstmChunked c) {
  constexpr int PARTS = sizeof(T) == 2 ? 1 : 3;
  const MlstmArgs& p = c.a;
  const int dim = p.dim, vdim = p.vdim, H = p.n_heads;
  extern __shared__ __align__(16) unsigned char cm_smem[];
  const int k_stride = dim + 8, k_part = CM_CHUNK * k_stride, s_part = max(dim, CM_CHUNK) * CM_ROW;
  __nv_bfloat16* k_s = reinterpret_cast<__nv_bfloat16*>(cm_smem);      // [PARTS][64][dim + 8]
  __nv_bfloat16* q_s = k_s + PARTS * k_part;                           // [PARTS][64][dim + 8]
  __nv_bfloat16* s_s = q_s + PARTS * k_part;                           // [3][dim][72] the state and, in column 64, n; then [PARTS][64][72] v
  __shared__ float g_a[MC], g_c[MC], f_s[MC], floor_s[MC];             // a_s - c_s, c_t - m_t, exp(c_t + m_in - m_t), exp(-m_t)
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / c.col_blocks, col0 = (blockIdx.y - head * c.col_blocks) * CM_COLS;
  const int first = p.seq_start[seq], n_new = p.seq_start[seq + 1] - first;
  if (chunk * MC >= n_new) return;
  const int len = min(MC, n_new - chunk * MC);
  const long long row0 = first + (long long)chunk * MC;
  const T* rows = proj + row0 * p.row_stride;
  const long long cell = ((long long)seq * c.max_chunks + chunk) * H + head;
  if (threadIdx.x < MC) {
    float ga = 0.f, gc = 0.f, gm = 0.f;
    if (threadIdx.x < len) {
      const long long g = (row0 + threadIdx.x) * H + head;
      ga = c.ga[g]; gc = c.gc[g]; gm = c.gm[g];
    }
    g_a[threadIdx.x] = ga - gc;
    g_c[threadIdx.x] = gc - gm;
    f_s[threadIdx.x] = threadIdx.x < len ? expf(gc + c.m_start[cell] - gm) : 0.f;
    floor_s[threadIdx.x] = expf(-gm);
  }
  const float* src = c.ds + cell * dim * vdim + col0;
  cm_fill<3>(s_s, dim, CM_ROW, CM_ROW, s_part, [&](int d, int ch, float (&x)[8]) {
    const bool state = ch < CM_COLS && col0 + ch < vdim;
    if (state) cm_load8(src + (long long)d * vdim + ch, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = state ? x[u] : 0.f;
    if (ch == CM_COLS) x[0] = c.dn[cell * dim + d];
  });
#pragma unroll
  for (int i = 0; i < 2; ++i)
    cm_fill<PARTS>(i ? q_s : k_s, MC, dim, k_stride, k_part, [&](int t, int ch, float (&x)[8]) {
      if (t < len) cm_load8(rows + t * p.row_stride + (i ? p.q_off : p.k_off) + head * dim + ch, x);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = t < len ? x[u] : 0.f;
    });
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  const int ta = warp * 16 + g, tb = ta + 8;      // this thread's rows
  auto query = [&](int d, unsigned (&a)[PARTS][4]) {      // the operand of 16 channels from d on
#pragma unroll
    for (int q = 0; q < PARTS; ++q) cm_ldmatrix(a[q], q_s + q * k_part + (warp * 16 + (lane & 15)) * k_stride + d + (lane >> 4) * 8);
  };
  float o[8][4], o_small[8][4], div_a, div_b;
  bool doubt_a, doubt_b;      // of the divisors
  float zeros[2];             // (zero times a row's numbers, where the divisor is not in doubt)
  {
    // f_t S_in^T q_t and f_t n_in . q_t
    float nq[4] = {}, nq_small[4] = {};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[j][i] = o_small[j][i] = 0.f;
    for (int d = 0; d < dim; d += 16) {
      unsigned a[PARTS][4];
      query(d, a);
      cm_step_rows<PARTS, 3, 8>(o, o_small, a, s_s, d, s_part);
#pragma unroll
      for (int pb = 2; pb >= 0; --pb) {
        unsigned b0, b1;
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(b0), "=r"(b1)
                     : "r"((unsigned)__cvta_generic_to_shared(s_s + pb * s_part + (d + (lane & 15)) * CM_ROW + CM_COLS)) : "memory");
#pragma unroll
        for (int pa = 0; pa < PARTS; ++pa) {
          if (pa + pb == 0) {
            float x[4];
            cm_mma_zero(x, a[0], b0, b1);
            cm_add(nq, x);
          } else if (pa + pb <= 2) {
            cm_mma(nq_small, a[pa], b0, b1);
          }
        }
      }
    }
    const float fa = f_s[ta] * p.q_scale, fb = f_s[tb] * p.q_scale;
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[j][i] = (o[j][i] + o_small[j][i]) * (i < 2 ? fa : fb);
      }
    div_a = __shfl_sync(0xffffffffu, nq[0] + nq_small[0], lane & ~3) * fa;
    div_b = __shfl_sync(0xffffffffu, nq[2] + nq_small[2], lane & ~3) * fb;
  }
  float sc[8][4];
  {
    // the weighted scores of this warp's tokens on those up to its last one, and their sums
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float small[2][4] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) sc[j][i] = sc[j + 1][i] = 0.f;
      if (j > 2 * warp) continue;
      for (int d = 0; d < dim; d += 16) {
        unsigned a[PARTS][4], b[PARTS][4];
        query(d, a);
        // (matrices: tokens 8 j.. of channels d.., of channels d + 8.., then tokens 8 j + 8..)
        const __nv_bfloat16* at = k_s + (8 * j + (lane & 7) + (lane >> 4) * 8) * k_stride + d + (lane >> 3 & 1) * 8;
#pragma unroll
        for (int q = 0; q < PARTS; ++q) cm_ldmatrix(b[q], at + q * k_part);
        cm_products<PARTS, PARTS>(sc[j], small[0], sc[j + 1], small[1], a, b);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sc[j][i] += small[0][i];
        sc[j + 1][i] += small[1][i];
      }
    }
    float den_a = 0.f, den_b = 0.f;
    const float ca = g_c[ta], cb = g_c[tb];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = i < 2 ? ta : tb, at = 8 * j + t2 + (i & 1);
        sc[j][i] = at <= t && t < len ? sc[j][i] * p.q_scale * expf((i < 2 ? ca : cb) + g_a[at]) : 0.f;
        if (i < 2) den_a += sc[j][i];
        else den_b += sc[j][i];
      }
#pragma unroll
    for (int x = 1; x < 4; x <<= 1) {
      den_a += __shfl_xor_sync(0xffffffffu, den_a, x);
      den_b += __shfl_xor_sync(0xffffffffu, den_b, x);
    }
    div_a += den_a;
    div_b += den_b;
    doubt_a = !isfinite(div_a);
    doubt_b = !isfinite(div_b);
    zeros[0] = doubt_a ? 1.f : 0.f;
    zeros[1] = doubt_b ? 1.f : 0.f;
    div_a = fmaxf(fabsf(div_a), floor_s[ta]) + 1e-6f;
    div_b = fmaxf(fabsf(div_b), floor_s[tb]) + 1e-6f;
  }
  __syncthreads();      // the state has been read
  cm_fill<PARTS>(s_s, MC, CM_COLS, CM_ROW, s_part, [&](int t, int ch, float (&x)[8]) {
    const bool in = t < len && col0 + ch < vdim;
    if (in) cm_load8(rows + t * p.row_stride + p.v_off + head * vdim + col0 + ch, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = in ? x[u] : 0.f;
  });
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) o_small[j][i] = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {      // 16 tokens s at a time
    if (j > warp) break;
    unsigned a[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      unsigned part[3];
      cm_split<3>(sc[2 * j + (i >> 1)][2 * (i & 1)], sc[2 * j + (i >> 1)][2 * (i & 1) + 1], part);
#pragma unroll
      for (int q = 0; q < 3; ++q) a[q][i] = part[q];
    }
    cm_step_rows<3, PARTS, 8>(o, o_small, a, s_s, 16 * j, s_part);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int ch = 8 * j + t2;
    if (col0 + ch >= vdim) break;
    float* at = p.out + row0 * p.out_row_stride + (long long)head * vdim + col0 + ch;
#pragma unroll
    for (int i = 0; i < 4; ++i) o[j][i] += o_small[j][i];
    zeros[0] = fmaf(o[j][0] + o[j][1], 0.f, zeros[0]);
    zeros[1] = fmaf(o[j][2] + o[j][3], 0.f, zeros[1]);
    if (ta < len) *reinterpret_cast<float2*>(at + ta * p.out_row_stride) = make_float2(o[j][0] / div_a, o[j][1] / div_a);
    if (tb < len) *reinterpret_cast<float2*>(at + tb * p.out_row_stride) = make_float2(o[j][2] / div_b, o[j][3] / div_b);
  }
  const unsigned redo = cm_bad_rows(ta < len && zeros[0] != 0.f, tb < len && zeros[1] != 0.f);
  if (redo == 0) return;
  __syncwarp();
  mlstm_plain_rows<T>(redo, cm_bad_rows(doubt_a, doubt_b), rows + head * dim, rows + p.v_off + head * vdim + col0, p.row_stride, p.q_off, p.k_off,
                      p.q_scale, src, vdim, c.dn + cell * dim, f_s, floor_s, g_c, g_a, warp * 16, dim, min(CM_COLS, vdim - col0),
                      p.out + row0 * p.out_row_stride + (long long)head * vdim + col0, p.out_row_stride);
}

// (den is asked for and not used by the kernels in parts; which kernels take a call is known with its addresses only.)
static long long mlstm_scratch_floats(long long n_rows, int n_seqs, int max_new, int n_heads, int dim, int vdim) {
  const long long chunks = (max_new + MC - 1) / MC;
  const long long cells = (long long)n_seqs * chunks * n_heads;
  return 4 * (n_rows * n_heads + 4) + 2 * (cells + 4) + cells * dim * (vdim + 1) + 64;
}

template <typename T>
static int launch_mlstm_chunked(const T* proj, MlstmArgs p, float* scratch, long long n_rows, int max_new, int n_seqs,
                                cudaStream_t stream) {
  MlstmChunked c;
  c.a = p;
  c.max_chunks = (max_new + MC - 1) / MC;
  c.col_blocks = (p.vdim + 63) / 64;
  const long long per_row = (n_rows * p.n_heads + 3) / 4 * 4;
  const long long cells = (long long)n_seqs * c.max_chunks * p.n_heads, cells4 = (cells + 3) / 4 * 4;
  c.ga = scratch;
  c.gc = c.ga + per_row;
  c.gm = c.gc + per_row;
  c.den = c.gm + per_row;
  c.m_start = c.den + per_row;
  c.carry = c.m_start + cells4;
  c.ds = c.carry + cells4;
  c.dn = c.ds + cells * p.dim * p.vdim;
  BT_CHECK((long long)p.n_heads * c.col_blocks <= 65535, "mlstm_scan: %d heads x %d column blocks are too many", p.n_heads,
           c.col_blocks);
  constexpr int V = 16 / (int)sizeof(T);
  c.vec = p.dim % V == 0 && p.vdim % V == 0 && p.q_off % V == 0 && p.k_off % V == 0 && p.v_off % V == 0 && p.row_stride % V == 0 &&
          p.out_row_stride % 4 == 0 && ((unsigned long long)proj | (unsigned long long)p.out | (unsigned long long)c.ds) % 16 == 0;
  // By the layer's sizes and addresses alone: a sequence's bits must not depend on what else is in the call.  Multiply-adds / parts, us:
  // bfloat16 heads of 64 x 64 36 blocks 24.5 / 26.6, 84 29.1 / 31.2, 132 45 / 36, 512 80 / 46; 128 x 128 16 blocks 33 / 29, 1,024 193 / 137.
  // 32-bit rows 64 x 64 36 blocks 25.7 / 24.7, 1,152 143 / 123; 128 x 64 256 blocks 74 / 67, 1,152 252 / 278.
  if (c.vec && p.dim % 16 == 0 && p.dim <= 128 && p.vdim % 8 == 0 && p.q_off % 8 == 0 && p.k_off % 8 == 0 && p.v_off % 8 == 0) {
    constexpr int PARTS = sizeof(T) == 2 ? 1 : 3;
    const dim3 cells(c.max_chunks, p.n_heads * c.col_blocks, n_seqs);
    const size_t rows_k = (size_t)MC * (p.dim + 8), rows_s = (size_t)(p.dim > MC ? p.dim : MC) * CM_ROW;
    const size_t smem_s = 2 * (3 * rows_k + PARTS * (size_t)MC * CM_ROW), smem_o = 2 * (2 * PARTS * rows_k + 3 * rows_s);
    static SharedMemoryAllowance allowed_s, allowed_o;
    BT_CHECK(allow_shared_memory(allowed_s, mlstm_state_kernel<T>, smem_s) && allow_shared_memory(allowed_o, mlstm_out_kernel<T>, smem_o),
             "mlstm_scan: cannot reserve %zu bytes of shared memory", smem_s > smem_o ? smem_s : smem_o);
    BT_PDL_OK("mlstm_gates", launch_pdl(mlstm_gates_kernel<T>, dim3(p.n_heads, n_seqs), dim3(256), 0, stream, 1, proj, c));
    BT_PDL_OK("mlstm_state", launch_pdl(mlstm_state_kernel<T>, cells, dim3(CM_THREADS), smem_s, stream, 1, proj, c));
    if (((unsigned long long)p.s | (unsigned long long)p.n | (unsigned long long)c.dn) % 16 == 0)
      BT_PDL_OK("mlstm_prefix", launch_pdl(mlstm_prefix_vec_kernel, dim3((p.dim * (p.vdim + 1) + 511) / 512, p.n_heads, n_seqs), dim3(128),
                                           0, stream, 1, c));
    else
      BT_PDL_OK("mlstm_prefix", launch_pdl(mlstm_prefix_kernel, dim3((p.dim * (p.vdim + 1) + 255) / 256, p.n_heads, n_seqs), dim3(256),
                                           0, stream, 1, c));
    BT_PDL_OK("mlstm_out", launch_pdl(mlstm_out_kernel<T>, cells, dim3(CM_THREADS), smem_o, stream, 1, proj, c));
    return 0;
  }
  const dim3 grid(c.max_chunks, p.n_heads * c.col_blocks, n_seqs), block(256);
  const size_t smem_a = ((size_t)2 * p.dim * MCP + (size_t)MC * 64 + (size_t)MC * MCP + 3 * MC) * sizeof(float);
  const size_t smem_c = ((size_t)p.dim * MCP + (size_t)p.dim * 64 + p.dim + 2 * MC) * sizeof(float);
  auto chunk_kernel = mlstm_chunk_kernel<T>;
  auto carry_kernel = mlstm_carry_kernel<T>;
  if (smem_a > 48 * 1024)
    BT_CHECK(cudaFuncSetAttribute(chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_a) == cudaSuccess,
             "mlstm_scan: cannot reserve %zu bytes of shared memory", smem_a);
  if (smem_c > 48 * 1024)
    BT_CHECK(cudaFuncSetAttribute(carry_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_c) == cudaSuccess,
             "mlstm_scan: cannot reserve %zu bytes of shared memory", smem_c);
  BT_PDL_OK("mlstm_gates", launch_pdl(mlstm_gates_kernel<T>, dim3(p.n_heads, n_seqs), block, 0, stream, 1, proj, c));
  BT_PDL_OK("mlstm_chunk", launch_pdl(chunk_kernel, grid, block, smem_a, stream, 1, proj, c));
  BT_PDL_OK("mlstm_prefix", launch_pdl(mlstm_prefix_kernel, dim3((p.dim * (p.vdim + 1) + 255) / 256, p.n_heads, n_seqs),
                                       block, 0, stream, 1, c));
  BT_PDL_OK("mlstm_carry", launch_pdl(carry_kernel, grid, block, smem_c, stream, 1, proj, c));
  return 0;
}

}  // namespace bt

// Whether bt_mlstm_scan can hold a whole head in one block, and so apply the per-head norm and the gate itself.
extern "C" int bt_mlstm_scan_fuses(int dim, int vdim) { return vdim <= 32 || (vdim <= 64 && dim <= 128); }

// norm_w .. mixed_row_stride: null / 0, or (where bt_mlstm_scan_fuses) the per-head RMS norm's weight [heads * vdim], its
// eps, the channel of the output gate in the rows of proj, and where the normed and gated rows go (proj's type); `out`
// is then not written.
extern "C" int bt_mlstm_scan(const void* proj, long long row_stride, int q_off, int k_off, int v_off, int i_off, int f_off,
                             const float* i_bias, const float* f_bias, float cap, float q_scale, float* s, float* n,
                             float* m, const int* slots, const int* seq_start, float* out, long long out_row_stride,
                             const float* norm_w, float eps, int g_off, void* mixed, long long mixed_row_stride,
                             int n_seqs, int n_heads, int dim, int vdim, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && dim > 0 && dim <= 256 && vdim > 0 && n_seqs >= 0 && n_seqs <= 65535 && n_heads <= 65535,
           "mlstm_scan: bad sizes seqs=%d heads=%d dim=%d vdim=%d (up to 256 key channels a head)", n_seqs, n_heads, dim,
           vdim);
  BT_CHECK(cap > 0.f, "mlstm_scan: the gates' cap must be positive");
  if (n_seqs == 0) return 0;
  MlstmArgs p;
  p.row_stride = row_stride;
  p.q_off = q_off; p.k_off = k_off; p.v_off = v_off; p.i_off = i_off; p.f_off = f_off;
  p.i_bias = i_bias; p.f_bias = f_bias; p.cap = cap; p.q_scale = q_scale;
  p.s = s; p.n = n; p.m = m; p.slots = slots; p.seq_start = seq_start; p.out = out; p.out_row_stride = out_row_stride;
  p.n_heads = n_heads; p.dim = dim; p.vdim = vdim; p.cols = 0;
  BT_CHECK(mixed == nullptr || (norm_w != nullptr && bt_mlstm_scan_fuses(dim, vdim)),
           "mlstm_scan: the norm of heads of %d x %d cannot be fused", dim, vdim);
  p.norm_w = norm_w; p.eps = eps; p.g_off = g_off; p.mixed = mixed; p.mixed_row_stride = mixed_row_stride;
  if (dtype == kF32) return launch_mlstm<float>((const float*)proj, p, n_seqs, stream);
  if (dtype == kBF16) return launch_mlstm<__nv_bfloat16>((const __nv_bfloat16*)proj, p, n_seqs, stream);
  return fail("mlstm_scan: unknown dtype %d", dtype);
}

// Floats of scratch the chunked form needs for a step of `n_rows` tokens whose longest run has `max_new`.
extern "C" long long bt_mlstm_chunked_scratch_floats(long long n_rows, int n_seqs, int max_new, int n_heads, int dim,
                                                     int vdim) {
  return bt::mlstm_scratch_floats(n_rows, n_seqs, max_new, n_heads, dim, vdim);
}

// The recurrence for steps that bring long runs of tokens: the same results as bt_mlstm_scan (beyond rounding), the
// chunks of a run worked side by side.  `max_new`: no sequence of the step brings more tokens than this; `n_rows`: the
// step's tokens.
extern "C" int bt_mlstm_chunked(const void* proj, long long row_stride, int q_off, int k_off, int v_off, int i_off,
                                int f_off, const float* i_bias, const float* f_bias, float cap, float q_scale, float* s,
                                float* n, float* m, const int* slots, const int* seq_start, float* out,
                                long long out_row_stride, float* scratch, long long n_rows, int max_new, int n_seqs,
                                int n_heads, int dim, int vdim, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && dim > 0 && dim <= 256 && vdim > 0 && n_seqs >= 0 && n_seqs <= 65535 && n_heads <= 65535 &&
               max_new > 0 && n_rows >= 0 && scratch,
           "mlstm_chunked: bad sizes seqs=%d heads=%d dim=%d vdim=%d max_new=%d", n_seqs, n_heads, dim, vdim, max_new);
  BT_CHECK(cap > 0.f, "mlstm_chunked: the gates' cap must be positive");
  if (n_seqs == 0) return 0;
  MlstmArgs p;
  p.row_stride = row_stride;
  p.q_off = q_off; p.k_off = k_off; p.v_off = v_off; p.i_off = i_off; p.f_off = f_off;
  p.i_bias = i_bias; p.f_bias = f_bias; p.cap = cap; p.q_scale = q_scale;
  p.s = s; p.n = n; p.m = m; p.slots = slots; p.seq_start = seq_start; p.out = out; p.out_row_stride = out_row_stride;
  p.n_heads = n_heads; p.dim = dim; p.vdim = vdim; p.cols = 64;
  p.norm_w = nullptr; p.eps = 0.f; p.g_off = 0; p.mixed = nullptr; p.mixed_row_stride = 0;
  if (dtype == kF32) return launch_mlstm_chunked<float>((const float*)proj, p, scratch, n_rows, max_new, n_seqs, stream);
  if (dtype == kBF16)
    return launch_mlstm_chunked<__nv_bfloat16>((const __nv_bfloat16*)proj, p, scratch, n_rows, max_new, n_seqs, stream);
  return fail("mlstm_chunked: unknown dtype %d", dtype);
}
