// Linear attention with a per-head decay, as a recurrence over a 32-bit state per (sequence, head):
//
//     S_t = decay_h * S_(t-1) + k_t v_t^T        (S: dim x vdim)
//     o_t = S_t^T q_t
//
// q, k, v are act(projection), applied here in 32-bit to the step's projections: act = x * sigmoid(x) (`act` 0) or the
// projection as it is (`act` 1: a caller that has prepared q, k, v itself, for instance rotated them).  Columns of
// S (value channels) never mix, so a block owns a group of value channels of one (sequence, head), keeps its part of
// the state in registers for all tokens of the step, and writes it back once.  Inside a block a value channel belongs
// to SPLIT adjacent lanes, each with DPT of the head's `dim` key channels; their partial outputs meet by shuffles.
// The state lives in `state[slot][head][dim][vdim]`; a sequence that starts finds zeros there.
#include "chunk_mma.cuh"
#include "common.cuh"

namespace bt {

constexpr int LS_TOKENS = 16;  // tokens staged in shared memory at a time

__device__ __forceinline__ float silu(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float feature(float x, int act) { return act == 0 ? silu(x) : x; }

template <typename T, int DPT, int SPLIT>
__global__ void __launch_bounds__(256)
lightning_scan_kernel(const T* __restrict__ proj, long long row_stride, int q_off, int k_off, int v_off,
                      float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ seq_start,
                      const float* __restrict__ decay, float* __restrict__ out, long long out_row_stride, int n_heads,
                      int dim, int vdim, int cols, int act) {
  extern __shared__ float sm[];
  float* q_s = sm;                          // [LS_TOKENS][dim]
  float* k_s = q_s + LS_TOKENS * dim;       // [LS_TOKENS][dim]
  float* v_s = k_s + LS_TOKENS * dim;       // [LS_TOKENS][cols]
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
  const float lam = decay[head];
  for (int t0 = 0; t0 < n_new; t0 += LS_TOKENS) {
    const int nt = min(LS_TOKENS, n_new - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < nt * dim; i += blockDim.x) {
      const int t = i / dim, d = i - t * dim;
      const T* row = proj + (long long)(first + t0 + t) * row_stride + (long long)head * dim + d;
      q_s[i] = feature(to_float(row[q_off]), act);
      k_s[i] = feature(to_float(row[k_off]), act);
    }
    for (int i = threadIdx.x; i < nt * cols; i += blockDim.x) {
      const int t = i / cols, c = i - t * cols;
      v_s[i] = col0 + c < vdim
                   ? feature(to_float(proj[(long long)(first + t0 + t) * row_stride + v_off + (long long)head * vdim + col0 + c]), act)
                   : 0.f;
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      const float v = col_local < cols ? v_s[t * cols + col_local] : 0.f;
      const float* kt = k_s + t * dim + d0;
      const float* qt = q_s + t * dim + d0;
      float o = 0.f;
#pragma unroll
      for (int i = 0; i < DPT; ++i) {
        if (d0 + i < dim) {
          s[i] = fmaf(lam, s[i], kt[i] * v);
          o = fmaf(s[i], qt[i], o);
        }
      }
#pragma unroll
      for (int x = 1; x < SPLIT; x <<= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
      if (owns && part == 0) out[(long long)(first + t0 + t) * out_row_stride + (long long)head * vdim + col] = o;
    }
  }
  if (owns) {
#pragma unroll
    for (int i = 0; i < DPT; ++i)
      if (d0 + i < dim) s_base[(long long)(d0 + i) * vdim + col] = s[i];
  }
}

template <typename T>
static int launch_lightning(const T* proj, long long row_stride, int q_off, int k_off, int v_off, float* state,
                            const int* slots, const int* seq_start, const float* decay, float* out,
                            long long out_row_stride, int n_seqs, int n_heads, int dim, int vdim, int act, cudaStream_t stream) {
  // DPT key channels per lane, SPLIT lanes per value channel: SPLIT * DPT >= dim
  int dpt, split;
  if (dim <= 32) { dpt = 8; split = 4; }
  else if (dim <= 64) { dpt = 8; split = 8; }
  else if (dim <= 128) { dpt = 16; split = 8; }
  else { dpt = 32; split = 8; }
  BT_CHECK(dim <= 256, "lightning_scan: %d key channels per head; the kernel takes up to 256", dim);
  const int cols = 256 / split < vdim ? 256 / split : vdim;   // value channels per block
  const dim3 grid((vdim + cols - 1) / cols, n_heads, n_seqs), block(256);
  const size_t smem = (size_t)LS_TOKENS * (2 * dim + cols) * sizeof(float);
#define BT_LS(DPT, SPLIT)                                                                                          \
  BT_PDL_OK("lightning_scan", launch_pdl(lightning_scan_kernel<T, DPT, SPLIT>, grid, block, smem, stream, 1, proj, \
                                         row_stride, q_off, k_off, v_off, state, slots, seq_start, decay, out,     \
                                         out_row_stride, n_heads, dim, vdim, cols, act))
  if (dpt == 8 && split == 4) BT_LS(8, 4);
  else if (dpt == 8) BT_LS(8, 8);
  else if (dpt == 16) BT_LS(16, 8);
  else BT_LS(32, 8);
#undef BT_LS
  return 0;
}

}  // namespace bt

extern "C" int bt_lightning_scan(const void* proj, long long row_stride, int q_off, int k_off, int v_off, float* state,
                                 const int* slots, const int* seq_start, const float* decay, float* out,
                                 long long out_row_stride, int n_seqs, int n_heads, int dim, int vdim, int act, int dtype,
                                 cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && dim > 0 && vdim > 0 && n_seqs >= 0 && n_seqs <= 65535 && n_heads <= 65535,
           "lightning_scan: bad sizes seqs=%d heads=%d dim=%d vdim=%d", n_seqs, n_heads, dim, vdim);
  if (n_seqs == 0) return 0;
  if (dtype == kF32)
    return launch_lightning<float>((const float*)proj, row_stride, q_off, k_off, v_off, state, slots, seq_start, decay,
                                   out, out_row_stride, n_seqs, n_heads, dim, vdim, act, stream);
  if (dtype == kBF16)
    return launch_lightning<__nv_bfloat16>((const __nv_bfloat16*)proj, row_stride, q_off, k_off, v_off, state, slots,
                                           seq_start, decay, out, out_row_stride, n_seqs, n_heads, dim, vdim, act, stream);
  return fail("lightning_scan: unknown dtype %d", dtype);
}

// ---- long runs of new tokens: the same recurrence by chunks ------------------------------------------------------
//
// Unrolled over a chunk of C tokens that starts from the state S_in, the recurrence reads
//
//     o_t   = decay^(t+1) S_in^T q_t + sum_{s <= t} decay^(t-s) (q_t . k_s) v_s          (t, s count inside the chunk)
//     S_out = decay^C S_in + sum_s decay^(C-1-s) k_s v_s^T
//
// so the chunks of a long prompt work side by side: lightning_chunk_kernel forms, per chunk, the sums over s (the part
// of o_t that needs no earlier chunk, and the chunk's own contribution to the state); lightning_prefix_kernel walks the
// chunks of a sequence in order, turning each contribution into the state its chunk starts from; lightning_carry_kernel
// adds decay^(t+1) S_in^T q_t.  Everything is 32-bit multiply-adds; powers of the decay come from powf.
namespace bt {

constexpr int LC = 64;    // tokens per chunk
constexpr int LCP = 68;   // row length of the transposed tiles: 16-byte rows, four-way conflicts at most when they are written

// What bounds the chunks' kernels is the way into and out of shared memory, not the multiply-adds: so rows are read 16 bytes a
// lane where they lie on such boundaries (`vec`; a warp's lanes are 32 tokens, whose numbers meet all banks when they are
// written channel by channel), the state's product reads four tokens of a channel at once, and results leave as 16 bytes.
// 2 x 1,024 tokens of 16 heads of 64 x 64 (chunk / carry kernel in a recorded layer, us): 60 / 25 with a number a lane, 39 / 18 so.
//
// Tiles of shared memory hold their 64 tokens along the fast axis ([channel][token], rows of LCP floats), so that a
// thread reads four tokens, or four value channels, with one 16-byte load and every product phase is 16 multiply-adds
// per two such loads.  Threads form a 16 x 16 grid; thread (ty, tx) owns a 4 x 4 patch of every product.

// grid (chunks, heads * column blocks, sequences); 256 threads; a block owns 64 value channels.
template <typename T>
__global__ void __launch_bounds__(256)
lightning_chunk_kernel(const T* __restrict__ proj, long long row_stride, int q_off, int k_off, int v_off,
                       const int* __restrict__ seq_start, const float* __restrict__ decay, float* __restrict__ out,
                       long long out_row_stride, float* __restrict__ scratch, int max_chunks, int n_heads, int dim, int vdim,
                       int col_blocks, int act, int vec) {
  extern __shared__ __align__(16) float sm[];
  float* q_t = sm;                       // [dim][LCP]   q_t[d][t]
  float* k_t = q_t + dim * LCP;          // [dim][LCP]   k_t[d][s]
  float* v_s = k_t + dim * LCP;          // [LC][64]     v_s[s][j]
  float* a_t = v_s + LC * 64;            // [LC][LCP]    a_t[s][t] = decay^(t-s) (q_t . k_s), zero for s > t
  float* pw = a_t + LC * LCP;            // [LC + 4] powers of the decay
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col0 = (blockIdx.y - head * col_blocks) * 64;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * LC >= n_new) return;
  const int len = min(LC, n_new - chunk * LC);
  const long long row0 = first + (long long)chunk * LC;
  const float lam = decay[head];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  for (int i = tid; i <= LC; i += 256) pw[i] = powf(lam, (float)i);
  constexpr int V = 16 / (int)sizeof(T);
  if (vec) {
    const int groups = dim / V;
#pragma unroll 4
    for (int i = tid; i < 2 * groups * LC; i += 256) {
      const int t = i % LC, g = i / LC;                    // (q's groups of channels, then k's)
      const bool key = g >= groups;
      const int d = (key ? g - groups : g) * V;
      float x[V];
      unpack16(t < len ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * row_stride + (key ? k_off : q_off) + (long long)head * dim + d))
                       : make_uint4(0u, 0u, 0u, 0u), x);
      float* dst = (key ? k_t : q_t) + d * LCP + t;
#pragma unroll
      for (int u = 0; u < V; ++u) dst[u * LCP] = t < len ? feature(x[u], act) : 0.f;
    }
#pragma unroll 2
    for (int i = tid; i < LC * 64 / V; i += 256) {
      const int t = i / (64 / V), c = i % (64 / V) * V;
      const bool in = t < len && col0 + c < vdim;
      float x[V];
      unpack16(in ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * row_stride + v_off + (long long)head * vdim + col0 + c))
                  : make_uint4(0u, 0u, 0u, 0u), x);
#pragma unroll
      for (int u = 0; u < V; ++u) v_s[t * 64 + c + u] = in ? feature(x[u], act) : 0.f;
    }
  } else {
    for (int i = tid; i < LC * dim; i += 256) {
      const int t = i / dim, d = i - t * dim;
      float qv = 0.f, kv = 0.f;
      if (t < len) {
        const T* row = proj + (row0 + t) * row_stride + (long long)head * dim + d;
        qv = feature(to_float(row[q_off]), act);
        kv = feature(to_float(row[k_off]), act);
      }
      q_t[d * LCP + t] = qv;
      k_t[d * LCP + t] = kv;
    }
    for (int i = tid; i < LC * 64; i += 256) {
      const int t = i >> 6, c = i & 63;
      v_s[i] = (t < len && col0 + c < vdim)
                   ? feature(to_float(proj[(row0 + t) * row_stride + v_off + (long long)head * vdim + col0 + c]), act) : 0.f;
    }
  }
  __syncthreads();
  // scores of the chunk: tokens t = 4 ty .. and s = 4 tx ..
  {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    if (tx <= ty) {                      // (patches above the diagonal are zeros)
      for (int d = 0; d < dim; ++d) {
        const float4 qv = *reinterpret_cast<const float4*>(q_t + d * LCP + ty * 4);
        const float4 kv = *reinterpret_cast<const float4*>(k_t + d * LCP + tx * 4);
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
        oa[i] = (sx <= t && t < len) ? acc[i][j] * pw[t - sx] : 0.f;
      }
      *reinterpret_cast<float4*>(a_t + sx * LCP + ty * 4) = o;
    }
  }
  __syncthreads();
  // the part of o_t that needs no earlier chunk: tokens 4 ty .., channels 4 tx ..
  {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int s_end = min(len, ty * 4 + 4);
    for (int sx = 0; sx < s_end; ++sx) {
      const float4 av = *reinterpret_cast<const float4*>(a_t + sx * LCP + ty * 4);
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
  // the chunk's contribution to the state: sum_s decay^(len-1-s) k_s[i] v_s[c], key channels 4 ty .. (+ 64, ...)
  float* dst = scratch + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim;
  for (int i0 = ty * 4; i0 < dim; i0 += 64) {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int sx = 0; sx < len; sx += 4) {
      // (tokens past the chunk's last one are zeros in both tiles)
      float w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) w[u] = pw[max(len - 1 - sx - u, 0)];
      float kw[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 kv = i0 + i < dim ? *reinterpret_cast<const float4*>(k_t + (i0 + i) * LCP + sx) : make_float4(0.f, 0.f, 0.f, 0.f);
        kw[i][0] = kv.x * w[0]; kw[i][1] = kv.y * w[1]; kw[i][2] = kv.z * w[2]; kw[i][3] = kv.w * w[3];
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

// One thread per (sequence, head, state element): walks the sequence's chunks in order; leaves in scratch[chunk] the
// state that chunk STARTS from and in `state` the state after the last one.  Four chunks' contributions are asked for
// at a time, so that the loads do not wait for one another.
__global__ void __launch_bounds__(256)
lightning_prefix_kernel(float* scratch, float* __restrict__ state, const int* __restrict__ slots,
                        const int* __restrict__ seq_start, const float* __restrict__ decay, int max_chunks, int n_heads,
                        int dim, int vdim) {
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y;
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (e >= dim * vdim) return;
  const int n_new = seq_start[seq + 1] - seq_start[seq];
  const int n_chunks = (n_new + LC - 1) / LC;
  const float lam = decay[head];
  const float full = powf(lam, (float)LC);
  const float tail = powf(lam, (float)(n_new - (n_chunks - 1) * LC));
  float* st = state + (((long long)slots[seq] * n_heads + head) * dim) * vdim + e;
  const long long stride = (long long)n_heads * dim * vdim;
  float* cell = scratch + (((long long)seq * max_chunks) * n_heads + head) * (long long)dim * vdim + e;
  float s = *st;
  for (int c = 0; c < n_chunks; c += 4) {
    float kv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) kv[u] = c + u < n_chunks ? __ldcg(cell + (c + u) * stride) : 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c + u < n_chunks) {
        cell[(c + u) * stride] = s;
        s = fmaf(c + u == n_chunks - 1 ? tail : full, s, kv[u]);
      }
    }
  }
  *st = s;
}

// The same, four neighbouring elements a thread and eight chunks asked for at a time, where a state is whole pieces of 16 bytes on
// such boundaries: two rounds of loads for 1,024 tokens instead of four.
__global__ void __launch_bounds__(128)
lightning_prefix_vec_kernel(float* scratch, float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ seq_start,
                            const float* __restrict__ decay, int max_chunks, int n_heads, int dim, int vdim) {
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.z, head = blockIdx.y;
  const int e = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (e >= dim * vdim) return;
  const int n_new = seq_start[seq + 1] - seq_start[seq];
  const int n_chunks = (n_new + LC - 1) / LC;
  const float lam = decay[head];
  const float full = powf(lam, (float)LC);
  const float tail = powf(lam, (float)(n_new - (n_chunks - 1) * LC));
  float* st = state + (((long long)slots[seq] * n_heads + head) * dim) * vdim + e;
  const long long stride = (long long)n_heads * dim * vdim;
  float* cell = scratch + (((long long)seq * max_chunks) * n_heads + head) * (long long)dim * vdim + e;
  float4 s = *reinterpret_cast<float4*>(st);
  for (int c = 0; c < n_chunks; c += 8) {
    float4 kv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      kv[u] = c + u < n_chunks ? __ldcg(reinterpret_cast<const float4*>(cell + (c + u) * stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (c + u < n_chunks) {
        *reinterpret_cast<float4*>(cell + (c + u) * stride) = s;
        const float f = c + u == n_chunks - 1 ? tail : full;
        s = make_float4(fmaf(f, s.x, kv[u].x), fmaf(f, s.y, kv[u].y), fmaf(f, s.z, kv[u].z), fmaf(f, s.w, kv[u].w));
      }
    }
  }
  *reinterpret_cast<float4*>(st) = s;
}

// out[t] += decay^(t+1) S_in^T q_t for the tokens of a chunk; grid and blocks as lightning_chunk_kernel.
template <typename T>
__global__ void __launch_bounds__(256)
lightning_carry_kernel(const T* __restrict__ proj, long long row_stride, int q_off, const int* __restrict__ seq_start,
                       const float* __restrict__ decay, float* __restrict__ out, long long out_row_stride,
                       const float* __restrict__ scratch, int max_chunks, int n_heads, int dim, int vdim, int col_blocks,
                       int act, int vec) {
  extern __shared__ __align__(16) float sm[];
  float* q_t = sm;                 // [dim][LCP], q_t[d][t] already scaled by decay^(t+1)
  float* s_s = q_t + dim * LCP;    // [dim][64]
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col0 = (blockIdx.y - head * col_blocks) * 64;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * LC >= n_new) return;
  const int len = min(LC, n_new - chunk * LC);
  const long long row0 = first + (long long)chunk * LC;
  const float lam = decay[head];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  float* pw = s_s + dim * 64;      // [LC + 1] powers of the decay
  for (int i = tid; i <= LC; i += 256) pw[i] = powf(lam, (float)i);
  __syncthreads();
  constexpr int V = 16 / (int)sizeof(T);
  const float* src = scratch + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim + col0;
  if (vec) {
#pragma unroll 2
    for (int i = tid; i < dim / V * LC; i += 256) {
      const int t = i % LC, d = i / LC * V;
      float x[V];
      unpack16(t < len ? __ldg(reinterpret_cast<const uint4*>(proj + (row0 + t) * row_stride + q_off + (long long)head * dim + d))
                       : make_uint4(0u, 0u, 0u, 0u), x);
#pragma unroll
      for (int u = 0; u < V; ++u) q_t[(d + u) * LCP + t] = t < len ? feature(x[u], act) * pw[t + 1] : 0.f;
    }
#pragma unroll 4
    for (int i = tid; i < dim * 16; i += 256) {
      const int d = i >> 4, c = (i & 15) * 4;
      *reinterpret_cast<float4*>(s_s + d * 64 + c) =
          col0 + c < vdim ? *reinterpret_cast<const float4*>(src + (long long)d * vdim + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {
    for (int i = tid; i < LC * dim; i += 256) {
      const int t = i / dim, d = i - t * dim;
      q_t[d * LCP + t] = t < len ? feature(to_float(proj[(row0 + t) * row_stride + q_off + (long long)head * dim + d]), act) * pw[t + 1] : 0.f;
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
    const float4 qv = *reinterpret_cast<const float4*>(q_t + d * LCP + ty * 4);
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

// The chunks on tensor cores (chunk_mma.cuh), for rows on 16-byte boundaries with channels in whole operand tiles: first every
// chunk's contribution to the state (lightning_state_kernel), then lightning_prefix_kernel, then all of o at once
// (lightning_out_kernel), which is written once.  PARTS: 1 where q, k and v are bfloat16 numbers as they are, else 3.
// The kernels above are bound by shared memory (an operand read for every other multiply-add) and write o, read it and write it
// again; these by the forming of the features and the parts, and by the products.  All three kernels, above and here, in us: 2 x 1,024
// tokens of 16 heads of 64 x 64 with act 0 68 and 47, 6 x 1,000 of 12 heads 115 and 92, with act 1 60 and 30, 105 and 60; 32-bit rows 2 x 1,024
// 71 and 46, with act 1 66 and 37.  Errors against 64 bits 1.2e-7 and 7e-8 (act 0), 1.8e-7 and 9e-8 (act 1).
// x * sigmoid(x) for these kernels: the library's division is half of its instructions; here a reciprocal and one Newton step, of a number
// between one and two: e^-|x| neither overflows nor makes the reciprocal a number that is not normal.
__device__ __forceinline__ float cm_feature(float x, int act) {
  if (act != 0) return x;
  const float e = expf(-fabsf(x)), y = 1.f + e;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(y));
  r = fmaf(r, fmaf(-y, r, 1.f), r);
  return x * (x < 0.f ? e * r : r);
}

// The numbers of a chunk's contribution to the state that are not finite, by multiply-adds (a call of its own: inside, it costs the kernel registers).
template <typename T>
__device__ __noinline__ void lightning_plain_state(const T* k, const T* v, long long stride, int act, const float* pw, int len, int dim, int cols,
                                                   float* dst, int vdim) {
  for (int i = threadIdx.x; i < dim * cols; i += CM_THREADS) {
    const int d = i / cols, c = i - d * cols;
    float* at = dst + (long long)d * vdim + c;
    if (isfinite(*at)) continue;
    float x = 0.f;
#pragma unroll 8
    for (int s = 0; s < len; ++s)
      x = fmaf(cm_feature(to_float(k[s * stride + d]), act) * pw[len - 1 - s], cm_feature(to_float(v[s * stride + c]), act), x);
    *at = x;
  }
}

template <typename T, int PARTS>
__global__ void __launch_bounds__(CM_THREADS, 4)
lightning_state_kernel(const T* __restrict__ proj, long long row_stride, int k_off, int v_off, const int* __restrict__ seq_start,
                       const float* __restrict__ decay, float* __restrict__ scratch, int max_chunks, int n_heads, int dim, int vdim,
                       int col_blocks, int act) {
  extern __shared__ __align__(16) unsigned char cm_smem[];
  __nv_bfloat16* k_s = reinterpret_cast<__nv_bfloat16*>(cm_smem);      // [3][64][dim + 8]: decay^(len - 1 - s) k_s
  const int k_stride = dim + 8, k_part = CM_CHUNK * k_stride, v_part = CM_CHUNK * CM_ROW;
  __nv_bfloat16* v_s = k_s + 3 * k_part;                               // [PARTS][64][72]
  __shared__ float pw[CM_CHUNK];
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col0 = (blockIdx.y - head * col_blocks) * CM_COLS;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * CM_CHUNK >= n_new) return;
  const int len = min(CM_CHUNK, n_new - chunk * CM_CHUNK);
  const T* rows = proj + (first + (long long)chunk * CM_CHUNK) * row_stride;
  if (threadIdx.x < CM_CHUNK) pw[threadIdx.x] = powf(decay[head], (float)threadIdx.x);
  __syncthreads();
  cm_fill<3>(k_s, CM_CHUNK, dim, k_stride, k_part, [&](int t, int c, float (&x)[8]) {
    if (t < len) cm_load8(rows + t * row_stride + k_off + head * dim + c, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = t < len ? cm_feature(x[u], act) * pw[len - 1 - t] : 0.f;
  });
  cm_fill<PARTS>(v_s, CM_CHUNK, CM_COLS, CM_ROW, v_part, [&](int t, int c, float (&x)[8]) {
    const bool in = t < len && col0 + c < vdim;
    if (in) cm_load8(rows + t * row_stride + v_off + head * vdim + col0 + c, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = in ? cm_feature(x[u], act) : 0.f;
  });
  __syncthreads();
  float* dst = scratch + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim + col0;
  const bool bad = cm_state<3, PARTS>(k_s, k_stride, k_part, v_s, v_part, dim, [&](int d, int c, float x, float y) {
    if (col0 + c < vdim) *reinterpret_cast<float2*>(dst + (long long)d * vdim + c) = make_float2(x, y);
  });
  if (__syncthreads_or(bad))
    lightning_plain_state<T>(rows + k_off + head * dim, rows + v_off + head * vdim + col0, row_stride, act, pw, len, dim, min(CM_COLS, vdim - col0), dst, vdim);
}

// The results of a chunk's tokens (bits of `redo`, from token `first` on) that are no finite numbers, by multiply-adds, a warp together: qk and v
// are the chunk's rows from the head's channels on, v's and out's the block's; pw: the decay's powers.
template <typename T>
__device__ __noinline__ void lightning_plain_rows(unsigned redo, const T* qk, const T* v, long long stride, int q_off, int k_off, int act,
                                                  const float* state, int vdim, const float* pw, int first, int dim, int cols, float* out,
                                                  long long out_stride) {
  const int lane = threadIdx.x & 31;
  auto in = [&](int d, int c) { return state[(long long)d * vdim + c]; };
  bool nan[2];
  cm_nan_columns(dim, cols, in, nan);
  for (; redo; redo &= redo - 1) {
    const int t = first + __ffs(redo) - 1;
    float* at = out + t * out_stride + lane;
    const bool need[2] = {!nan[0] && !isfinite(at[0]), !nan[1] && !isfinite(at[32])};
    if (!__any_sync(0xffffffffu, need[0] || need[1])) continue;
    float x[2];
    cm_plain_row(t, dim, cols, pw[t + 1], [&](int d) { return cm_feature(to_float(qk[t * stride + q_off + d]), act); },
                 [&](int s, int d) { return cm_feature(to_float(qk[s * stride + k_off + d]), act); },
                 [&](int s, int c) { return cm_feature(to_float(v[s * stride + c]), act); }, in, [&](int s, float w) { return w * pw[t - s]; }, x);
    if (need[0]) at[0] = x[0];
    if (need[1]) at[32] = x[1];
  }
}

template <typename T, int PARTS>
__global__ void __launch_bounds__(CM_THREADS, 4)
lightning_out_kernel(const T* __restrict__ proj, long long row_stride, int q_off, int k_off, int v_off, const int* __restrict__ seq_start,
                     const float* __restrict__ decay, float* __restrict__ out, long long out_row_stride,
                     const float* __restrict__ scratch, int max_chunks, int n_heads, int dim, int vdim, int col_blocks, int act) {
  extern __shared__ __align__(16) unsigned char cm_smem[];
  const int k_stride = dim + 8, k_part = CM_CHUNK * k_stride, s_part = max(dim, CM_CHUNK) * CM_ROW;
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(cm_smem);      // [PARTS][64][dim + 8]
  __nv_bfloat16* s_s = q_s + PARTS * k_part;                           // [3][dim][72] the state; then [PARTS][64][dim + 8] k; then [PARTS][64][72] v
  __shared__ float pw[CM_CHUNK + 1];
  pdl_trigger();
  pdl_wait();
  const int chunk = blockIdx.x, seq = blockIdx.z;
  const int head = blockIdx.y / col_blocks, col0 = (blockIdx.y - head * col_blocks) * CM_COLS;
  const int first = seq_start[seq], n_new = seq_start[seq + 1] - first;
  if (chunk * CM_CHUNK >= n_new) return;
  const int len = min(CM_CHUNK, n_new - chunk * CM_CHUNK);
  const long long row0 = first + (long long)chunk * CM_CHUNK;
  const T* rows = proj + row0 * row_stride;
  if (threadIdx.x <= CM_CHUNK) pw[threadIdx.x] = powf(decay[head], (float)threadIdx.x);
  const float* src = scratch + ((((long long)seq * max_chunks + chunk) * n_heads + head) * dim) * vdim + col0;
  cm_fill<3>(s_s, dim, CM_COLS, CM_ROW, s_part, [&](int d, int c, float (&x)[8]) {
    if (col0 + c < vdim) cm_load8(src + (long long)d * vdim + c, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = col0 + c < vdim ? x[u] : 0.f;
  });
  auto fill = [&](__nv_bfloat16* dst, int off) {      // q or k
    cm_fill<PARTS>(dst, CM_CHUNK, dim, k_stride, k_part, [&](int t, int c, float (&x)[8]) {
      if (t < len) cm_load8(rows + t * row_stride + off + head * dim + c, x);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = t < len ? cm_feature(x[u], act) : 0.f;
    });
  };
  fill(q_s, q_off);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  const int ta = warp * 16 + g, tb = ta + 8;      // this thread's rows
  auto query = [&](int d, unsigned (&a)[PARTS][4]) {      // the operand of 16 channels from d on
#pragma unroll
    for (int q = 0; q < PARTS; ++q) cm_ldmatrix(a[q], q_s + q * k_part + (warp * 16 + (lane & 15)) * k_stride + d + (lane >> 4) * 8);
  };
  float o[8][4], o_small[8][4];
  {
    // decay^(t + 1) S_in^T q_t
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) o[j][i] = o_small[j][i] = 0.f;
    for (int d = 0; d < dim; d += 16) {
      unsigned a[PARTS][4];
      query(d, a);
      cm_step_rows<PARTS, 3, 8>(o, o_small, a, s_s, d, s_part);
    }
    const float pa = pw[ta + 1], pb = pw[tb + 1];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[j][i] = (o[j][i] + o_small[j][i]) * (i < 2 ? pa : pb);
      }
  }
  __syncthreads();      // the state has been read
  fill(s_s, k_off);
  __syncthreads();
  float sc[8][4];
  {
    // the scores of this warp's tokens on those up to its last one
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
        const __nv_bfloat16* at = s_s + (8 * j + (lane & 7) + (lane >> 4) * 8) * k_stride + d + (lane >> 3 & 1) * 8;
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
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = i < 2 ? ta : tb, at = 8 * j + t2 + (i & 1);
        sc[j][i] = at <= t ? sc[j][i] * pw[t - at] : 0.f;
      }
  }
  __syncthreads();      // k has been read
  cm_fill<PARTS>(s_s, CM_CHUNK, CM_COLS, CM_ROW, s_part, [&](int t, int c, float (&x)[8]) {
    const bool in = t < len && col0 + c < vdim;
    if (in) cm_load8(rows + t * row_stride + v_off + head * vdim + col0 + c, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = in ? cm_feature(x[u], act) : 0.f;
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
  unsigned redo = cm_bad_rows(ta < len && zeros[0] != 0.f, tb < len && zeros[1] != 0.f);
  if (redo == 0) return;
  __syncwarp();
  const int cols = min(CM_COLS, vdim - col0);
  lightning_plain_rows<T>(redo, rows + head * dim, rows + v_off + head * vdim + col0, row_stride, q_off, k_off, act, src, vdim, pw, warp * 16,
                          dim, min(CM_COLS, vdim - col0), out + row0 * out_row_stride + (long long)head * vdim + col0, out_row_stride);
}

template <typename T, int PARTS>
static int launch_lightning_mma(const T* proj, long long row_stride, int q_off, int k_off, int v_off, float* state, const int* slots,
                                const int* seq_start, const float* decay, float* out, long long out_row_stride, float* scratch,
                                int max_chunks, int n_seqs, int n_heads, int dim, int vdim, int act, cudaStream_t stream) {
  const int col_blocks = (vdim + CM_COLS - 1) / CM_COLS;
  const dim3 grid(max_chunks, n_heads * col_blocks, n_seqs), block(CM_THREADS);
  const size_t rows_k = (size_t)CM_CHUNK * (dim + 8), rows_v = (size_t)CM_CHUNK * CM_ROW;
  const size_t smem_s = 2 * (3 * rows_k + PARTS * rows_v), rows_s = 3 * (size_t)(dim > CM_CHUNK ? dim : CM_CHUNK) * CM_ROW;
  const size_t smem_o = 2 * (PARTS * rows_k + (rows_s > PARTS * rows_k ? rows_s : PARTS * rows_k));
  static SharedMemoryAllowance allowed_s, allowed_o;
  BT_CHECK(allow_shared_memory(allowed_s, lightning_state_kernel<T, PARTS>, smem_s) &&
               allow_shared_memory(allowed_o, lightning_out_kernel<T, PARTS>, smem_o),
           "lightning_scan: cannot reserve %zu bytes of shared memory", smem_s > smem_o ? smem_s : smem_o);
  BT_PDL_OK("lightning_state", launch_pdl(lightning_state_kernel<T, PARTS>, grid, block, smem_s, stream, 1, proj, row_stride, k_off, v_off,
                                          seq_start, decay, scratch, max_chunks, n_heads, dim, vdim, col_blocks, act));
  if ((unsigned long long)state % 16 == 0)
    BT_PDL_OK("lightning_prefix", launch_pdl(lightning_prefix_vec_kernel, dim3((dim * vdim + 511) / 512, n_heads, n_seqs), dim3(128), 0,
                                             stream, 1, scratch, state, slots, seq_start, decay, max_chunks, n_heads, dim, vdim));
  else
    BT_PDL_OK("lightning_prefix", launch_pdl(lightning_prefix_kernel, dim3((dim * vdim + 255) / 256, n_heads, n_seqs), dim3(256), 0,
                                             stream, 1, scratch, state, slots, seq_start, decay, max_chunks, n_heads, dim, vdim));
  BT_PDL_OK("lightning_out", launch_pdl(lightning_out_kernel<T, PARTS>, grid, block, smem_o, stream, 1, proj, row_stride, q_off, k_off,
                                        v_off, seq_start, decay, out, out_row_stride, (const float*)scratch, max_chunks, n_heads, dim,
                                        vdim, col_blocks, act));
  return 0;
}

template <typename T>
static int launch_lightning_chunked(const T* proj, long long row_stride, int q_off, int k_off, int v_off, float* state,
                                    const int* slots, const int* seq_start, const float* decay, float* out,
                                    long long out_row_stride, float* scratch, int max_new, int n_seqs, int n_heads, int dim,
                                    int vdim, int act, cudaStream_t stream) {
  const int col_blocks = (vdim + 63) / 64;
  const int max_chunks = (max_new + LC - 1) / LC;
  BT_CHECK((long long)n_heads * col_blocks <= 65535, "lightning_scan: %d heads x %d column blocks are too many", n_heads, col_blocks);
  const dim3 grid(max_chunks, n_heads * col_blocks, n_seqs), block(256);
  const size_t smem_a = ((size_t)2 * dim * LCP + (size_t)LC * 64 + (size_t)LC * LCP + LC + 4) * sizeof(float);
  const size_t smem_c = ((size_t)dim * LCP + (size_t)dim * 64 + LC + 4) * sizeof(float);
  // 16-byte accesses: every head of every row, of the results and of the states on such a boundary
  constexpr int V = 16 / (int)sizeof(T);
  const int vec = dim % V == 0 && vdim % V == 0 && q_off % V == 0 && k_off % V == 0 && v_off % V == 0 && row_stride % V == 0 &&
                  out_row_stride % 4 == 0 && ((unsigned long long)proj | (unsigned long long)out | (unsigned long long)scratch) % 16 == 0;
  // By the layer's sizes and addresses alone: a sequence's bits must not depend on what else is in the call.  Multiply-adds / parts, us,
  // bfloat16: heads of 64 x 64 with x sigmoid(x) 36 blocks 27 / 32, 192 40 / 39, 512 68 / 47, without it 23 / 21, 35 / 24, 60 / 30; heads
  // of 128 x 128 with it 16 blocks 40 / 49, 256 64 / 55, 1,024 205 / 207.  So few blocks with x sigmoid(x) pay for many.
  if (vec && dim % 16 == 0 && dim <= 128 && vdim % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0) {
    if constexpr (sizeof(T) == 2)
      if (act == 1)
        return launch_lightning_mma<T, 1>(proj, row_stride, q_off, k_off, v_off, state, slots, seq_start, decay, out, out_row_stride,
                                          scratch, max_chunks, n_seqs, n_heads, dim, vdim, act, stream);
    return launch_lightning_mma<T, 3>(proj, row_stride, q_off, k_off, v_off, state, slots, seq_start, decay, out, out_row_stride,
                                      scratch, max_chunks, n_seqs, n_heads, dim, vdim, act, stream);
  }
  auto chunk_kernel = lightning_chunk_kernel<T>;
  auto carry_kernel = lightning_carry_kernel<T>;
  if (smem_a > 48 * 1024)
    BT_CHECK(cudaFuncSetAttribute(chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_a) == cudaSuccess,
             "lightning_scan: cannot reserve %zu bytes of shared memory", smem_a);
  if (smem_c > 48 * 1024)
    BT_CHECK(cudaFuncSetAttribute(carry_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_c) == cudaSuccess,
             "lightning_scan: cannot reserve %zu bytes of shared memory", smem_c);
  BT_PDL_OK("lightning_chunk", launch_pdl(chunk_kernel, grid, block, smem_a, stream, 1, proj, row_stride, q_off, k_off, v_off,
                                          seq_start, decay, out, out_row_stride, scratch, max_chunks, n_heads, dim, vdim,
                                          col_blocks, act, vec));
  BT_PDL_OK("lightning_prefix", launch_pdl(lightning_prefix_kernel, dim3((dim * vdim + 255) / 256, n_heads, n_seqs), block, 0,
                                           stream, 1, scratch, state, slots, seq_start, decay, max_chunks, n_heads, dim,
                                           vdim));
  BT_PDL_OK("lightning_carry", launch_pdl(carry_kernel, grid, block, smem_c, stream, 1, proj, row_stride, q_off, seq_start,
                                          decay, out, out_row_stride, (const float*)scratch, max_chunks, n_heads, dim, vdim,
                                          col_blocks, act, vec));
  return 0;
}

}  // namespace bt

// Floats of scratch the chunked form needs for runs of up to `max_new` new tokens.
extern "C" long long bt_lightning_chunked_scratch_floats(int n_seqs, int max_new, int n_heads, int dim, int vdim) {
  return (long long)n_seqs * ((max_new + bt::LC - 1) / bt::LC) * n_heads * dim * vdim;
}

// The recurrence for steps that bring long runs of tokens: the same results as bt_lightning_scan (beyond rounding), the
// chunks of a run worked side by side.  `max_new`: no sequence of the step brings more tokens than this.
extern "C" int bt_lightning_chunked(const void* proj, long long row_stride, int q_off, int k_off, int v_off, float* state,
                                    const int* slots, const int* seq_start, const float* decay, float* out,
                                    long long out_row_stride, float* scratch, int max_new, int n_seqs, int n_heads, int dim,
                                    int vdim, int act, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && dim > 0 && dim <= 256 && vdim > 0 && n_seqs >= 0 && n_seqs <= 65535 && max_new > 0 && scratch,
           "lightning_chunked: bad sizes seqs=%d heads=%d dim=%d vdim=%d max_new=%d", n_seqs, n_heads, dim, vdim, max_new);
  if (n_seqs == 0) return 0;
  if (dtype == kF32)
    return launch_lightning_chunked<float>((const float*)proj, row_stride, q_off, k_off, v_off, state, slots, seq_start,
                                           decay, out, out_row_stride, scratch, max_new, n_seqs, n_heads, dim, vdim, act, stream);
  if (dtype == kBF16)
    return launch_lightning_chunked<__nv_bfloat16>((const __nv_bfloat16*)proj, row_stride, q_off, k_off, v_off, state,
                                                   slots, seq_start, decay, out, out_row_stride, scratch, max_new, n_seqs,
                                                   n_heads, dim, vdim, act, stream);
  return fail("lightning_chunked: unknown dtype %d", dtype);
}
