// Causal attention for steps that bring several tokens per sequence, with plain 32-bit
// arithmetic: scores, online softmax, and the value mix are all fused multiply-adds in 32-bit,
// so this kernel serves the true 32-bit path (but for what attention_prefill_parts.cuh takes: more than a few queries of heads of 16,
// 32, 48 or 64 channels on 16-byte boundaries) and any head size the tensor-core kernel refuses.
// The S x S score plane is never stored.
//
// A block is 8 Q queries of one (sequence, head) and walks their keys in tiles of 64; a thread holds Q queries x 4 keys of the
// scores and Q queries x 4 channels (of every 64) of the output, so that at Q = 4 a 16-byte read of shared memory, which takes
// a warp four cycles of the multiprocessor, feeds eight multiply-adds: these reads are what bounds it.  Keys, values and
// queries lie in shared memory as rows (+ 4 numbers: eight consecutive rows meet all 32 banks once).  A tile's keys are asked
// for when the scores of the tile before it are done, its values when that tile's value mix is: by cp.async where 32-bit heads
// lie on 16-byte boundaries, else through registers, several reads at once.
// Q is 4 where blocks of 32 queries are three a multiprocessor, 2 where blocks of 16 are four for every three
// multiprocessors, else 1 (decode steps of head sizes that the decode kernels do not take, short or few prompts).  A query's sums
// are formed in the same order whatever Q is.  Measured with 12 heads, in us: with a warp a query and a lane a key, the version
// before; with 32 queries in every block; and so.  Prompts of 64 channels, 32-bit: of 37, 268 and 499 tokens 217 / 79 / 76, one of
// 129 28 / 22 / 12; 2 x 1,024 tokens of 96 channels, bfloat16, 1,097 / 494 / 303; one token for each of 64 sequences behind 900:
// 50 channels, 32-bit, 267 / 1,187 / 179, 96 channels, bfloat16, 330 / 2,184 / 202.
//
// Query t of sequence s sits at position past[s] + (t - seq_start[s]); key j is visible when
// j <= position (causal) and j > position - window (window > 0).  A query that sees no key
// yields zeros.
#include "common.cuh"

#include <type_traits>

namespace bt {

constexpr int PF_BK = 64;      // keys per tile
constexpr int PF_THREADS = 128;
constexpr int PF_MAXG = 4;     // groups of 64 channels: head_dim <= 256

// numbers between rows of queries, keys and values in shared memory
__host__ __device__ __forceinline__ int pf_stride(int head_dim) { return (head_dim + 3) / 4 * 4 + 4; }

// G: groups of 64 channels that hold a head.  VEC: rows whose heads start on 16-byte boundaries.  Q: queries a thread holds.
// the block's part of sequence `seq` and head `head`: queries q0 to q0 + 8 Q
template <typename T, int G, bool VEC, int Q>
__device__ __forceinline__ void pf_block(float* smem, const T* __restrict__ q, long long q_row_stride, const KvView& kv, T* __restrict__ out,
                                         int seq, int head, int q0, int t0, int n_new, int past, int n_heads, int n_kv_heads, int head_dim,
                                         float scale, int causal, int window) {
  constexpr int BQ = 8 * Q;      // queries per block
  const int kv_len = past + n_new;
  const int kv_head = head / (n_heads / n_kv_heads);
  const int nq = min(BQ, n_new - q0);
  const int S = pf_stride(head_dim), wide = S - 4;    // (channels past the head's are zeros)
  float* Qs = smem;                        // [BQ][S]
  float* Ks = Qs + BQ * S;                 // [PF_BK][S]
  float* Vs = Ks + PF_BK * S;              // [PF_BK][S]
  float* Ps = Vs + PF_BK * S;              // [BQ][PF_BK + 4]
  constexpr int PS = PF_BK + 4;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;  // keys tx, tx + 16, ... and channels 4 tx .. (of every 64); queries Q ty ..
  const bool works = (tid >> 5) * 2 * Q < nq;         // (a warp without a query only copies)

  for (int i = tid; i < BQ * wide; i += PF_THREADS) {
    const int r = i / wide, c = i - r * wide;
    Qs[r * S + c] = r < nq && c < head_dim ? to_float(q[(long long)(t0 + q0 + r) * q_row_stride + head * head_dim + c]) * scale : 0.f;
  }
  // key range this block can see
  const int pos_first = past + q0, pos_last = past + q0 + nq - 1;
  int k_hi = causal ? min(kv_len, pos_last + 1) : kv_len;
  int k_lo = window > 0 ? max(0, pos_first - window + 1) : 0;
  const int tile_lo = k_lo / PF_BK, tile_hi = (k_hi + PF_BK - 1) / PF_BK;

  // A tile's rows of keys or values that some query sees, up to a multiple of four (the rest zeros).  Where a tile lies in one
  // page, as with the library's pages of 64, its rows lie evenly apart.
  const bool together = kv.table == nullptr || kv.page_size % PF_BK == 0;
  const long long apart = kv.table ? head_dim : kv.row_stride;
  auto stage = [&](int tile, const void* base, float* dst) {
    if (tile < tile_hi) {
      const int rows = min(PF_BK, k_hi - tile * PF_BK), need = (rows + 3) & ~3;
      const T* first = kv.table ? kv_row<T>(base, kv, seq, kv_head, n_kv_heads, head_dim, tile * PF_BK)
                                : reinterpret_cast<const T*>(base) + (long long)(t0 + tile * PF_BK) * apart + kv_head * head_dim;
      auto row_at = [&](int r) { return together ? first + r * apart : kv_row<T>(base, kv, seq, kv_head, n_kv_heads, head_dim, tile * PF_BK + r); };
      if constexpr (VEC && sizeof(T) == 2) {
        // pieces of 8 numbers one after the other, several reads in flight together
        constexpr int AHEAD = Q == 1 ? 8 : 4;
        const int pieces = head_dim / 8, step_row = PF_THREADS / pieces, step_piece = PF_THREADS - step_row * pieces;
        int r = tid / pieces, c = tid - r * pieces;
        while (r < need) {
          uint4 raw[AHEAD] = {};
          float* at[AHEAD];
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            at[u] = r < need ? dst + r * S + 8 * c : nullptr;
            if (r < rows) raw[u] = *reinterpret_cast<const uint4*>(row_at(r) + 8 * c);
            r += step_row;
            c += step_piece;
            if (c >= pieces) {
              c -= pieces;
              ++r;
            }
          }
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            if (at[u] == nullptr) break;
            float x[8];
            unpack16(raw[u], x);
            *reinterpret_cast<float4*>(at[u]) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4*>(at[u] + 4) = make_float4(x[4], x[5], x[6], x[7]);
          }
        }
      } else if constexpr (VEC && Q == 4) {
        // piece by piece (with eight threads a row, prompts of 1,024 took up to a fifth longer where a head is no multiple of 32)
        const int pieces = head_dim / 4;
        for (int i = tid; i < need * pieces; i += PF_THREADS) {
          const int r = i / pieces, c = (i - r * pieces) * 4;
          const T* src = row_at(min(r, rows - 1)) + c;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst + r * S + c)),
                       "l"(src), "r"(r < rows ? 16 : 0) : "memory");
        }
      } else {
        // eight threads a row, PASSES rows a thread
        constexpr int BY = PF_THREADS / 8, PASSES = PF_BK / BY;
        const int part = tid & 7, row0 = tid >> 3;
        const T* src[PASSES];
#pragma unroll
        for (int i = 0; i < PASSES; ++i) src[i] = row_at(min(row0 + i * BY, rows - 1));
        if constexpr (VEC) {
#pragma unroll
          for (int i = 0; i < PASSES; ++i) {
            const int r = row0 + i * BY;
            if (r >= need) break;
            for (int c = 4 * part; c < head_dim; c += 32)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst + r * S + c)),
                           "l"(src[i] + c), "r"(r < rows ? 16 : 0) : "memory");
          }
        } else {
          for (int c = part; c < wide; c += 8) {
            float x[PASSES];
#pragma unroll
            for (int i = 0; i < PASSES; ++i) x[i] = c < head_dim && row0 + i * BY < rows ? to_float(src[i][c]) : 0.f;
#pragma unroll
            for (int i = 0; i < PASSES; ++i)
              if (row0 + i * BY < need) dst[(row0 + i * BY) * S + c] = x[i];
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  float m[Q], l[Q], acc[Q][4 * G];
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < 4 * G; ++c) acc[i][c] = 0.f;
  }

  stage(tile_lo, kv.k, Ks);
  stage(tile_lo, kv.v, Vs);
  for (int tile = tile_lo; tile < tile_hi; ++tile) {
    const int rows = min(PF_BK, k_hi - tile * PF_BK);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");      // the keys (the values may still be on their way)
    __syncthreads();
    float s[Q][4];
#pragma unroll
    for (int i = 0; i < Q; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
    // the scores of a tile's first 16 J keys (what lies behind the tile's rows is not looked at below)
    auto scores = [&](auto groups) {
      constexpr int J = decltype(groups)::value;
#pragma unroll 4
      for (int c = 0; c < wide; c += 4) {
        float4 a[Q], b[J];
#pragma unroll
        for (int i = 0; i < Q; ++i) a[i] = *reinterpret_cast<const float4*>(Qs + (Q * ty + i) * S + c);
#pragma unroll
        for (int j = 0; j < J; ++j) b[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * S + c);
#pragma unroll
        for (int i = 0; i < Q; ++i)
#pragma unroll
          for (int j = 0; j < J; ++j) {
            s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
            s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
            s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
            s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
          }
      }
    };
    if (works) {
      if (rows > 32) scores(std::integral_constant<int, 4>{});
      else if (rows > 16) scores(std::integral_constant<int, 2>{});
      else scores(std::integral_constant<int, 1>{});
    }
    __syncthreads();                        // everyone has read the keys
    stage(tile + 1, kv.k, Ks);
    // online softmax: a query's sixteen lanes agree on its maximum and sum
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      if (!works) break;
      const int qpos = past + q0 + Q * ty + i;
      bool seen[4];
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kp = tile * PF_BK + tx + 16 * j;
        seen[j] = kp < k_hi && (!causal || kp <= qpos) && (window <= 0 || kp > qpos - window);
        if (seen[j]) top = fmaxf(top, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float m_new = fmaxf(m[i], top);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float corr = expf(m[i] - m_use);          // m = -inf gives 0
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = seen[j] ? expf(s[i][j] - m_use) : 0.f;
        Ps[(Q * ty + i) * PS + tx + 16 * j] = p;
        sum += p;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[i] = l[i] * corr + sum;
      m[i] = m_new;
#pragma unroll
      for (int c = 0; c < 4 * G; ++c) acc[i][c] *= corr;
    }
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");      // the values (the next keys may still be on their way)
    __syncthreads();                        // (and the weights, which a warp alone reads and writes)
#pragma unroll 2
    for (int k = 0; k < rows && works; k += 4) {
      float4 p[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i) p[i] = *reinterpret_cast<const float4*>(Ps + (Q * ty + i) * PS + k);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int c = 64 * g + 4 * tx;
        if (c >= wide) continue;
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(Vs + (k + u) * S + c);
#pragma unroll
        for (int i = 0; i < Q; ++i) {
          const float w[4] = {p[i].x, p[i].y, p[i].z, p[i].w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            acc[i][4 * g] = fmaf(w[u], v[u].x, acc[i][4 * g]);
            acc[i][4 * g + 1] = fmaf(w[u], v[u].y, acc[i][4 * g + 1]);
            acc[i][4 * g + 2] = fmaf(w[u], v[u].z, acc[i][4 * g + 2]);
            acc[i][4 * g + 3] = fmaf(w[u], v[u].w, acc[i][4 * g + 3]);
          }
        }
      }
    }
    __syncthreads();                        // everyone has read the values
    stage(tile + 1, kv.v, Vs);
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int qi = Q * ty + i;
    if (qi >= nq) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    T* dst = out + (long long)(t0 + q0 + qi) * ((long long)n_heads * head_dim) + head * head_dim;
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = 64 * g + 4 * tx + u;
        if (c < head_dim) dst[c] = from_float<T>(acc[i][4 * g + u] * inv);
      }
  }
}

template <typename T, int G, bool VEC, int Q>
__global__ void __launch_bounds__(PF_THREADS)
attention_prefill_simt_kernel(const T* __restrict__ q, long long q_row_stride, KvView kv, T* __restrict__ out,
                              const int* __restrict__ seq_start, const int* __restrict__ past_len, int n_heads,
                              int n_kv_heads, int head_dim, float scale, int causal, int window) {
  extern __shared__ __align__(16) float smem[];
  const int seq = blockIdx.y, t0 = seq_start[seq], n_new = seq_start[seq + 1] - t0;
  // longest tiles first: they see the most keys
  const int q0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * 8 * Q;
  if (q0 >= n_new) return;
  pf_block<T, G, VEC, Q>(smem, q, q_row_stride, kv, out, seq, blockIdx.z, q0, t0, n_new, past_len[seq], n_heads, n_kv_heads, head_dim, scale,
                         causal, window);
}

template <typename T, int G, bool VEC, int Q>
static int launch_pf(const void* q, long long q_row_stride, const KvView& view, void* out, const int* seq_start, const int* past_len,
                     int n_seqs, int max_new, int n_heads, int n_kv_heads, int head_dim, float scale, int causal, int window,
                     cudaStream_t stream) {
  constexpr int BQ = 8 * Q;
  auto kern = attention_prefill_simt_kernel<T, G, VEC, Q>;
  constexpr size_t most = sizeof(float) * ((size_t)(BQ + 2 * PF_BK) * (64 * G + 4) + (size_t)BQ * (PF_BK + 4));
  const size_t smem = sizeof(float) * ((size_t)(BQ + 2 * PF_BK) * pf_stride(head_dim) + (size_t)BQ * (PF_BK + 4));
  static SharedMemoryAllowance allowed;
  BT_CHECK(allow_shared_memory(allowed, kern, most), "attention_prefill_simt: cannot reserve %zu bytes of shared memory", most);
  const dim3 grid((max_new + BQ - 1) / BQ, n_seqs, n_heads);
  kern<<<grid, PF_THREADS, smem, stream>>>((const T*)q, q_row_stride, view, (T*)out, seq_start, past_len, n_heads, n_kv_heads,
                                           head_dim, scale, causal, window);
  return 0;
}

template <typename T, bool VEC, int Q, typename... Args>
static int launch_pf_sized(int head_dim, Args... args) {
  if (head_dim <= 64) return launch_pf<T, 1, VEC, Q>(args...);
  if (head_dim <= 128) return launch_pf<T, 2, VEC, Q>(args...);
  if (head_dim <= 192) return launch_pf<T, 3, VEC, Q>(args...);
  return launch_pf<T, 4, VEC, Q>(args...);
}

template <typename T, bool VEC, typename... Args>
static int launch_pf_queries(int queries, int head_dim, Args... args) {
  if (queries == 1) return launch_pf_sized<T, VEC, 1>(head_dim, args...);
  if (queries == 2) return launch_pf_sized<T, VEC, 2>(head_dim, args...);
  return launch_pf_sized<T, VEC, 4>(head_dim, args...);
}

}  // namespace bt

#include "attention_prefill_parts.cuh"

// kv_table == nullptr selects the packed view: keys and values are read from the step's own
// projections (k, v point at the first key/value channel of row 0, rows kv_row_stride apart).
extern "C" int bt_attention_prefill_simt(const void* q, long long q_row_stride, const void* k, const void* v,
                                         const int* kv_table, int table_stride, int table_len, int page_size,
                                         long long kv_row_stride, void* out, const int* seq_start,
                                         const int* past_len, int n_seqs, int max_new, int n_heads, int n_kv_heads,
                                         int head_dim, float scale, int causal, int window, int dtype,
                                         cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(head_dim > 0 && head_dim <= 64 * PF_MAXG,
           "attention_prefill_simt: head_dim %d must be at least 1 and at most %d", head_dim, 64 * PF_MAXG);
  BT_CHECK(n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0,
           "attention_prefill_simt: %d query heads cannot share %d key heads", n_heads, n_kv_heads);
  BT_CHECK(n_seqs <= 65535 && n_heads <= 65535, "attention_prefill_simt: too many sequences or heads for one launch");
  if (n_seqs == 0 || max_new == 0) return 0;
  KvView view{k, v, kv_table, table_stride, table_len > 0 ? table_len : 1, page_size > 0 ? page_size : 1,
              kv_row_stride, seq_start};
  if (dtype == kF32 && attention_prefill_parts_takes(q, q_row_stride, view, out, head_dim, max_new))
    return launch_attention_prefill_parts((const float*)q, q_row_stride, view, (float*)out, seq_start, past_len, n_seqs, max_new, n_heads,
                                          n_kv_heads, head_dim, scale, causal, window, stream);
  // 16-byte copies need every head of every row on a 16-byte boundary
  const int piece = dtype == kF32 ? 4 : 8;
  const bool vec = head_dim % piece == 0 && ((unsigned long long)k | (unsigned long long)v) % 16 == 0 &&
                   (kv_table != nullptr || kv_row_stride % piece == 0);
  const int sms = sm_count();
  BT_CHECK(sms > 0, "attention_prefill_simt: cannot read the number of multiprocessors of the current device");
  const long long columns = (long long)n_seqs * n_heads;
  const int queries = max_new > 16 && columns * ((max_new + 31) / 32) >= 3ll * sms      ? 4
                      : max_new > 8 && 3 * columns * ((max_new + 15) / 16) >= 4ll * sms ? 2
                                                                                         : 1;
  int rc;
#define BT_PF(T, VEC)                                                                                                          \
  rc = launch_pf_queries<T, VEC>(queries, head_dim, q, q_row_stride, view, out, seq_start, past_len, n_seqs, max_new, n_heads, \
                                 n_kv_heads, head_dim, scale, causal, window, stream)
  if (dtype == kF32) {
    if (vec) BT_PF(float, true); else BT_PF(float, false);
  } else if (dtype == kBF16) {
    if (vec) BT_PF(__nv_bfloat16, true); else BT_PF(__nv_bfloat16, false);
  } else {
    return fail("attention_prefill_simt: unknown dtype %d", dtype);
  }
#undef BT_PF
  if (rc != 0) return rc;
  BT_LAUNCH_OK("attention_prefill_simt");
  return 0;
}
