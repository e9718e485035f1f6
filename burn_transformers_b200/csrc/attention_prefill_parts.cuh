// Causal attention for steps that bring several tokens per sequence in the true 32-bit path, on tensor cores with no operand's bits
// given up (chunk_mma.cuh: numbers as three bfloat16 parts; the first parts' products begin from zero at every 16 of a sum and are
// added in 32-bit registers).  Scores, online softmax and value mix are those of attention_prefill_simt.cu, which takes every other
// head size and type; the S x S score plane is never stored.
//
// A block is 16, 32 or 64 queries of one (sequence, head) and walks their keys in tiles of 64; two or four warps share 16 queries: each
// forms the scores of a part of a tile's keys, reads all of them back, forms the same softmax and mixes a part of the channels.  The
// parts of the queries, of a tile's keys and of its values lie in shared memory; the next tile waits in registers as 32-bit numbers.  The
// multiply-add kernel is bound by its reads of shared memory, this one by its instructions and the chains of a tile (45 % of all issue
// slots and 41 % of the tensor pipe at 64 queries).  A sequence with eight new tokens or fewer is formed by multiply-adds here too: of a
// tile's 16 rows most would be empty, and splitting the keys and values costs what it does for 16 (64 sequences with one token
// behind 900: 153 us in parts, 123 by multiply-adds).  Multiply-adds / parts, us, 12 heads of 64: prompts of 37, 268 and 499 tokens 76 / 36,
// one of 129 11.4 / 10.0, one of 1,024 116 / 69, 24 tokens behind 300 for each of 32 sequences 67 / 51; 16 heads, 4 x 1,000 428 / 214; three of
// 300 tokens with heads of 16, 32 and 48 channels 29 / 13, 31 / 16 and 36 / 22.  Error against 64 bits: 1.3e-7 where it was 3.2e-7 (4 x 1,000).
//
// A query's sums do not depend on which others are in the call: tiles begin at multiples of 64 keys, and what a query does not see
// adds zeros.  Query t of sequence s sits at position past[s] + (t - seq_start[s]); key j is visible when j <= position (causal) and
// j > position - window (window > 0).  A query that sees no key yields zeros.
#pragma once
#include "chunk_mma.cuh"
#include "common.cuh"

namespace bt {

constexpr int AP_BK = 64;                // keys per tile
constexpr int AP_FEW = 8;                // new tokens of a sequence that are left to the multiply-adds
constexpr int AP_SCORES = AP_BK + 8;     // numbers between the rows of scores (pairs of a half warp's rows meet all banks once)

// big += a0 b0, small += the other products of the parts, for tiles of eight columns side by side (b: for two tiles their operands, part
// by part, the first's two registers, then the second's).  A tile's five smaller products wait for one another; the tiles do not.
template <int TILES>
__device__ __forceinline__ void ap_products(float (&big)[TILES][4], float (&small)[TILES][4], const unsigned (&a)[3][4],
                                            const unsigned (&b)[TILES / 2][3][4]) {
  float x[TILES][4];
#pragma unroll
  for (int t = 0; t < TILES; ++t) cm_mma_zero(x[t], a[0], b[t / 2][0][2 * (t & 1)], b[t / 2][0][2 * (t & 1) + 1]);
#pragma unroll
  for (int q = 2; q > 0; --q)
#pragma unroll
    for (int pa = 0; pa <= q; ++pa)
#pragma unroll
      for (int t = 0; t < TILES; ++t) cm_mma(small[t], a[pa], b[t / 2][q - pa][2 * (t & 1)], b[t / 2][q - pa][2 * (t & 1) + 1]);
#pragma unroll
  for (int t = 0; t < TILES; ++t) cm_add(big[t], x[t]);
}

// A sequence with AP_FEW new tokens or fewer, by multiply-adds.
template <int HD>
__device__ __noinline__ void ap_few(float* smem, const float* q, long long q_row_stride, KvView kv, float* out, int seq, int head, int t0,
                                    int n_new, int past, int n_heads, int n_kv_heads, float scale, int causal, int window) {
  pf_block<float, 1, true, 1>(smem, q, q_row_stride, kv, out, seq, head, 0, t0, n_new, past, n_heads, n_kv_heads, HD, scale, causal, window);
}

// One query's result by multiply-adds, a warp together, in the sets of 16 channels that are the warp's: for the queries whose parts are
// not all numbers (an infinity, or a number that rounds to one, has no parts).
template <int HD, int SHARE>
__device__ __noinline__ void ap_plain(const float* __restrict__ q, KvView kv, float* __restrict__ out, int seq, int t0, int kv_head,
                                      int n_kv_heads, float scale, int first, int last, int part) {
  const int lane = threadIdx.x & 31;
  float m = -INFINITY, l = 0.f, acc[2] = {0.f, 0.f};
  for (int j = first; j <= last && !isnan(l); ++j) {      // (once the sum of the weights is NaN the rest changes nothing)
    const long long at = (long long)(t0 + j) * kv.row_stride + kv_head * HD;
    const float* k = kv.table ? kv_row<float>(kv.k, kv, seq, kv_head, n_kv_heads, HD, j) : reinterpret_cast<const float*>(kv.k) + at;
    const float* v = kv.table ? kv_row<float>(kv.v, kv, seq, kv_head, n_kv_heads, HD, j) : reinterpret_cast<const float*>(kv.v) + at;
    float s = 0.f;
    for (int c = lane; c < HD; c += 32) s = fmaf(q[c] * scale, k[c], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float m_new = fmaxf(m, s), use = m_new == -INFINITY ? 0.f : m_new, corr = expf(m - use), p = expf(s - use);
    l = l * corr + p;
    m = m_new;
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (lane + 32 * i < HD) acc[i] = fmaf(p, v[lane + 32 * i], acc[i] * corr);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (lane + 32 * i < HD && (lane + 32 * i) / 16 % SHARE == part) out[lane + 32 * i] = l > 0.f || isnan(l) ? acc[i] / l : 0.f;
}

template <int HD, int BQ, int WARPS, int BLOCKS>
__global__ void __launch_bounds__(WARPS * 32, BLOCKS)
attention_prefill_parts_kernel(const float* __restrict__ q, long long q_row_stride, KvView kv, float* __restrict__ out,
                               const int* __restrict__ seq_start, const int* __restrict__ past_len, int n_heads, int n_kv_heads,
                               float scale, int causal, int window) {
  constexpr int THREADS = WARPS * 32, QS = HD + 8, Q_PART = BQ * QS, K_PART = AP_BK * QS;
  constexpr int SHARE = WARPS / (BQ / 16);                 // warps for the same 16 queries
  constexpr int OWN = 8 / SHARE;                           // tiles of eight keys whose scores a warp forms
  constexpr int SETS = (HD / 16 + SHARE - 1) / SHARE;      // of 16 channels that a warp mixes: its number among the SHARE, then every SHARE-th
  constexpr int PIECES = AP_BK * HD / 8 / THREADS > 0 ? AP_BK * HD / 8 / THREADS : 1;      // of eight numbers, a thread's share of a tile
  constexpr bool UNEVEN = PIECES * THREADS * 8 != AP_BK * HD;
  constexpr int MINE = UNEVEN ? PIECES + 1 : PIECES;
  extern __shared__ __align__(16) unsigned char ap_smem[];
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(ap_smem);      // [3][BQ][HD + 8], times the scale
  __nv_bfloat16* k_s = q_s + 3 * Q_PART;                               // [3][64][HD + 8]
  __nv_bfloat16* v_s = k_s + 3 * K_PART;                               // [3][64][HD + 8]
  float* s_s = reinterpret_cast<float*>(v_s + 3 * K_PART);             // [BQ][72]
  pdl_trigger();
  pdl_wait();
  const int seq = blockIdx.y, head = blockIdx.x;
  const int t0 = seq_start[seq], n_new = seq_start[seq + 1] - t0;
  // every head's and sequence's last queries first: they see the most keys
  const int q0 = ((int)gridDim.z - 1 - (int)blockIdx.z) * BQ;
  if (q0 >= n_new) return;
  if (n_new <= AP_FEW) {
    if (threadIdx.x < PF_THREADS)
      ap_few<HD>(reinterpret_cast<float*>(ap_smem), q, q_row_stride, kv, out, seq, head, t0, n_new, past_len[seq], n_heads, n_kv_heads, scale,
                 causal, window);
    return;
  }
  const int past = past_len[seq], kv_head = head / (n_heads / n_kv_heads), nq = min(BQ, n_new - q0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  const int rows = warp / SHARE * 16, part = warp % SHARE;
  // key range this block can see
  const int pos_first = past + q0, pos_last = past + q0 + nq - 1;
  const int k_hi = causal ? min(past + n_new, pos_last + 1) : past + n_new;
  const int k_lo = window > 0 ? max(0, pos_first - window + 1) : 0;
  const int tile_lo = k_lo / AP_BK, tile_hi = (k_hi + AP_BK - 1) / AP_BK;
  // a tile's rows lie evenly apart where it lies in one page (the library's pages of 64) or in the step's own rows
  const bool together = kv.table == nullptr || kv.page_size % AP_BK == 0;
  const long long apart = kv.table ? HD : kv.row_stride;
  auto fetch = [&](int tile, const void* base, float (&x)[MINE][8]) {
    if (tile >= tile_hi) return;
    const int n = min(AP_BK, k_hi - tile * AP_BK);
    const float* first = kv.table ? kv_row<float>(base, kv, seq, kv_head, n_kv_heads, HD, tile * AP_BK)
                                  : reinterpret_cast<const float*>(base) + (long long)(t0 + tile * AP_BK) * apart + kv_head * HD;
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      const int r = (tid + i * THREADS) / (HD / 8), c = (tid + i * THREADS) % (HD / 8) * 8;
      if (UNEVEN && r >= AP_BK) break;
      const float* src = together ? first + r * apart : kv_row<float>(base, kv, seq, kv_head, n_kv_heads, HD, min(tile * AP_BK + r, k_hi - 1));
      if (r < n) cm_load8(src + c, x[i]);
      else
#pragma unroll
        for (int u = 0; u < 8; ++u) x[i][u] = 0.f;
    }
  };
  auto put = [&](__nv_bfloat16* dst, const float (&x)[MINE][8]) {
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      const int r = (tid + i * THREADS) / (HD / 8), c = (tid + i * THREADS) % (HD / 8) * 8;
      if (UNEVEN && r >= AP_BK) break;
      unsigned parts[4][3];
#pragma unroll
      for (int u = 0; u < 4; ++u) cm_split<3>(x[i][2 * u], x[i][2 * u + 1], parts[u]);
#pragma unroll
      for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(dst + p * K_PART + r * QS + c) = make_uint4(parts[0][p], parts[1][p], parts[2][p], parts[3][p]);
    }
  };
  float kx[MINE][8], vx[MINE][8];
  fetch(tile_lo, kv.k, kx);
  fetch(tile_lo, kv.v, vx);
  for (int i = tid; i < BQ * HD / 8; i += THREADS) {
    const int r = i / (HD / 8), c = i % (HD / 8) * 8;
    float x[8] = {};
    if (r < nq) cm_load8(q + (long long)(t0 + q0 + r) * q_row_stride + head * HD + c, x);
    unsigned parts[4][3];
#pragma unroll
    for (int u = 0; u < 4; ++u) cm_split<3>(x[2 * u] * scale, x[2 * u + 1] * scale, parts[u]);
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint4*>(q_s + p * Q_PART + r * QS + c) = make_uint4(parts[0][p], parts[1][p], parts[2][p], parts[3][p]);
  }
  const bool works = rows < nq;                            // (warps without a query only copy)
  const int warp_first = pos_first + rows, warp_last = min(pos_last, pos_first + rows + 15);
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};  // of this thread's two queries
  float o[SETS][2][4] = {}, o_small[SETS][2][4] = {};
  // is any of the 16 keys from `key` on seen by any of the warp's queries?
  auto any = [&](int key) { return key < k_hi && (!causal || key <= warp_last) && (window <= 0 || key + 15 > warp_first - window); };
  for (int tile = tile_lo; tile < tile_hi; ++tile) {
    const int key0 = tile * AP_BK;
    put(k_s, kx);
    put(v_s, vx);
    __syncthreads();
    fetch(tile + 1, kv.k, kx);
    fetch(tile + 1, kv.v, vx);
    if (works && (!causal || key0 <= warp_last)) {
      // the scores of this warp's share of the keys
      const int own = part * OWN;
      float s[OWN][4] = {}, s_small[OWN][4] = {};
      if (any(key0 + 8 * own) || (OWN > 2 && any(key0 + 8 * own + 16))) {
#pragma unroll
        for (int d = 0; d < HD; d += 16) {
          unsigned a[3][4], b[OWN / 2][3][4];
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            cm_ldmatrix(a[p], q_s + p * Q_PART + (rows + (lane & 15)) * QS + d + (lane >> 4) * 8);
#pragma unroll
            for (int j = 0; j < OWN / 2; ++j)
              cm_ldmatrix(b[j][p], k_s + p * K_PART + (8 * own + 16 * j + (lane & 7) + (lane >> 4) * 8) * QS + d + (lane >> 3 & 1) * 8);
          }
          ap_products<OWN>(s, s_small, a, b);
        }
      }
      const bool all = key0 + AP_BK <= k_hi && (!causal || key0 + AP_BK - 1 <= warp_first) && (window <= 0 || key0 > warp_last - window);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int pos = warp_first + g + 8 * e;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
          float x[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int kp = key0 + 8 * (own + j) + t2 + u;
            const bool seen = all || (kp < k_hi && (!causal || kp <= pos) && (window <= 0 || kp > pos - window));
            x[u] = seen ? s[j][2 * e + u] + s_small[j][2 * e + u] : -INFINITY;
          }
          *reinterpret_cast<float2*>(s_s + (rows + g + 8 * e) * AP_SCORES + 8 * (own + j) + t2) = make_float2(x[0], x[1]);
        }
      }
      asm volatile("bar.sync %0, %1;\n" ::"r"(1 + warp / SHARE), "n"(32 * SHARE) : "memory");
      // softmax over all 64 keys: the warps of the same queries form the same numbers
      float w[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 x = *reinterpret_cast<const float2*>(s_s + (rows + g + 8 * e) * AP_SCORES + 8 * j + t2);
          w[j][2 * e] = x.x;
          w[j][2 * e + 1] = x.y;
        }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float top = -INFINITY, sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) top = fmaxf(top, fmaxf(w[j][2 * e], w[j][2 * e + 1]));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float m_new = fmaxf(m[e], top), use = m_new == -INFINITY ? 0.f : m_new;
        const float corr = expf(m[e] - use);          // m = -inf gives 0
        m[e] = m_new;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            w[j][2 * e + u] = expf(w[j][2 * e + u] - use);      // (what is not seen: exp of minus infinity)
            sum += w[j][2 * e + u];
          }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l[e] = l[e] * corr + sum;
#pragma unroll
        for (int c = 0; c < SETS; ++c)
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              o[c][i][2 * e + u] *= corr;
              o_small[c][i][2 * e + u] *= corr;
            }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {      // 16 keys at a time
        if (!any(key0 + 16 * j)) continue;
        unsigned a[3][4], b[SETS][3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          unsigned parts[3];
          cm_split<3>(w[2 * j + (i >> 1)][2 * (i & 1)], w[2 * j + (i >> 1)][2 * (i & 1) + 1], parts);
#pragma unroll
          for (int p = 0; p < 3; ++p) a[p][i] = parts[p];
        }
#pragma unroll
        for (int c = 0; c < SETS; ++c)
#pragma unroll
          for (int p = 0; p < 3; ++p)      // (a set past the head's last: the first one's, not used)
            cm_ldmatrix_t(b[c][p], v_s + p * K_PART + (16 * j + (lane & 15)) * QS + (lane >> 4) * 8 +
                                       16 * (part + c * SHARE < HD / 16 ? part + c * SHARE : 0));
        ap_products<2 * SETS>(reinterpret_cast<float(&)[2 * SETS][4]>(o), reinterpret_cast<float(&)[2 * SETS][4]>(o_small), a, b);
      }
    }
    __syncthreads();      // everyone has read the keys, the values and the scores
  }
  if (!works) return;
  bool plain[2];      // queries with a sum that is no number
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = rows + g + 8 * e;
    const float inv = l[e] > 0.f ? 1.f / l[e] : 0.f;
    plain[e] = !(fabsf(l[e]) < INFINITY);
    float* dst = out + (long long)(t0 + q0 + r) * ((long long)n_heads * HD) + head * HD + t2;
#pragma unroll
    for (int c = 0; c < SETS; ++c) {
      if (part + c * SHARE >= HD / 16) continue;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 x = make_float2((o[c][i][2 * e] + o_small[c][i][2 * e]) * inv, (o[c][i][2 * e + 1] + o_small[c][i][2 * e + 1]) * inv);
        plain[e] |= !(fabsf(x.x) < INFINITY && fabsf(x.y) < INFINITY);
        if (r < nq) *reinterpret_cast<float2*>(dst + 16 * (part + c * SHARE) + 8 * i) = x;
      }
    }
    plain[e] &= r < nq;
  }
  const unsigned redo[2] = {__ballot_sync(0xffffffffu, plain[0]), __ballot_sync(0xffffffffu, plain[1])};
  if ((redo[0] | redo[1]) == 0) return;
  __syncwarp();
  for (int r = 0; r < 16; ++r) {
    if ((redo[r >> 3] >> (4 * (r & 7)) & 15u) == 0) continue;
    const int pos = warp_first + r;
    const long long row = t0 + q0 + rows + r;
    ap_plain<HD, SHARE>(q + row * q_row_stride + head * HD, kv, out + row * ((long long)n_heads * HD) + head * HD, seq, t0, kv_head, n_kv_heads,
                 scale, window > 0 ? max(0, pos - window + 1) : 0, causal ? min(pos, k_hi - 1) : k_hi - 1, part);
  }
}

// Which calls take this kernel.  (A sequence's results are the same bits in each call: what has AP_FEW new tokens or fewer is formed by
// the same multiply-adds here and there.)
inline bool attention_prefill_parts_takes(const void* q, long long q_row_stride, const KvView& kv, const void* out, int head_dim, int max_new) {
  return head_dim % 16 == 0 && head_dim <= 64 && q_row_stride % 4 == 0 && (kv.table != nullptr || kv.row_stride % 4 == 0) &&
         ((unsigned long long)q | (unsigned long long)kv.k | (unsigned long long)kv.v | (unsigned long long)out) % 16 == 0 && max_new > AP_FEW &&
         max_new <= 65535 * 16;
}

template <int HD, int BQ, int WARPS, int BLOCKS>
static int launch_parts(const float* q, long long q_row_stride, const KvView& kv, float* out, const int* seq_start, const int* past_len,
                        int n_seqs, int max_new, int n_heads, int n_kv_heads, float scale, int causal, int window, cudaStream_t stream) {
  constexpr size_t smem = 2 * 3 * (size_t)(BQ + 2 * AP_BK) * (HD + 8) + sizeof(float) * BQ * AP_SCORES;
  auto kern = attention_prefill_parts_kernel<HD, BQ, WARPS, BLOCKS>;
  static SharedMemoryAllowance allowed;
  BT_CHECK(allow_shared_memory(allowed, kern, smem), "attention_prefill_parts: cannot reserve %zu bytes of shared memory", smem);
  const dim3 grid(n_heads, n_seqs, (max_new + BQ - 1) / BQ);
  BT_PDL_OK("attention_prefill_parts", launch_pdl(kern, grid, dim3(WARPS * 32), smem, stream, 1, q, q_row_stride, kv, out, seq_start,
                                                  past_len, n_heads, n_kv_heads, scale, causal, window));
  return 0;
}

template <int HD, typename... Args>
static int launch_parts_queries(int queries, Args... args) {
  if (queries == 16) return launch_parts<HD, 16, 4, 3>(args...);
  if (queries == 32) return launch_parts<HD, 32, 4, 2>(args...);
  return launch_parts<HD, 64, 8, 2>(args...);
}

// Queries a block: 16 where no sequence has more or blocks of 32 leave multiprocessors without one, 64 where such blocks are three a
// multiprocessor, else 32.  A query's bits are the same in each.  Blocks of 16 / 32 / 64, us, 12 heads of 64: one prompt of 129 tokens 10.0 / 11.0 /
// 12.6; 24 behind 300 for 32 sequences 55 / 51 / 68; one of 2,048 251 / 194 / 226; 16 x 120 27 / 23 / 20; 16 heads, 4 x 1,000 331 / 252 / 214.
inline int launch_attention_prefill_parts(const float* q, long long q_row_stride, const KvView& kv, float* out, const int* seq_start,
                                          const int* past_len, int n_seqs, int max_new, int n_heads, int n_kv_heads, int head_dim,
                                          float scale, int causal, int window, cudaStream_t stream) {
  const int sms = sm_count();
  BT_CHECK(sms > 0, "attention_prefill_simt: cannot read the number of multiprocessors of the current device");
  const long long columns = (long long)n_seqs * n_heads;
  const int queries = max_new <= 16 || columns * ((max_new + 31) / 32) < sms      ? 16
                      : max_new <= 32 || columns * ((max_new + 63) / 64) < 3ll * sms ? 32
                                                                                     : 64;
#define BT_AP(HD)                                                                                                                       \
  if (head_dim == HD)                                                                                                                   \
  return launch_parts_queries<HD>(queries, q, q_row_stride, kv, out, seq_start, past_len, n_seqs, max_new, n_heads, n_kv_heads, scale, \
                                  causal, window, stream)
  BT_AP(16);
  BT_AP(32);
  BT_AP(48);
  BT_AP(64);
#undef BT_AP
  return fail("attention_prefill_simt: no kernel for heads of %d channels", head_dim);
}

}  // namespace bt
