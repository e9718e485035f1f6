// A selective state-space scan: per channel c and state index n a 32-bit state that every token decays and feeds,
//
//     dt[t, c] = softplus(sum_r W_dt[c, r] * low[t, r] + b_dt[c])                       (selective_scan_dt)
//     S[c, n] <- exp(dt[t, c] * A[c, n]) * S[c, n] + dt[t, c] * x[t, c] * B[t, n]       A = -exp(A_log)
//     y[t, c]  = (sum_n S[c, n] * C[t, n] + D[c] * x[t, c]) * z[t, c] * sigmoid(z[t, c]) * out_scale
//
// B and C are channels of the step's rows `low` (one vector per token, shared by all channels); x and z are channels
// of other rows.  Step sizes, decays, the state and all sums are 32-bit.  A channel belongs to LANES adjacent lanes,
// each with NS of the `n_state` indices in registers for all tokens of the step; their partial sums meet by shuffles.
// The tokens of a run are staged in shared memory TT at a time.  state: [slots][channels][n_state].
//
// A long run is cut into pieces of `piece` tokens that run side by side.  A first launch (ENDS) runs every piece but a
// sequence's last from a zero state and leaves, per channel, what it ends with, E[n], and the sum of its step sizes, d;
// the state after the piece is then exp(A[n] d) * (state before it) + E[n], since the recurrence is linear in the state
// and its decays multiply to exp(A[n] * sum dt).  The second launch gives every piece its own block, which first walks
// the earlier pieces' (E, d) from the state before the run to its own start and then runs its tokens as the single
// run would; the last piece writes the state back.  `ends`: [pieces of the step][channels][n_state + 1], where the
// pieces of sequence s begin at first_row(s) / piece + s.  Nothing orders the second launch's blocks, so none of them may
// read what another one writes: the first launch copies the stored state into the cell of the sequence's last piece (which
// leaves no ends), and all pieces start from that copy.
#include "chunk_mma.cuh"
#include "common.cuh"

namespace bt {

constexpr int SS_TT = 16;        // tokens staged at a time
constexpr int SS_THREADS = 128;
constexpr int SS_WS = 257;       // floats between the rank indices of the step sizes' weights in shared memory

__device__ __forceinline__ float ss_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// exp(d * a) for the decay of a step, a <= 0.  With bfloat16 rows the exponent is formed in base 2 (a_scaled = a log2 e)
// and raised by the special-function unit (2 units in the last place); 32-bit rows take the library's exp.
template <typename T>
__device__ __forceinline__ float ss_decay(float d, float a_scaled) {
  if constexpr (sizeof(T) == 2) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(d * a_scaled));
    return y;
  } else {
    return expf(d * a_scaled);
  }
}

__device__ __forceinline__ unsigned long long ss_pack(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void ss_unpack(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long ss_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long ss_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// dt[t, c], a block: 256 channels x SS_TT tokens; W_dt's rows of these channels lie transposed in shared memory
template <typename T>
__global__ void __launch_bounds__(256)
selective_scan_dt_kernel(const T* __restrict__ low, long long low_row_stride, const float* __restrict__ w_dt,
                         const float* __restrict__ b_dt, float* __restrict__ dt, long long n_tokens, int channels,
                         int rank) {
  extern __shared__ float sm[];
  float* low_s = sm;                       // [rank][SS_TT]
  float* w_s = low_s + rank * SS_TT;       // [rank][SS_WS]: padded, so that the transposing stores spread over the banks
  pdl_trigger();
  const int c0 = blockIdx.x * 256, c = c0 + threadIdx.x;
  for (int i = threadIdx.x; i < rank * 256; i += 256) {
    const int cl = i / rank, r = i - cl * rank;
    w_s[r * SS_WS + cl] = c0 + cl < channels ? w_dt[(long long)(c0 + cl) * rank + r] : 0.f;
  }
  const float bias = c < channels ? b_dt[c] : 0.f;
  pdl_wait();
  for (long long t0 = (long long)blockIdx.y * SS_TT; t0 < n_tokens; t0 += (long long)gridDim.y * SS_TT) {
    const int nt = (int)min((long long)SS_TT, n_tokens - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < SS_TT * rank; i += 256) {
      const int t = i / rank, r = i - t * rank;
      low_s[r * SS_TT + t] = t < nt ? to_float(low[(t0 + t) * low_row_stride + r]) : 0.f;
    }
    __syncthreads();
    // a thread a channel: its weight once per rank index against the SS_TT tokens' numbers, read four at a time
    float acc[SS_TT];
#pragma unroll
    for (int t = 0; t < SS_TT; ++t) acc[t] = bias;
    for (int r = 0; r < rank; ++r) {
      const float w = w_s[r * SS_WS + threadIdx.x];
#pragma unroll
      for (int t4 = 0; t4 < SS_TT / 4; ++t4) {
        const float4 x = *reinterpret_cast<const float4*>(low_s + r * SS_TT + t4 * 4);
        acc[t4 * 4 + 0] = fmaf(w, x.x, acc[t4 * 4 + 0]);
        acc[t4 * 4 + 1] = fmaf(w, x.y, acc[t4 * 4 + 1]);
        acc[t4 * 4 + 2] = fmaf(w, x.z, acc[t4 * 4 + 2]);
        acc[t4 * 4 + 3] = fmaf(w, x.w, acc[t4 * 4 + 3]);
      }
    }
    if (c < channels) {
#pragma unroll
      for (int t = 0; t < SS_TT; ++t)
        if (t < nt) dt[(t0 + t) * channels + c] = ss_softplus(acc[t]);
    }
  }
}

// The same for bfloat16 rows and a rank of at most 64, on tensor cores: W_dt's 32-bit numbers go in as three bfloat16 parts, which
// hold all of their bits (chunk_mma.cuh; the first parts' sums begin from zero every 16 of the rank).  Errors against 64 bits, above and
// here, rank 48: 1.3e-7 and 1.9e-8 with normal numbers, 1.8e-7 and 1.2e-7 beside one large channel (3.2e-7 in one accumulator).  A warp keeps 32 channels' weights in registers as the operand wants them and walks over tiles of 16 tokens, with
// neither shared memory nor barriers; the softplus, about 45 instructions a number, is what is left.  The kernel above is bound by
// instructions, a third of them for its weights' way through shared memory.  In us, above and here: 2,439 tokens of 1,536 channels
// and rank 48 27.8 and 18.2, 2,048 of 1,024 and rank 16 12.5 and 9.6, 100 of 1,536 and rank 48 6.9 and 3.9.
template <int KS>
__global__ void __launch_bounds__(128, KS <= 2 ? 5 : KS == 3 ? 4 : 3)
selective_scan_dt_mma_kernel(const __nv_bfloat16* __restrict__ low, long long low_row_stride, const float* __restrict__ w_dt,
                             const float* __restrict__ b_dt, float* __restrict__ dt, int n_tokens, int channels, int rank,
                             int groups, int walkers) {
  pdl_trigger();
  const int warp = (int)(blockIdx.x * 4 + (threadIdx.x >> 5)), lane = threadIdx.x & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  const int group = warp % groups, walker = warp / groups;
  if (walker >= walkers) return;
  const int c0 = group * 32;
  unsigned w[3][KS][4][2];
#pragma unroll
  for (int k = 0; k < KS; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + 8 * j + g, r = 16 * k + 8 * h + t2;
        float2 v = c < channels && r < rank ? *reinterpret_cast<const float2*>(w_dt + (long long)c * rank + r) : make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const __nv_bfloat162 part = __floats2bfloat162_rn(v.x, v.y);
          const float2 back = __bfloat1622float2(part);
          w[q][k][j][h] = *reinterpret_cast<const unsigned*>(&part);
          v.x -= back.x;
          v.y -= back.y;
        }
      }
  float2 bias[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = c0 + 8 * j + t2;
    bias[j] = make_float2(c < channels ? b_dt[c] : 0.f, c + 1 < channels ? b_dt[c + 1] : 0.f);
  }
  const bool pairs = channels % 2 == 0 && (unsigned long long)dt % 8 == 0;
  pdl_wait();
  for (int t0 = walker * 16; t0 < n_tokens; t0 += walkers * 16) {
    unsigned a[KS][4];
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = t0 + g + 8 * (i & 1), r = 16 * k + 8 * (i >> 1) + t2;
        a[k][i] = t < n_tokens && r < rank ? *reinterpret_cast<const unsigned*>(low + t * low_row_stride + r) : 0u;
      }
    float acc[4][4] = {}, small[4][4] = {};
#pragma unroll
    for (int q = 2; q > 0; --q)
#pragma unroll
      for (int k = 0; k < KS; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) cm_mma(small[j], a[k], w[q][k][j][0], w[q][k][j][1]);
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x[4];
        cm_mma_zero(x, a[k], w[0][k][j][0], w[0][k][j][1]);
        cm_add(acc[j], x);
      }
    bool whole = true;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[j][i] = acc[j][i] + small[j][i] + (i & 1 ? bias[j].y : bias[j].x);
        whole = whole && isfinite(acc[j][i]);
      }
    if (!whole) {      // an infinity times the parts of a weight is no number: such sums are formed again by multiply-adds
#pragma unroll 1
      for (int n = 0; n < 16; ++n) {
        const int t = t0 + g + 8 * (n >> 1 & 1), c = c0 + 8 * (n >> 2) + t2 + (n & 1);
        if (t >= n_tokens || c >= channels) continue;
        float z = b_dt[c];
        for (int r = 0; r < rank; ++r) z = fmaf(w_dt[(long long)c * rank + r], to_float(low[t * low_row_stride + r]), z);
#pragma unroll
        for (int m = 0; m < 16; ++m)
          if (m == n && !isfinite(acc[m >> 2][m & 3])) acc[m >> 2][m & 3] = z;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = t0 + g + 8 * h, c = c0 + 8 * j + t2;
        const float y0 = ss_softplus(acc[j][2 * h]), y1 = ss_softplus(acc[j][2 * h + 1]);
        float* at = dt + (long long)t * channels + c;
        if (t >= n_tokens) continue;
        if (pairs) {
          if (c < channels) *reinterpret_cast<float2*>(at) = make_float2(y0, y1);
        } else {
          if (c < channels) at[0] = y0;
          if (c + 1 < channels) at[1] = y1;
        }
      }
  }
}

template <typename T, int NS, int LANES, bool ENDS>
__global__ void __launch_bounds__(SS_THREADS)
selective_scan_kernel(const T* __restrict__ x, long long x_row_stride, const T* __restrict__ z, long long z_row_stride,
                      const float* __restrict__ dt, const T* __restrict__ low, long long low_row_stride, int b_off,
                      int c_off, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                      float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ seq_start,
                      T* __restrict__ out, long long out_row_stride, int channels, int n_state, float out_scale, int piece,
                      float* __restrict__ ends, int stage) {
  constexpr int CPB = SS_THREADS / LANES;      // channels per block
  extern __shared__ float sm[];
  float* bc_s = sm;                            // [stage][2 * n_state]
  float* dt_s = bc_s + stage * 2 * n_state;    // [stage][CPB]
  float* x_s = dt_s + stage * CPB;
  float* z_s = x_s + stage * CPB;
  pdl_trigger();
  const int seq = blockIdx.y, c_local = threadIdx.x / LANES, part = threadIdx.x % LANES;
  const int c = blockIdx.x * CPB + c_local;
  const bool owns = c < channels;
  const int n0 = part * NS;
  float a[NS], s[NS];      // a: A = -exp(A_log), times log2 e where the decays are raised in base 2
#pragma unroll
  for (int i = 0; i < NS; ++i)
    a[i] = owns && n0 + i < n_state ? -expf(a_log[(long long)c * n_state + n0 + i]) * (sizeof(T) == 2 ? 1.4426950408889634f : 1.f)
                                    : 0.f;
  const float skip = owns ? d_skip[c] : 0.f;
  pdl_wait();
  const int first = seq_start[seq], n_all = seq_start[seq + 1] - first;
  // this block's piece of the run: tokens [t_lo, t_hi); the whole run when piece == 0
  const int n_pieces = piece > 0 ? (n_all + piece - 1) / piece : 1;
  const int my_piece = piece > 0 ? (int)blockIdx.z : 0;
  if (my_piece >= n_pieces - (ENDS ? 1 : 0)) return;
  const int t_lo = my_piece * piece, t_hi = piece > 0 ? min(n_all, t_lo + piece) : n_all;
  const bool last_piece = my_piece == n_pieces - 1;
  const long long es = (long long)channels * (n_state + 1);
  float* e_base = piece > 0 ? ends + ((long long)(first / piece + seq)) * es + (long long)(owns ? c : 0) * (n_state + 1) : nullptr;
  float* s_base = state + ((long long)slots[seq] * channels + (owns ? c : 0)) * n_state;
  float dt_sum = 0.f;
  // the state before the run: where it is stored if this block alone reads and writes it, else its copy
  float* before = n_pieces > 1 ? e_base + (long long)(n_pieces - 1) * es : s_base;
  if (ENDS && owns && my_piece == 0) {
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (n0 + i < n_state) before[n0 + i] = s_base[n0 + i];
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) s[i] = !ENDS && owns && n0 + i < n_state ? before[n0 + i] : 0.f;
  if (!ENDS && owns) {
#pragma unroll 4
    for (int j = 0; j < my_piece; ++j) {      // (several pieces' numbers are asked for at once)
      const float* e = e_base + (long long)j * es;
      const float d = e[n_state];
#pragma unroll
      for (int i = 0; i < NS; ++i)
        if (n0 + i < n_state) s[i] = fmaf(ss_decay<T>(d, a[i]), s[i], e[n0 + i]);
    }
  }
  // B and C of a token as 16-byte pieces where the lane's state indices are whole pieces of a row
  const bool vec = (n_state & 3) == 0 && n0 + NS <= n_state;
  for (int t0 = t_lo; t0 < t_hi; t0 += stage) {
    const int nt = min(stage, t_hi - t0);
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < nt * 2 * n_state; i += SS_THREADS) {
      const int t = i / (2 * n_state), n = i - t * 2 * n_state;
      const T* row = low + (long long)(first + t0 + t) * low_row_stride;
      bc_s[i] = to_float(n < n_state ? row[b_off + n] : row[c_off + n - n_state]);
    }
    // (the gates are formed here, by every thread: in the tokens' loop one lane of a channel would, the others waiting)
#pragma unroll 4
    for (int i = threadIdx.x; i < nt * CPB; i += SS_THREADS) {
      const int t = i / CPB, cl = i - t * CPB, cc = blockIdx.x * CPB + cl;
      const long long r = first + t0 + t;
      const bool in = cc < channels;
      dt_s[i] = in ? dt[r * channels + cc] : 0.f;
      x_s[i] = in ? to_float(x[r * x_row_stride + cc]) : 0.f;
      if (!ENDS) {
        const float zv = in ? to_float(z[r * z_row_stride + cc]) : 0.f;
        z_s[i] = zv / (1.f + expf(-zv));
      }
    }
    __syncthreads();
    // (a token waits for the one before only in the state's multiply-add: four are worked on at once.  2,440 tokens of 1,536
    // channels x 16 indices in a recorded layer: the second launch 93 us with a token at a time and the gates in this loop, 76
    // so; what is left is the chain of 64 tokens a block and the shared-memory reads of B and C)
#pragma unroll 4
    for (int t = 0; t < nt; ++t) {
      const float d = dt_s[t * CPB + c_local], xv = x_s[t * CPB + c_local];
      const float dx = d * xv;
      const float* bt_ = bc_s + t * 2 * n_state + n0;
      const float* ct_ = bt_ + n_state;
      float y = 0.f;
      if (vec) {
#pragma unroll
        for (int i4 = 0; i4 < NS / 4; ++i4) {
          const float4 b4 = *reinterpret_cast<const float4*>(bt_ + 4 * i4), c4 = *reinterpret_cast<const float4*>(ct_ + 4 * i4);
          const float bs[4] = {b4.x, b4.y, b4.z, b4.w}, cs[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int i = 4 * i4 + k;
            s[i] = fmaf(ss_decay<T>(d, a[i]), s[i], dx * bs[k]);
            y = fmaf(s[i], cs[k], y);
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          if (n0 + i < n_state) {
            s[i] = fmaf(ss_decay<T>(d, a[i]), s[i], dx * bt_[i]);
            y = fmaf(s[i], ct_[i], y);
          }
        }
      }
      if (!ENDS) {
        __syncwarp();
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      }
      dt_sum += d;
      if (ENDS) continue;
      // (the token's x has been read by all lanes of its channel, which met in the shuffles)
      if (part == 0) x_s[t * CPB + c_local] = (y + skip * xv) * z_s[t * CPB + c_local] * out_scale;
    }
    if (ENDS) continue;
    __syncthreads();
    for (int i = threadIdx.x; i < nt * CPB; i += SS_THREADS) {
      const int t = i / CPB, cl = i - t * CPB, cc = blockIdx.x * CPB + cl;
      if (cc < channels) out[(long long)(first + t0 + t) * out_row_stride + cc] = from_float<T>(x_s[i]);
    }
  }
  if (ENDS) {
    if (owns) {
      float* e = e_base + (long long)my_piece * es;
#pragma unroll
      for (int i = 0; i < NS; ++i)
        if (n0 + i < n_state) e[n0 + i] = s[i];
      if (part == 0) e[n_state] = dt_sum;
    }
    return;
  }
  if (owns && last_piece) {
#pragma unroll
    for (int i = 0; i < NS; ++i)
      if (n0 + i < n_state) s_base[n0 + i] = s[i];
  }
}

// The pieces of long runs for up to 16 state indices: a channel belongs to one thread, or two neighbours above 8 indices, with 8
// indices each, whose numbers go two an instruction; a token's B and C are read once a warp, and four tokens are worked on at once
// without a branch between them.  What bounds it: the special-function unit's exponentials, one an index and token, take 14 us a
// launch at 2,439 tokens of 1,536 channels x 16 indices (its pipe is busy 50 and 32 % of the two launches), the instructions about 11 (the first launch) and 20; the rest is the
// latency of a warp's chain.  Both launches there, in us, with selective_scan_kernel and so: 90 and 70; 2 x 1,024 tokens of 1,024
// channels 63 and 51; one run of 300 32 and 31; 8 indices 114 and 51; 32-bit rows 121 and 98.  (A thread for all 16 indices: 84,
// too few warps to hide an exponential behind.  72 registers a thread, so that 2,439 tokens are one wave of blocks: 68, but 2 x 70
// tokens 37 instead of 24.)
// A piece's tokens are asked for SP_AHEAD at a time, one group ahead.  The walk over the earlier pieces goes through the cells as
// they lie, n_state + 1 numbers a channel in a row over the block's threads, and meets the channels' layout in shared memory.
constexpr int SP_THREADS = 64, SP_STAGE = 64, SP_AHEAD = 4;

// FULL: every thread's 8 indices are a channel's; else those past n_state stay zero (a zero times an infinite step would not).
template <typename T, int LANES, bool ENDS, bool FULL>
__global__ void __launch_bounds__(SP_THREADS, ENDS ? 12 : 10)
selective_scan_piece_kernel(const T* __restrict__ x, long long x_row_stride, const T* __restrict__ z, long long z_row_stride,
                            const float* __restrict__ dt, const T* __restrict__ low, long long low_row_stride, int b_off,
                            int c_off, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                            float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ seq_start,
                            T* __restrict__ out, long long out_row_stride, int channels, int n_state, float out_scale,
                            int piece, float* __restrict__ ends) {
  constexpr float kLog2e = sizeof(T) == 2 ? 1.4426950408889634f : 1.f;      // (see ss_decay)
  constexpr int NS = 8, PAD = NS * LANES;                                   // indices a thread, and a channel, has room for
  constexpr int ROW = ENDS ? PAD : 2 * PAD;                                 // a token's B, and C where it is read
  constexpr int CPB = SP_THREADS / LANES, CELLS = (CPB * (PAD + 1) + SP_THREADS - 1) / SP_THREADS;
  __shared__ __align__(16) float bc_s[SP_STAGE * ROW];
  __shared__ float walk_s[ENDS ? 1 : CPB * (PAD + 1)];
  pdl_trigger();
  const int tid = threadIdx.x, seq = blockIdx.y, cl = tid / LANES, n0 = tid % LANES * NS, c0 = blockIdx.x * CPB, c = c0 + cl;
  const bool owns = c < channels;
  float a[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) a[i] = owns && n0 + i < n_state ? -expf(a_log[(long long)c * n_state + n0 + i]) * kLog2e : 0.f;
#pragma unroll
  for (int i = 0; i < NS; ++i)
    if (a[i] == -INFINITY) a[i] = -3.4e38f;      // (times a step of zero must be a number, see fetch below)
  const float skip = !ENDS && owns ? d_skip[c] : 0.f;
  pdl_wait();
  const int first = seq_start[seq], n_all = seq_start[seq + 1] - first;
  const int n_pieces = (n_all + piece - 1) / piece, my_piece = blockIdx.z;
  if (my_piece >= n_pieces - (ENDS ? 1 : 0)) return;
  const int t_lo = my_piece * piece, t_hi = min(n_all, t_lo + piece);
  const int n1 = n_state + 1;
  const long long es = (long long)channels * n1;
  float* e_block = ends + ((long long)(first / piece + seq)) * es + (long long)c0 * n1;
  float* s_block = state + ((long long)slots[seq] * channels + c0) * n_state;
  float s[NS];
  if (ENDS) {
    if (my_piece == 0 && owns) {
      float* copy = e_block + (long long)(n_pieces - 1) * es + cl * n1;
#pragma unroll
      for (int i = 0; i < NS; ++i)
        if (n0 + i < n_state) copy[n0 + i] = s_block[cl * n_state + n0 + i];
    }
#pragma unroll
    for (int i = 0; i < NS; ++i) s[i] = 0.f;
  } else if (my_piece == 0) {
    const float* before = n_pieces > 1 ? e_block + (long long)(n_pieces - 1) * es + cl * n1 : s_block + cl * n_state;
#pragma unroll
    for (int i = 0; i < NS; ++i) s[i] = owns && n0 + i < n_state ? before[n0 + i] : 0.f;
  } else {
    // number k of this thread is number `tid + 64 k` of the block's cells: channel ch, index n (index n_state: the sum of dt)
    float w[CELLS], wa[CELLS];
    int at_d[CELLS];
    const float* copy = e_block + (long long)(n_pieces - 1) * es;
    const int step_c = SP_THREADS / n1, step_n = SP_THREADS % n1;
    int ch = tid / n1, n = tid % n1;
#pragma unroll
    for (int k = 0; k < CELLS; ++k) {
      const bool mine = ch < CPB && c0 + ch < channels && n < n_state;
      w[k] = mine ? copy[tid + SP_THREADS * k] : 0.f;
      wa[k] = mine ? -expf(a_log[(long long)(c0 + ch) * n_state + n]) * kLog2e : 0.f;
      at_d[k] = mine ? ch * n1 + n_state : -1;
      ch += step_c; n += step_n;
      if (n >= n1) { n -= n1; ++ch; }
    }
#pragma unroll 2
    for (int j = 0; j < my_piece; ++j) {      // (two pieces' numbers are asked for at once)
      const float* e = e_block + (long long)j * es;
      float ev[CELLS], dv[CELLS];
#pragma unroll
      for (int k = 0; k < CELLS; ++k) {
        ev[k] = at_d[k] >= 0 ? e[tid + SP_THREADS * k] : 0.f;
        dv[k] = at_d[k] >= 0 ? e[at_d[k]] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < CELLS; ++k) w[k] = fmaf(ss_decay<T>(dv[k], wa[k]), w[k], ev[k]);
    }
#pragma unroll
    for (int k = 0; k < CELLS; ++k)
      if (at_d[k] >= 0) walk_s[tid + SP_THREADS * k] = w[k];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NS; ++i) s[i] = owns && n0 + i < n_state ? walk_s[cl * n1 + n0 + i] : 0.f;
  }
  unsigned long long s2[NS / 2], a2[NS / 2];
#pragma unroll
  for (int i = 0; i < NS / 2; ++i) {
    s2[i] = ss_pack(s[2 * i], s[2 * i + 1]);
    a2[i] = ss_pack(a[2 * i], a[2 * i + 1]);
  }
  const long long cc = owns ? c : 0;      // (a thread past the channels reads the first one's numbers and writes nothing)
  float dt_sum = 0.f;
  for (int t0 = t_lo; t0 < t_hi; t0 += SP_STAGE) {
    const int nt = min(SP_STAGE, t_hi - t0);
    const long long row0 = first + t0;
    const float* dt_at = dt + row0 * channels + cc;
    const T* x_at = x + row0 * x_row_stride + cc;
    const T* z_at = z + row0 * z_row_stride + cc;
    T* out_at = out + row0 * out_row_stride + cc;
    float d[SP_AHEAD];
    T xv[SP_AHEAD], zv[SP_AHEAD];
    // the next SP_AHEAD tokens' numbers; a token past the piece has a step of zero, which leaves the state as it is
    auto fetch = [&](int left, float (&dd)[SP_AHEAD], T (&xx)[SP_AHEAD], T (&zz)[SP_AHEAD]) {
      if (left >= SP_AHEAD) {
#pragma unroll
        for (int u = 0; u < SP_AHEAD; ++u) {
          dd[u] = dt_at[u * channels];
          xx[u] = x_at[u * x_row_stride];
          if (!ENDS) zz[u] = z_at[u * z_row_stride];
        }
      } else {
#pragma unroll
        for (int u = 0; u < SP_AHEAD; ++u) {
          const bool in = u < left;
          dd[u] = in ? dt_at[u * channels] : 0.f;
          xx[u] = in ? x_at[u * x_row_stride] : from_float<T>(0.f);
          if (!ENDS) zz[u] = in ? z_at[u * z_row_stride] : from_float<T>(0.f);
        }
      }
      dt_at += (long long)SP_AHEAD * channels;
      x_at += SP_AHEAD * x_row_stride;
      if (!ENDS) z_at += SP_AHEAD * z_row_stride;
    };
    fetch(nt, d, xv, zv);
    __syncthreads();
#pragma unroll 8
    for (int i = tid; i < SP_STAGE * ROW; i += SP_THREADS) {      // (zeros past the piece: a number there times zero is no number)
      const int t = i / ROW, m = i % ROW, n = m % PAD;
      bc_s[i] = t < nt && n < n_state ? to_float(low[(row0 + t) * low_row_stride + (m < PAD ? b_off : c_off) + n]) : 0.f;
    }
    __syncthreads();
    for (int t = 0; t < nt; t += SP_AHEAD) {
      float dn[SP_AHEAD];
      T xn[SP_AHEAD], zn[SP_AHEAD];
      fetch(nt - t - SP_AHEAD, dn, xn, zn);
      float y[SP_AHEAD];
#pragma unroll
      for (int u = 0; u < SP_AHEAD; ++u) {
        const float dx = d[u] * to_float(xv[u]);
        const unsigned long long d2 = ss_pack(d[u], d[u]), dx2 = ss_pack(dx, dx);
        const ulonglong2* b2 = reinterpret_cast<const ulonglong2*>(bc_s + (t + u) * ROW + n0);
        unsigned long long y2[2] = {0ull, 0ull};
#pragma unroll
        for (int i4 = 0; i4 < NS / 4; ++i4) {
          const ulonglong2 b = b2[i4];
          ulonglong2 cv;
          if (!ENDS) cv = b2[PAD / 4 + i4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = 2 * i4 + h;
            float e0, e1;
            ss_unpack(ss_mul2(d2, a2[i]), e0, e1);
            if constexpr (sizeof(T) == 2) {
              asm("ex2.approx.ftz.f32 %0, %0;\n" : "+f"(e0));
              asm("ex2.approx.ftz.f32 %0, %0;\n" : "+f"(e1));
            } else {
              e0 = expf(e0);
              e1 = expf(e1);
            }
            s2[i] = ss_fma2(ss_pack(e0, e1), s2[i], ss_mul2(dx2, h ? b.y : b.x));
            if (!FULL) {
              float lo, hi;
              ss_unpack(s2[i], lo, hi);
              s2[i] = ss_pack(n0 + 2 * i < n_state ? lo : 0.f, n0 + 2 * i + 1 < n_state ? hi : 0.f);
            }
            if (!ENDS) y2[h] = ss_fma2(s2[i], h ? cv.y : cv.x, y2[h]);
          }
        }
        if (ENDS) {
          dt_sum += d[u];
        } else {
          float y0, y1, y3, y4;
          ss_unpack(y2[0], y0, y1);
          ss_unpack(y2[1], y3, y4);
          y[u] = (y0 + y1) + (y3 + y4);
          if (LANES > 1) y[u] += __shfl_xor_sync(0xffffffffu, y[u], 1);
        }
      }
      if (!ENDS) {
#pragma unroll
        for (int v = 0; v < SP_AHEAD / LANES; ++v) {      // (a channel's lanes take the tokens' gates in turn)
          const int u = v * LANES + (LANES > 1 ? tid % LANES : 0);
          const float yu = LANES == 1 ? y[v] : (tid % LANES ? y[v * LANES + LANES - 1] : y[v * LANES]);
          const float xf = to_float(LANES == 1 ? xv[v] : (tid % LANES ? xv[v * LANES + LANES - 1] : xv[v * LANES]));
          const float zf = to_float(LANES == 1 ? zv[v] : (tid % LANES ? zv[v * LANES + LANES - 1] : zv[v * LANES]));
          const float gate = zf / (1.f + expf(-zf));
          if (owns && t + u < nt) out_at[u * out_row_stride] = from_float<T>((yu + skip * xf) * gate * out_scale);
        }
        out_at += SP_AHEAD * out_row_stride;
      }
#pragma unroll
      for (int u = 0; u < SP_AHEAD; ++u) {
        d[u] = dn[u];
        xv[u] = xn[u];
        if (!ENDS) zv[u] = zn[u];
      }
    }
  }
  if (!owns || (!ENDS && my_piece != n_pieces - 1)) return;
  float* dst = ENDS ? e_block + (long long)my_piece * es + cl * n1 + n0 : s_block + cl * n_state + n0;
#pragma unroll
  for (int i = 0; i < NS / 2; ++i) {
    float lo, hi;
    ss_unpack(s2[i], lo, hi);
    if (n0 + 2 * i < n_state) dst[2 * i] = lo;
    if (n0 + 2 * i + 1 < n_state) dst[2 * i + 1] = hi;
  }
  if (ENDS && n0 == 0) dst[n_state] = dt_sum;
}

template <typename T>
static int launch_selective_scan(const T* x, long long xs, const T* z, long long zs, const float* dt, const T* low,
                                 long long ls, int b_off, int c_off, const float* a_log, const float* d_skip, float* state,
                                 const int* slots, const int* seq_start, T* out, long long os, int n_seqs, int channels,
                                 int n_state, float out_scale, int piece, int max_pieces, float* ends,
                                 cudaStream_t stream) {
  int ns, lanes;
  if (n_state <= 16) { ns = 4; lanes = 4; }
  else if (n_state <= 32) { ns = 8; lanes = 4; }
  else if (n_state <= 64) { ns = 16; lanes = 4; }
  else if (n_state <= 128) { ns = 16; lanes = 8; }
  else if (n_state <= 256) { ns = 16; lanes = 16; }
  else { ns = 16; lanes = 32; }
  BT_CHECK(n_state <= 512, "selective_scan: %d state indices a channel; the kernel takes up to 512", n_state);
  if (piece > 0 && n_state <= 16) {      // (steps without pieces are few tokens a sequence: more lanes a channel answer sooner)
#define BT_SP(LANES, ENDS, FULL)                                                                                             \
  BT_PDL_OK("selective_scan", launch_pdl(selective_scan_piece_kernel<T, LANES, ENDS, FULL>,                                  \
                                         dim3((channels + SP_THREADS / LANES - 1) / (SP_THREADS / LANES), n_seqs, max_pieces), \
                                         dim3(SP_THREADS), 0, stream, 1, x, xs, z, zs, dt, low, ls, b_off, c_off, a_log,     \
                                         d_skip, state, slots, seq_start, out, os, channels, n_state, out_scale, piece, ends))
    if (n_state == 8) { BT_SP(1, true, true); BT_SP(1, false, true); }
    else if (n_state < 8) { BT_SP(1, true, false); BT_SP(1, false, false); }
    else if (n_state == 16) { BT_SP(2, true, true); BT_SP(2, false, true); }
    else { BT_SP(2, true, false); BT_SP(2, false, false); }
#undef BT_SP
    return 0;
  }
  const int cpb = SS_THREADS / lanes;
  const dim3 grid((channels + cpb - 1) / cpb, n_seqs, piece > 0 ? max_pieces : 1);
  const int stage = n_state <= 64 ? 2 * SS_TT : SS_TT;      // tokens staged in shared memory at a time
  const size_t smem = sizeof(float) * ((size_t)stage * 2 * n_state + 3 * (size_t)stage * cpb);
#define BT_SS(NS, LANES)                                                                                              \
  do {                                                                                                                \
    if (smem > 48 * 1024)                                                                                             \
      BT_CHECK(cudaFuncSetAttribute(selective_scan_kernel<T, NS, LANES, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                    (int)smem) == cudaSuccess &&                                                      \
               cudaFuncSetAttribute(selective_scan_kernel<T, NS, LANES, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                    (int)smem) == cudaSuccess, "selective_scan: cannot reserve %zu bytes of shared memory", smem); \
    if (piece > 0)                                                                                                    \
      BT_PDL_OK("selective_scan", launch_pdl(selective_scan_kernel<T, NS, LANES, true>, grid, dim3(SS_THREADS), smem, \
                                             stream, 1, x, xs, z, zs, dt, low, ls, b_off, c_off, a_log, d_skip, state, \
                                             slots, seq_start, out, os, channels, n_state, out_scale, piece, ends,     \
                                             stage));                                                                 \
    BT_PDL_OK("selective_scan", launch_pdl(selective_scan_kernel<T, NS, LANES, false>, grid, dim3(SS_THREADS), smem,   \
                                           stream, 1, x, xs, z, zs, dt, low, ls, b_off, c_off, a_log, d_skip, state,   \
                                           slots, seq_start, out, os, channels, n_state, out_scale, piece, ends,       \
                                           stage));                                                                   \
  } while (0)
  if (ns == 4)      // (its pieces went the other way)
    BT_PDL_OK("selective_scan", launch_pdl(selective_scan_kernel<T, 4, 4, false>, grid, dim3(SS_THREADS), smem, stream, 1, x, xs, z,
                                           zs, dt, low, ls, b_off, c_off, a_log, d_skip, state, slots, seq_start, out, os,
                                           channels, n_state, out_scale, piece, ends, stage));
  else if (ns == 8) BT_SS(8, 4);
  else if (lanes == 4) BT_SS(16, 4);
  else if (lanes == 8) BT_SS(16, 8);
  else if (lanes == 16) BT_SS(16, 16);
  else BT_SS(16, 32);
#undef BT_SS
  return 0;
}

}  // namespace bt

// dt [tokens, channels] 32-bit from the first `rank` channels of the rows of low
extern "C" int bt_selective_scan_dt(const void* low, long long low_row_stride, const float* w_dt, const float* b_dt,
                                    float* dt, long long n_tokens, int channels, int rank, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(channels > 0 && rank > 0 && rank <= 160 && n_tokens >= 0,
           "selective_scan_dt: bad sizes channels=%d rank=%d (at most 160)", channels, rank);
  if (n_tokens == 0) return 0;
  if (dtype == kBF16 && rank % 2 == 0 && rank <= 64 && n_tokens <= 0x7ffffff0ll && low_row_stride % 2 == 0 &&
      (unsigned long long)low % 4 == 0 && (unsigned long long)w_dt % 8 == 0) {
    // (one wave of blocks: 12 warps a multiprocessor and more are resident, with as many tiles of tokens each as that leaves)
    const int sms = sm_count();
    BT_CHECK(sms > 0, "selective_scan_dt: cannot read the number of multiprocessors of the current device");
    const int groups = (channels + 31) / 32, tiles = (int)((n_tokens + 15) / 16);
    const int most = 12 * sms / groups > 0 ? 12 * sms / groups : 1, walkers = tiles < most ? tiles : (tiles + (tiles + most - 1) / most - 1) / ((tiles + most - 1) / most);
    const dim3 grid((unsigned)(((long long)groups * walkers + 3) / 4));
#define BT_SSM(KS)                                                                                                    \
  BT_PDL_OK("selective_scan_dt", launch_pdl(selective_scan_dt_mma_kernel<KS>, grid, dim3(128), 0, stream, 1,          \
                                            (const __nv_bfloat16*)low, low_row_stride, w_dt, b_dt, dt, (int)n_tokens, \
                                            channels, rank, groups, walkers))
    if (rank <= 16) BT_SSM(1);
    else if (rank <= 32) BT_SSM(2);
    else if (rank <= 48) BT_SSM(3);
    else BT_SSM(4);
#undef BT_SSM
    return 0;
  }
  const size_t smem = sizeof(float) * ((size_t)rank * SS_WS + (size_t)SS_TT * rank);
  const long long tiles = (n_tokens + SS_TT - 1) / SS_TT;
  const long long col_blocks = (channels + 255) / 256, want_rows = (4 * 148 + col_blocks - 1) / col_blocks;
  const dim3 grid((unsigned)col_blocks, (unsigned)(tiles < want_rows ? tiles : want_rows));      // (about four blocks an SM)
#define BT_SSD(T)                                                                                                     \
  do {                                                                                                                \
    auto kern = selective_scan_dt_kernel<T>;                                                                          \
    if (smem > 48 * 1024)                                                                                             \
      BT_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess,     \
               "selective_scan_dt: cannot reserve %zu bytes of shared memory", smem);                                 \
    BT_PDL_OK("selective_scan_dt", launch_pdl(kern, grid, dim3(256), smem, stream, 1, (const T*)low, low_row_stride, w_dt, \
                                              b_dt, dt, n_tokens, channels, rank));                                    \
  } while (0)
  if (dtype == kF32) BT_SSD(float);
  else if (dtype == kBF16) BT_SSD(__nv_bfloat16);
  else return fail("selective_scan_dt: unknown dtype %d", dtype);
#undef BT_SSD
  return 0;
}

// x, z, out: first channel of [tokens, channels] views; low: the rows that hold B at b_off and C at c_off.
// piece > 0: runs are cut into pieces of `piece` tokens (a multiple of 16), none has more than max_pieces, and `ends`
// holds (n_tokens / piece + n_seqs + 1) * channels * (n_state + 1) floats; piece == 0: a block walks a whole run.
extern "C" int bt_selective_scan(const void* x, long long x_row_stride, const void* z, long long z_row_stride,
                                 const float* dt, const void* low, long long low_row_stride, int b_off, int c_off,
                                 const float* a_log, const float* d_skip, float* state, const int* slots,
                                 const int* seq_start, void* out, long long out_row_stride, int n_seqs, int channels,
                                 int n_state, float out_scale, int piece, int max_pieces, float* ends, int dtype,
                                 cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(piece == 0 || (piece % SS_TT == 0 && max_pieces > 0 && max_pieces <= 65535 && ends != nullptr),
           "selective_scan: pieces of %d tokens (a multiple of %d), at most %d a run, need scratch", piece, SS_TT, max_pieces);
  BT_CHECK(channels > 0 && n_state > 0 && n_seqs >= 0 && n_seqs <= 65535, "selective_scan: bad sizes seqs=%d channels=%d "
           "state=%d", n_seqs, channels, n_state);
  if (n_seqs == 0) return 0;
  if (dtype == kF32)
    return launch_selective_scan((const float*)x, x_row_stride, (const float*)z, z_row_stride, dt, (const float*)low,
                                 low_row_stride, b_off, c_off, a_log, d_skip, state, slots, seq_start, (float*)out,
                                 out_row_stride, n_seqs, channels, n_state, out_scale, piece, max_pieces, ends, stream);
  if (dtype == kBF16)
    return launch_selective_scan((const __nv_bfloat16*)x, x_row_stride, (const __nv_bfloat16*)z, z_row_stride, dt,
                                 (const __nv_bfloat16*)low, low_row_stride, b_off, c_off, a_log, d_skip, state, slots,
                                 seq_start, (__nv_bfloat16*)out, out_row_stride, n_seqs, channels, n_state, out_scale, piece,
                                 max_pieces, ends, stream);
  return fail("selective_scan: unknown dtype %d", dtype);
}
