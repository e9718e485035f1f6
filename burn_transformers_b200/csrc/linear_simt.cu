// out[M,N] = act(A[M,K] @ W + bias) (+ residual), accumulated in 32-bit with plain fused
// multiply-adds (no tensor cores, no reduced-precision matrix mode).  This is the matrix
// product of the true 32-bit path (weights with a long K: linear_split_tcgen05.cu) and the fallback for shapes the tensor-core kernels refuse.
// W is either [K,N] with N contiguous (a Conv1D weight as stored) or [N,K] with K contiguous
// (an embedding table used as a tied readout).  Every output element is a sum over k in an order
// that its sizes alone decide, so a row's result does not depend on which other rows are in the call.
#include "common.cuh"

namespace bt {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TIn, typename TOut, bool W_IS_NK>
__global__ void __launch_bounds__(256)
linear_simt_kernel(const TIn* __restrict__ A, const TIn* __restrict__ W, const float* __restrict__ bias,
                   const float* residual, TOut* out, int M, int N, int K, int act) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    {  // A tile: thread -> row tid/4, four consecutive k
      const int r = tid >> 2, kq = (tid & 3) * 4;
      const int gm = m0 + r;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int gk = k0 + kq + u;
        As[kq + u][r] = (gm < M && gk < K) ? to_float(A[(long long)gm * K + gk]) : 0.f;
      }
    }
    if (W_IS_NK) {  // thread -> n tid/4, four consecutive k
      const int c = tid >> 2, kq = (tid & 3) * 4;
      const int gn = n0 + c;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int gk = k0 + kq + u;
        Bs[kq + u][c] = (gn < N && gk < K) ? to_float(W[(long long)gn * K + gk]) : 0.f;
      }
    } else {  // thread -> k tid/16, four consecutive n
      const int kr = tid >> 4, nq = (tid & 15) * 4;
      const int gk = k0 + kr;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int gn = n0 + nq + u;
        Bs[kr][nq + u] = (gn < N && gk < K) ? to_float(W[(long long)gk * N + gn]) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[gn];
      v = apply_activation(v, act);
      if (residual) v += residual[(long long)gm * N + gn];
      out[(long long)gm * N + gn] = from_float<TOut>(v);
    }
  }
}

// 32-bit operands in rows of 16-byte pieces (K, and N of a [K,N] weight, multiples of 4).  What bounds such a product on
// this GPU is the way from shared memory to the registers: a 16-byte read of a warp takes four cycles of the
// multiprocessor whatever its lanes share, so 8 x 4 numbers a thread (12 reads for 128 multiply-adds) run at half the
// multiply-add rate.  Hence few threads with large tiles: a warp owns the whole BM x BN tile of its block (16 x 4 numbers a
// thread at 64 x 32: 20 reads for 256), and the four warps of a block share K: warp g takes the numbers 4 g .. 4 g + 3 of
// every 16, in pairs (two multiply-adds an instruction, each rounded as fmaf rounds).  At the end the four sums are added in
// warp order through shared memory.  The split is the same for every tile, so a row's result does not depend on M.
// Pieces of 32 along k travel through a ring of STAGES by cp.async.  Both operands lie in shared memory as they lie in
// global memory: A as rows of 32 + 4 numbers; W [K,N] as rows of BN + 4 columns, a thread's columns being groups of four; W
// [N,K] as A, a thread's columns being BN / TN apart (rows 36 numbers apart: eight of them meet all 32 banks once).
constexpr int FK = 32;                 // k of a piece
constexpr int FMA_GROUPS = 4;          // warps that share K
constexpr int FMA_THREADS = 32 * FMA_GROUPS;

template <int BM, int BN, int STAGES, bool W_IS_NK>
struct FmaTile {
  static constexpr int KS = FK + 4;                                          // numbers between rows of a k-contiguous operand
  static constexpr int A_NUMBERS = BM * KS, W_NUMBERS = W_IS_NK ? BN * KS : FK * (BN + 4);
  static constexpr int RING = STAGES * (A_NUMBERS + W_NUMBERS);
  static constexpr int SUMS = BM * (BN + 4);                                 // one warp's sums, at the end
  static constexpr size_t SMEM = sizeof(float) * (size_t)(RING > SUMS ? RING : SUMS);
};
// 16 bytes from global to shared memory, or zeros (an address that is not read must still be one of the operand's)
__device__ __forceinline__ void fma_copy16(float* dst, const float* src, bool read) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(read ? 16 : 0) : "memory");
}
// d += a * b for two 32-bit numbers that lie in one 64-bit register, each product and sum rounded once
__device__ __forceinline__ void fma_pair(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 fma_halves(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// TM x TN numbers a thread: 32 threads cover BM x BN
template <int BM, int BN, int TM, int TN, int STAGES, bool W_IS_NK>
__global__ void __launch_bounds__(FMA_THREADS)
linear_fma_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                  const float* residual, float* out, int M, int N, int K, int act, int tiles_n, int rows16) {
  using Tile = FmaTile<BM, BN, STAGES, W_IS_NK>;
  constexpr int TX = BN / TN, TY = BM / TM, KS = Tile::KS;
  static_assert(TX * TY == 32, "a warp covers the tile");
  constexpr int LA = BM * FK / 4 / FMA_THREADS, LB = BN * FK / 4 / FMA_THREADS;      // 16-byte copies a thread
  static_assert(LA * FMA_THREADS * 4 == BM * FK && LB * FMA_THREADS * 4 == BN * FK, "a piece is whole copies of every thread");
  constexpr int GN = TN / 4;
  extern __shared__ __align__(16) float fma_smem[];
  const int tid = threadIdx.x, group = tid >> 5, lane = tid & 31;
  const int tx = lane % TX, ty = lane / TX;
  const int m0 = (int)(blockIdx.x / tiles_n) * BM, n0 = (int)(blockIdx.x % tiles_n) * BN;
  const int pieces = (K + FK - 1) / FK;
  auto fetch = [&](int piece) {
    if (piece < pieces) {
      float* as = fma_smem + (piece % STAGES) * (Tile::A_NUMBERS + Tile::W_NUMBERS);
      float* ws = as + Tile::A_NUMBERS;
      const int k0 = piece * FK;
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        const int at = tid + i * FMA_THREADS, r = at / (FK / 4), kq = (at % (FK / 4)) * 4;
        const bool in = m0 + r < M && k0 + kq < K;
        fma_copy16(as + r * KS + kq, in ? A + (long long)(m0 + r) * K + k0 + kq : A, in);
      }
#pragma unroll
      for (int i = 0; i < LB; ++i) {
        const int at = tid + i * FMA_THREADS;
        if (W_IS_NK) {
          const int c = at / (FK / 4), kq = (at % (FK / 4)) * 4;
          const bool in = n0 + c < N && k0 + kq < K;
          fma_copy16(ws + c * KS + kq, in ? W + (long long)(n0 + c) * K + k0 + kq : W, in);
        } else {
          const int kr = at / (BN / 4), nq = (at % (BN / 4)) * 4;
          const bool in = n0 + nq < N && k0 + kr < K;
          fma_copy16(ws + kr * (BN + 4) + nq, in ? W + (long long)(k0 + kr) * N + n0 + nq : W, in);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");      // (empty groups past the end keep the count)
  };
  // sums in pairs: of two adjacent columns where W is [K,N], of the even and the odd k of one column where it is [N,K]
  constexpr int PAIRS = W_IS_NK ? TN : TN / 2;
  unsigned long long acc[TM][PAIRS];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) acc[i][j] = 0ull;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  for (int it = 0; it < pieces; ++it) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                  // piece `it` has landed for every thread, and everyone has left piece `it` - 1
    fetch(it + STAGES - 1);           // into the stage of piece `it` - 1
    const float* as = fma_smem + (it % STAGES) * (Tile::A_NUMBERS + Tile::W_NUMBERS) + ty * KS;
    const float* ws = fma_smem + (it % STAGES) * (Tile::A_NUMBERS + Tile::W_NUMBERS) + Tile::A_NUMBERS;
#pragma unroll
    for (int half = 0; half < FK / 16; ++half) {
      const int k4 = half * 16 + group * 4;
      if (W_IS_NK) {
        ulonglong2 w[TN];             // four consecutive k of a column, as two pairs
#pragma unroll
        for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + (tx + j * TX) * KS + k4);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * TY * KS + k4);      // rows ty, ty + TY, ...
#pragma unroll
          for (int j = 0; j < TN; ++j) fma_pair(acc[i][j], a.x, w[j].x);
#pragma unroll
          for (int j = 0; j < TN; ++j) fma_pair(acc[i][j], a.y, w[j].y);
        }
      } else {
        ulonglong2 w[4][GN];          // [k][group of four columns]
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int g = 0; g < GN; ++g) w[k][g] = *reinterpret_cast<const ulonglong2*>(ws + (k4 + k) * (BN + 4) + g * (BN / GN) + tx * 4);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(as + i * TY * KS + k4);
          const float ak[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            unsigned long long twice;
            asm("mov.b64 %0, {%1, %1};" : "=l"(twice) : "f"(ak[k]));
#pragma unroll
            for (int g = 0; g < GN; ++g) {
              fma_pair(acc[i][2 * g], twice, w[k][g].x);
              fma_pair(acc[i][2 * g + 1], twice, w[k][g].y);
            }
          }
        }
      }
    }
  }
  // the warps' sums, one warp after the other into one tile in shared memory (over the ring: its readers are through)
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  for (int g = 0; g < FMA_GROUPS; ++g) {
    __syncthreads();
    if (group != g) continue;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      float* row = fma_smem + (ty + i * TY) * (BN + 4);
      if (W_IS_NK) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float2 h = fma_halves(acc[i][j]);
          const float v = h.x + h.y;
          row[tx + j * TX] = g == 0 ? v : row[tx + j * TX] + v;
        }
      } else {
#pragma unroll
        for (int q = 0; q < GN; ++q) {
          const float2 lo = fma_halves(acc[i][2 * q]), hi = fma_halves(acc[i][2 * q + 1]);
          float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
          float4* at = reinterpret_cast<float4*>(row + q * (BN / GN) + tx * 4);
          if (g > 0) {
            const float4 before = *at;
            v.x += before.x; v.y += before.y; v.z += before.z; v.w += before.w;
          }
          *at = v;
        }
      }
    }
  }
  __syncthreads();
#pragma unroll 2
  for (int i = tid; i < BM * BN / 4; i += FMA_THREADS) {
    const int r = i / (BN / 4), c = (i % (BN / 4)) * 4, gm = m0 + r, gn = n0 + c;
    if (gm >= M || gn >= N) continue;
    const float4 sum = *reinterpret_cast<const float4*>(fma_smem + r * (BN + 4) + c);
    float v[4] = {sum.x, sum.y, sum.z, sum.w};
    const long long o = (long long)gm * N + gn;
    if (rows16) {
      if (bias) {
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(bias + gn));
        v[0] += b4.x; v[1] += b4.y; v[2] += b4.z; v[3] += b4.w;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = apply_activation(v[j], act);
      if (residual) {
        const float4 r4 = *reinterpret_cast<const float4*>(residual + o);
        v[0] += r4.x; v[1] += r4.y; v[2] += r4.z; v[3] += r4.w;
      }
      *reinterpret_cast<float4*>(out + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (gn + j >= N) continue;
        if (bias) v[j] += bias[gn + j];
        v[j] = apply_activation(v[j], act);
        if (residual) v[j] += residual[o + j];
        out[o + j] = v[j];
      }
    }
  }
}

template <int BM, int BN, int TM, int TN, int STAGES, bool W_IS_NK>
static int launch_fma(const float* A, const float* W, const float* bias, const float* residual, float* out, int M, int N,
                      int K, int act, int rows16, cudaStream_t stream) {
  using Tile = FmaTile<BM, BN, STAGES, W_IS_NK>;
  auto kern = linear_fma_kernel<BM, BN, TM, TN, STAGES, W_IS_NK>;
  static SharedMemoryAllowance allowed;
  BT_CHECK(allow_shared_memory(allowed, kern, Tile::SMEM), "linear: cannot reserve %zu bytes of shared memory", Tile::SMEM);
  const int tiles_n = (N + BN - 1) / BN;
  const dim3 grid((unsigned)((long long)tiles_n * ((M + BM - 1) / BM)));
  kern<<<grid, FMA_THREADS, Tile::SMEM, stream>>>(A, W, bias, residual, out, M, N, K, act, tiles_n, rows16);
  return 0;
}

// The tile: large ones read less from shared memory per multiply-add, small ones leave fewer multiprocessors idle and end
// sooner.  Measured per k of 768 (us): a tile alone 18 / 12.5 / 10.5 at 64 x 32 / 32 x 32 / 16 x 32; each further one on the
// same multiprocessor 13 / 6.5 / 3.7 (W [N,K]: 16 / 7.1 / 3.7).  The sum for the fullest multiprocessor decides; all of
// it grows with K alike.
// GPT-2 small's products at 804 rows, before (one 64 x 64 tile of 4 x 4 a thread, kernel above) and with this rule: 2304 x
// 768 145 to 82 us, 768 x 768 76 to 36, 3072 x 768 181 to 103, 768 x 3072 292 to 127; 768 x 768 at one row 48 to 11.
template <bool NK>
static int launch_fma_best(const float* A, const float* W, const float* bias, const float* residual, float* out, int M, int N,
                           int K, int act, int rows16, cudaStream_t stream) {
  const int sms = sm_count();
  BT_CHECK(sms > 0, "linear: cannot read the number of multiprocessors of the current device");
  auto cost = [&](int bm, int alone, int more) {
    const long long tiles = (long long)((M + bm - 1) / bm) * ((N + 31) / 32);
    return alone - more + (tiles + sms - 1) / sms * more;
  };
  const long long large = cost(64, 180, NK ? 160 : 130), middle = cost(32, 125, NK ? 71 : 65), small = cost(16, 105, 37);
  if (large <= middle && large <= small)
    return launch_fma<64, 32, 16, 4, 4, NK>(A, W, bias, residual, out, M, N, K, act, rows16, stream);
  if (middle <= small) return launch_fma<32, 32, 8, 4, 4, NK>(A, W, bias, residual, out, M, N, K, act, rows16, stream);
  return launch_fma<16, 32, 4, 4, 4, NK>(A, W, bias, residual, out, M, N, K, act, rows16, stream);
}

template <typename TIn, typename TOut>
static void launch(const void* A, const void* W, const float* bias, const float* residual, void* out, int M, int N,
                   int K, int w_is_nk, int act, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (w_is_nk)
    linear_simt_kernel<TIn, TOut, true><<<grid, 256, 0, stream>>>((const TIn*)A, (const TIn*)W, bias, residual,
                                                                  (TOut*)out, M, N, K, act);
  else
    linear_simt_kernel<TIn, TOut, false><<<grid, 256, 0, stream>>>((const TIn*)A, (const TIn*)W, bias, residual,
                                                                   (TOut*)out, M, N, K, act);
}

}  // namespace bt

// in_dtype: type of A and W.  out_dtype: type of out (32-bit when it is the residual stream or logits).
extern "C" int bt_linear_simt(const void* A, const void* W, const float* bias, const float* residual, void* out,
                              int M, int N, int K, int w_is_nk, int act, int in_dtype, int out_dtype,
                              cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(M >= 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
  BT_CHECK(act >= 0 && act <= 2, "linear: unknown activation %d", act);
  BT_CHECK((long long)((M + BM - 1) / BM) <= 65535, "linear: M=%d needs more than 65535 row tiles", M);
  BT_CHECK(!(residual && out_dtype != kF32), "linear: a residual needs a 32-bit output");
  if (M == 0) return 0;
  const bool pieces16 = K % 4 == 0 && (w_is_nk || N % 4 == 0) && ((unsigned long long)A | (unsigned long long)W) % 16 == 0;
  // (16-byte accesses of the epilogue need every row of every operand there on a 16-byte boundary)
  const bool rows16 = N % 4 == 0 && ((unsigned long long)out | (unsigned long long)residual | (unsigned long long)bias) % 16 == 0;
  if (in_dtype == kF32 && out_dtype == kF32 && pieces16) {
    const int rc = w_is_nk ? launch_fma_best<true>((const float*)A, (const float*)W, bias, residual, (float*)out, M, N, K, act, rows16, stream)
                           : launch_fma_best<false>((const float*)A, (const float*)W, bias, residual, (float*)out, M, N, K, act, rows16, stream);
    if (rc != 0) return rc;
  } else if (in_dtype == kF32 && out_dtype == kF32)
    launch<float, float>(A, W, bias, residual, out, M, N, K, w_is_nk, act, stream);
  else if (in_dtype == kBF16 && out_dtype == kF32)
    launch<__nv_bfloat16, float>(A, W, bias, residual, out, M, N, K, w_is_nk, act, stream);
  else if (in_dtype == kBF16 && out_dtype == kBF16)
    launch<__nv_bfloat16, __nv_bfloat16>(A, W, bias, residual, out, M, N, K, w_is_nk, act, stream);
  else
    return fail("linear: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  BT_LAUNCH_OK("linear_simt");
  return 0;
}
