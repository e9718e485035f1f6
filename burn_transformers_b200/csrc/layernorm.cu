// LayerNorm over the last axis of 32-bit rows: statistics and normalisation in 32-bit,
// the result rounded once to the output type.  mean, then the mean of squared deviations
// (two passes, no E[x^2]-E[x]^2 cancellation).  `rows` (optional) picks the input rows.
#include "common.cuh"

namespace bt {

template <typename TOut, int THREADS>
__global__ void __launch_bounds__(THREADS)
layernorm_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ gamma,
                 const float* __restrict__ beta, TOut* __restrict__ out, int width, float eps) {
  __shared__ float scratch[33];
  extern __shared__ float row_cache[];  // width floats
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  const float* src = x + (long long)(rows ? rows[r] : r) * width;
  float s = 0.f;
  for (int c = threadIdx.x; c < width; c += THREADS) {
    const float v = src[c];
    row_cache[c] = v;
    s += v;
  }
  const float mean = block_sum(s, scratch) / (float)width;
  float q = 0.f;
  for (int c = threadIdx.x; c < width; c += THREADS) {
    const float d = row_cache[c] - mean;
    q += d * d;
  }
  const float var = block_sum(q, scratch) / (float)width;
  const float rstd = 1.f / sqrtf(var + eps);
  TOut* dst = out + (long long)r * width;
  for (int c = threadIdx.x; c < width; c += THREADS) {
    float v = (row_cache[c] - mean) * rstd;
    v = v * gamma[c] + (beta ? beta[c] : 0.f);
    dst[c] = from_float<TOut>(v);
  }
}

// The same for many rows that are not long: a warp holds one row in registers (J vectors of four per lane), so the
// row is read once and nothing is handed over between warps.  width is a multiple of 4, at most 128 J.
// EARLY: gamma and beta, which no step writes, are asked for before the wait for the predecessor and held in registers: a step of few
// rows is a chain of latencies, and from memory they are the longest of this kernel's two.  The last rows come first: the
// kernel before wrote them last, so that of many rows more are still in L2 (16,384 x 1,600 after the residual stream was written: 34 to 30 us).
template <typename TOut, int J, bool EARLY>
__global__ void __launch_bounds__(256)
layernorm_rows_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ gamma,
                      const float* __restrict__ beta, TOut* __restrict__ out, int n_rows, int width, float eps) {
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = n_rows - 1 - (int)(blockIdx.x * (blockDim.x >> 5) + warp);
  auto weights = [&](int j, float4& g, float4& b) {
    const int c = (j * 32 + lane) * 4;
    g = b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= width) return;
    g = *reinterpret_cast<const float4*>(gamma + c);
    if (beta) b = *reinterpret_cast<const float4*>(beta + c);
  };
  float4 gs[EARLY ? J : 1], bs[EARLY ? J : 1];
  if constexpr (EARLY)
#pragma unroll
    for (int j = 0; j < J; ++j) weights(j, gs[j], bs[j]);
  pdl_wait();
  if (r < 0) return;
  const float* src = x + (long long)(rows ? rows[r] : r) * width;
  float4 v[J];
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int c = (j * 32 + lane) * 4;
    v[j] = c < width ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < J; ++j) s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
  const float mean = warp_sum(s) / (float)width;
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < J; ++j)
    if ((j * 32 + lane) * 4 < width) {
      const float a = v[j].x - mean, b = v[j].y - mean, c = v[j].z - mean, d = v[j].w - mean;
      q += (a * a + b * b) + (c * c + d * d);
    }
  const float rstd = 1.f / sqrtf(warp_sum(q) / (float)width + eps);
  TOut* dst = out + (long long)r * width;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int c = (j * 32 + lane) * 4;
    if (c < width) {
      float4 g, b;
      if constexpr (EARLY) {
        g = gs[j];
        b = bs[j];
      } else {
        weights(j, g, b);
      }
      const float o0 = (v[j].x - mean) * rstd * g.x + b.x, o1 = (v[j].y - mean) * rstd * g.y + b.y;
      const float o2 = (v[j].z - mean) * rstd * g.z + b.z, o3 = (v[j].w - mean) * rstd * g.w + b.w;
      if constexpr (sizeof(TOut) == 4) {
        *reinterpret_cast<float4*>(dst + c) = make_float4(o0, o1, o2, o3);
      } else {
        __nv_bfloat162 lo = __floats2bfloat162_rn(o0, o1), hi = __floats2bfloat162_rn(o2, o3);
        uint2 packed;
        packed.x = *reinterpret_cast<unsigned*>(&lo);
        packed.y = *reinterpret_cast<unsigned*>(&hi);
        *reinterpret_cast<uint2*>(dst + c) = packed;
      }
    }
  }
}

template <typename TOut>
static int launch_layernorm(const float* x, const int* rows, const float* gamma, const float* beta, TOut* out, int n_rows,
                            int width, float eps, cudaStream_t stream) {
  constexpr int T = 256;
  const bool aligned = width % 4 == 0 && ((unsigned long long)x % 16) == 0 && ((unsigned long long)gamma % 16) == 0 &&
                       ((unsigned long long)beta % 16) == 0 && ((unsigned long long)out % (sizeof(TOut) == 4 ? 16 : 8)) == 0;
  // (the choice must not depend on the number of rows: a row's result is the same alone and in a batch)
  if (aligned && width <= 2048) {
    // (a warp's arithmetic does not depend on how many warps share its block.  Two: blocks that come and go singly keep more
    // rows in flight than blocks of eight, and registers only for the vectors that a row has do the same: 16,384 rows of 1,600
    // took 37.5 us with eight warps and 16 vectors, 31.0 so; of 1,024 22.5, 21.6 so)
    const dim3 grid((n_rows + 1) / 2), block(64);
    // (gamma and beta ahead of the wait: rows and weights cold, before / after, us: 64 x 1,600 4.2 / 2.1, 2,048 x 768 4.3 / 3.2, 4,096 x 1,600
    // 13.6 / 11.9, 8,192 x 1,600 16.8 / 21.3, 16,384 x 1,024 18.4 / 19.4: beyond 4,096 rows the registers cost more than the wait did)
    const bool early = n_rows <= 4096;
#define BT_LN_ROWS(J)                                                                                                              \
  BT_PDL_OK("layernorm", early ? launch_pdl(layernorm_rows_kernel<TOut, J, true>, grid, block, 0, stream, 1, x, rows, gamma, beta, \
                                            out, n_rows, width, eps)                                                              \
                               : launch_pdl(layernorm_rows_kernel<TOut, J, false>, grid, block, 0, stream, 1, x, rows, gamma, beta, \
                                            out, n_rows, width, eps))
    if (width <= 1024) BT_LN_ROWS(8);
    else if (width <= 1280) BT_LN_ROWS(10);
    else if (width <= 1664) BT_LN_ROWS(13);
    else BT_LN_ROWS(16);
#undef BT_LN_ROWS
    return 0;
  }
  const size_t smem = (size_t)width * sizeof(float);
  BT_PDL_OK("layernorm", launch_pdl(layernorm_kernel<TOut, T>, dim3(n_rows), dim3(T), smem, stream, 1, x, rows, gamma, beta, out,
                                    width, eps));
  return 0;
}

}  // namespace bt

extern "C" int bt_layernorm(const float* x, const int* rows, const float* gamma, const float* beta, void* out,
                            int n_rows, int width, float eps, int out_dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_rows >= 0 && width > 0, "layernorm: bad sizes rows=%d width=%d", n_rows, width);
  BT_CHECK(width <= 12000, "layernorm: width %d exceeds the supported 12000", width);
  if (n_rows == 0) return 0;
  if (out_dtype == kF32) return launch_layernorm<float>(x, rows, gamma, beta, (float*)out, n_rows, width, eps, stream);
  if (out_dtype == kBF16)
    return launch_layernorm<__nv_bfloat16>(x, rows, gamma, beta, (__nv_bfloat16*)out, n_rows, width, eps, stream);
  return fail("layernorm: unknown dtype %d", out_dtype);
}
