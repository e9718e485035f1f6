// The small steps around the latent attention, fused for steps of few tokens (decode): with a handful of rows every
// kernel is a link in a chain of launches, so the three steps before the attention and the two after it are one kernel
// each.  One block per (token, head), or tensor cores where the channels are whole operand tiles; 32-bit sums; T is the type of projections, weights, cache rows and results.
//
//   latent_decode_prep    q~ = W_uk,h^T q_plain | rotated q_rot  ->  the query as the latent rows meet it;
//                         the block of head 0 also RMS-norms the token's latent, rotates its shared key part and files
//                         both in the page (what bt_latent_append does)
//   latent_decode_finish  joins the attention's splits (or reads its result), multiplies by W_uv,h and by sigmoid(gate)
#include "chunk_mma.cuh"
#include "common.cuh"

namespace bt {

constexpr int LD_THREADS = 256;

// y[j] = sum_k x[k] * W[k][j] for one block: x (K floats) in shared memory, W [K][N] with N contiguous in global memory.
// A thread reads 16 bytes of a row of W at a time; the threads that do not fit beside one another along a row take
// other rows (slices of K), and the slices' partial sums meet in `red` (LD_THREADS * 8 floats of shared memory).
// The results are left in `y` (N <= LD_MAX_N floats of shared memory).  N must be a multiple of the 16-byte piece and W
// 16-byte aligned: `ld_matvec_ok` says so; otherwise the caller loops column by column.
constexpr int LD_MAX_N = 1024;
template <typename T>
__device__ __forceinline__ bool ld_matvec_ok(const T* w, int N) {
  constexpr int VEC = 16 / sizeof(T);
  return N % VEC == 0 && N / VEC <= LD_THREADS && N <= LD_MAX_N && ((unsigned long long)w % 16) == 0;
}

template <typename T>
__device__ __forceinline__ void ld_matvec(const float* x, const T* __restrict__ w, int K, int N, float* red, float* y) {
  constexpr int VEC = 16 / sizeof(T);
  const int groups = N / VEC;                       // threads side by side along a row
  const int slices = LD_THREADS / groups;           // rows of W in flight at once
  const int tid = threadIdx.x, cg = tid % groups, sl = tid / groups;
  float acc[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
  if (sl < slices) {
#pragma unroll 4
    for (int k = sl; k < K; k += slices) {
      const uint4 raw = *reinterpret_cast<const uint4*>(w + (long long)k * N + cg * VEC);
      const T* e = reinterpret_cast<const T*>(&raw);
      const float xv = x[k];
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] = fmaf(xv, to_float(e[v]), acc[v]);
    }
#pragma unroll
    for (int v = 0; v < VEC; ++v) red[(sl * groups + cg) * VEC + v] = acc[v];
  }
  __syncthreads();
  for (int j = tid; j < N; j += LD_THREADS) {
    const int g = j / VEC, v = j - g * VEC;
    float sum = 0.f;
    for (int s2 = 0; s2 < slices; ++s2) sum += red[(s2 * groups + g) * VEC + v];
    y[j] = sum;
  }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(LD_THREADS)
latent_decode_prep_kernel(const T* __restrict__ proj, long long row_stride, int q_off,
                          const T* __restrict__ latent_rows, long long latent_row_stride,   // the tokens' [latent | key part]
                          const T* __restrict__ uk,                 // [heads][dim][rank]
                          const float* __restrict__ norm_weight, float eps, const int* __restrict__ positions,
                          const int* __restrict__ token_seq, const float* __restrict__ inv_freq, int rot_dims,
                          const int* __restrict__ table, int table_stride, int table_len, int page_size,
                          T* __restrict__ pool, T* __restrict__ q_latent, int n_heads, int dim, int rank, int rot,
                          int owns) {
  extern __shared__ float sm[];      // [dim] the plain query
  __shared__ float scratch[33];
  __shared__ __align__(16) float red[LD_THREADS * 8];
  __shared__ float y_s[LD_MAX_N];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  const int pos = positions[t];
  const T* row = proj + (long long)t * row_stride;
  const T* q = row + q_off + (long long)h * (dim + rot);
  for (int d = threadIdx.x; d < dim; d += blockDim.x) sm[d] = to_float(q[d]);
  __syncthreads();
  const int dk = rank + rot;
  T* dst = q_latent + ((long long)t * n_heads + h) * dk;
  const T* w = uk + (long long)h * dim * rank;
  if (ld_matvec_ok(w, rank)) {
    ld_matvec(sm, w, dim, rank, red, y_s);
    for (int r = threadIdx.x; r < rank; r += blockDim.x) dst[r] = from_float<T>(y_s[r]);
  } else {
    for (int r = threadIdx.x; r < rank; r += blockDim.x) {
      float acc = 0.f;
      for (int d = 0; d < dim; ++d) acc = fmaf(sm[d], to_float(w[(long long)d * rank + r]), acc);
      dst[r] = from_float<T>(acc);
    }
  }
  const int half = rot_dims / 2;
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    float s, c;
    sincosf((float)pos * inv_freq[i], &s, &c);
    const float u = to_float(q[dim + 2 * i]), v = to_float(q[dim + 2 * i + 1]);
    dst[rank + 2 * i] = from_float<T>(u * c - v * s);
    dst[rank + 2 * i + 1] = from_float<T>(v * c + u * s);
  }
  for (int c = rot_dims + threadIdx.x; c < rot; c += blockDim.x) dst[rank + c] = q[dim + c];
  if (!owns || h != 0) return;
  // the token's own latent row: norm, rotation, page (the same arithmetic as latent_append_kernel)
  const T* lat = latent_rows + (long long)t * latent_row_stride;
  float ss = 0.f;
  for (int c = threadIdx.x; c < rank; c += blockDim.x) {
    const float v = to_float(lat[c]);
    ss += v * v;
  }
  const float inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)rank + eps);
  const int seq = token_seq[t];
  const int lp = pos / page_size;
  const int page = table[(long long)seq * table_stride + (lp % table_len)];
  T* cell = pool + ((long long)page * page_size + (pos - lp * page_size)) * dk;
  for (int c = threadIdx.x; c < rank; c += blockDim.x) cell[c] = from_float<T>(to_float(lat[c]) * inv * norm_weight[c]);
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    float s, c;
    sincosf((float)pos * inv_freq[i], &s, &c);
    const float u = to_float(lat[rank + 2 * i]), v = to_float(lat[rank + 2 * i + 1]);
    cell[rank + 2 * i] = from_float<T>(u * c - v * s);
    cell[rank + 2 * i + 1] = from_float<T>(v * c + u * s);
  }
  for (int c = rot_dims + threadIdx.x; c < rot; c += blockDim.x) cell[rank + c] = lat[rank + c];
}

// The same for bfloat16 with channels in whole operand tiles, on tensor cores.  Above, every (token, head) reads the head's
// W_uk for itself, 64 KB at rank 512, and 64 tokens of 16 heads read 67 MB from L2; here a block of the grid's first part takes 64
// columns of one head's W_uk for 64 tokens (its weights travel before the wait for the kernel before), and a block of the second
// part one token's rotations and latent row.  64 tokens of
// 16 heads, rank 512, in a recorded layer: 13 to 6 us.
constexpr int LP_THREADS = 128;
__global__ void __launch_bounds__(LP_THREADS)
latent_decode_prep_mma_kernel(const __nv_bfloat16* __restrict__ proj, long long row_stride, int q_off,
                              const __nv_bfloat16* __restrict__ latent_rows, long long latent_row_stride,
                              const __nv_bfloat16* __restrict__ uk, const float* __restrict__ norm_weight, float eps,
                              const int* __restrict__ positions, const int* __restrict__ token_seq,
                              const float* __restrict__ inv_freq, int rot_dims, const int* __restrict__ table, int table_stride,
                              int table_len, int page_size, __nv_bfloat16* __restrict__ pool, __nv_bfloat16* __restrict__ q_latent,
                              int n_tokens, int n_heads, int dim, int rank, int rot, int owns, int product_blocks) {
  extern __shared__ __align__(16) unsigned char lp_smem[];
  __shared__ float scratch[33];
  pdl_trigger();
  const int dk = rank + rot, tid = threadIdx.x;
  if ((int)blockIdx.x < product_blocks) {
    __nv_bfloat16* w_s = reinterpret_cast<__nv_bfloat16*>(lp_smem);      // [dim][72]
    const int chunks = rank / CM_COLS, unit = blockIdx.x % (n_heads * chunks), head = unit / chunks, r0 = (unit - head * chunks) * CM_COLS;
    const __nv_bfloat16* w = uk + (long long)head * dim * rank + r0;
#pragma unroll 4
    for (int i = tid; i < dim * (CM_COLS / 8); i += LP_THREADS) {
      const int d = i / (CM_COLS / 8), c = i % (CM_COLS / 8) * 8;
      *reinterpret_cast<uint4*>(w_s + d * CM_ROW + c) = __ldg(reinterpret_cast<const uint4*>(w + (long long)d * rank + c));
    }
    __syncthreads();
    pdl_wait();
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t2 = (lane & 3) * 2;
    const int ta = (int)(blockIdx.x / (n_heads * chunks)) * 64 + warp * 16 + g, tb = ta + 8;
    if (ta - g >= n_tokens) return;
    const __nv_bfloat16* q = proj + q_off + (long long)head * (dim + rot) + t2;
    float o[8][4] = {}, none[8][4];
#pragma unroll 4
    for (int d = 0; d < dim; d += 16) {
      unsigned x[1][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = i & 1 ? tb : ta;
        x[0][i] = t < n_tokens ? *reinterpret_cast<const unsigned*>(q + t * row_stride + d + 8 * (i >> 1)) : 0u;
      }
      cm_step_rows<1, 1, 8>(o, none, x, w_s, d, 0);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = h ? tb : ta;
      if (t >= n_tokens) break;
      __nv_bfloat16* dst = q_latent + ((long long)t * n_heads + head) * dk + r0 + t2;
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<__nv_bfloat162*>(dst + 8 * j) = __floats2bfloat162_rn(o[j][2 * h], o[j][2 * h + 1]);
    }
    return;
  }
  pdl_wait();
  const int t = blockIdx.x - product_blocks, half = rot_dims / 2, pos = positions[t];
  const __nv_bfloat16* q = proj + t * row_stride + q_off;
  __nv_bfloat16* dst = q_latent + (long long)t * n_heads * dk;
  for (int i = tid; i < n_heads * half; i += LP_THREADS) {
    const int h = i / half, c = i - h * half;
    float s, co;
    sincosf((float)pos * inv_freq[c], &s, &co);
    const __nv_bfloat16* src = q + h * (dim + rot) + dim + 2 * c;
    const float u = to_float(src[0]), v = to_float(src[1]);
    dst[h * dk + rank + 2 * c] = from_float<__nv_bfloat16>(u * co - v * s);
    dst[h * dk + rank + 2 * c + 1] = from_float<__nv_bfloat16>(v * co + u * s);
  }
  const int plain = rot - rot_dims;
  for (int i = tid; i < n_heads * plain; i += LP_THREADS) {
    const int h = i / plain, c = rot_dims + i - h * plain;
    dst[h * dk + rank + c] = q[h * (dim + rot) + dim + c];
  }
  if (!owns) return;
  // the token's own latent row: norm, rotation, page (the same arithmetic as latent_append_kernel)
  const __nv_bfloat16* lat = latent_rows + t * latent_row_stride;
  float ss = 0.f;
  for (int c = tid; c < rank; c += LP_THREADS) {
    const float v = to_float(lat[c]);
    ss += v * v;
  }
  const float inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)rank + eps);
  const int lp = pos / page_size;
  const int page = table[(long long)token_seq[t] * table_stride + (lp % table_len)];
  __nv_bfloat16* cell = pool + ((long long)page * page_size + (pos - lp * page_size)) * dk;
  for (int c = tid; c < rank; c += LP_THREADS) cell[c] = from_float<__nv_bfloat16>(to_float(lat[c]) * inv * norm_weight[c]);
  for (int i = tid; i < half; i += LP_THREADS) {
    float s, co;
    sincosf((float)pos * inv_freq[i], &s, &co);
    const float u = to_float(lat[rank + 2 * i]), v = to_float(lat[rank + 2 * i + 1]);
    cell[rank + 2 * i] = from_float<__nv_bfloat16>(u * co - v * s);
    cell[rank + 2 * i + 1] = from_float<__nv_bfloat16>(v * co + u * s);
  }
  for (int c = rot_dims + tid; c < rot; c += LP_THREADS) cell[rank + c] = lat[rank + c];
}

constexpr int LD_MAX_SPLITS = 64;

template <typename T>
__global__ void __launch_bounds__(LD_THREADS)
latent_decode_finish_kernel(const float* __restrict__ part, const T* __restrict__ mixed_latent, int n_splits,
                            const T* __restrict__ uv,               // [heads][rank][vdim]
                            const T* __restrict__ gate, long long gate_row_stride, int gate_per_head, T* __restrict__ out,
                            long long out_row_stride, int n_heads, int rank, int vdim) {
  extern __shared__ float sm[];      // [rank] the weighted sum of latents, then [LD_MAX_SPLITS] the splits' weights
  float* o_s = sm;
  float* w_s = sm + rank;
  __shared__ __align__(16) float red[LD_THREADS * 8];
  __shared__ float y_s[LD_MAX_N];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  const long long unit = (long long)t * n_heads + h;
  if (n_splits > 1) {
    const float* src = part + unit * n_splits * (rank + 2);
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      float m[LD_MAX_SPLITS / 32], l[LD_MAX_SPLITS / 32];
      float top = -INFINITY;
#pragma unroll
      for (int i = 0; i < LD_MAX_SPLITS / 32; ++i) {
        const int s = lane + 32 * i;
        m[i] = s < n_splits ? src[(long long)s * (rank + 2) + rank] : -INFINITY;
        l[i] = s < n_splits ? src[(long long)s * (rank + 2) + rank + 1] : 0.f;
        top = fmaxf(top, m[i]);
      }
      top = warp_max(top);
      float denom = 0.f;
#pragma unroll
      for (int i = 0; i < LD_MAX_SPLITS / 32; ++i) {
        m[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
        denom += l[i] * m[i];
      }
      denom = warp_sum(denom);
      const float inv = denom > 0.f ? 1.f / denom : 0.f;
#pragma unroll
      for (int i = 0; i < LD_MAX_SPLITS / 32; ++i)
        if (lane + 32 * i < n_splits) w_s[lane + 32 * i] = m[i] * inv;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < rank; c += blockDim.x) {
      float v = 0.f;
#pragma unroll 8
      for (int s = 0; s < n_splits; ++s) v = fmaf(src[(long long)s * (rank + 2) + c], w_s[s], v);
      o_s[c] = v;
    }
  } else {
    const T* src = mixed_latent + unit * rank;
    for (int c = threadIdx.x; c < rank; c += blockDim.x) o_s[c] = to_float(src[c]);
  }
  __syncthreads();
  const T* w = uv + (long long)h * rank * vdim;
  const bool wide = ld_matvec_ok(w, vdim);
  if (wide) ld_matvec(o_s, w, rank, vdim, red, y_s);
  for (int j = threadIdx.x; j < vdim; j += blockDim.x) {
    float acc = wide ? y_s[j] : 0.f;
    if (!wide)
      for (int r = 0; r < rank; ++r) acc = fmaf(o_s[r], to_float(w[(long long)r * vdim + j]), acc);
    if (gate) acc *= 1.f / (1.f + expf(-to_float(gate[(long long)t * gate_row_stride + (gate_per_head ? h : (long long)h * vdim + j)])));
    out[(long long)t * out_row_stride + (long long)h * vdim + j] = from_float<T>(acc);
  }
}

// The same for bfloat16 with channels in whole operand tiles, on tensor cores: a block takes one head's W_uv (which travels before
// the wait for the kernel before) for 8 tokens, where every (token, head) read it for itself; its eight warps share the latent
// channels, join the splits' parts of theirs (in 32 bits, in split order) and multiply them as the sum of three bfloat16 numbers,
// which hold all of their bits; the warps' sums are added in warp order.  64 tokens of 16 heads, four
// splits of rank 512, in a recorded layer: 17 to 9 us.
constexpr int LF_TOKENS = 8, LF_WARPS = LD_THREADS / 32;
template <bool JOIN>
__global__ void __launch_bounds__(LD_THREADS)
latent_decode_finish_mma_kernel(const float* __restrict__ part, const __nv_bfloat16* __restrict__ mixed_latent, int n_splits,
                                const __nv_bfloat16* __restrict__ uv, const __nv_bfloat16* __restrict__ gate,
                                long long gate_row_stride, int gate_per_head, __nv_bfloat16* __restrict__ out,
                                long long out_row_stride, int n_tokens, int n_heads, int rank, int vdim) {
  extern __shared__ __align__(16) unsigned char lf_smem[];
  constexpr int PARTS = JOIN ? 3 : 1;
  const int ld = vdim + 8;
  __nv_bfloat16* w_s = reinterpret_cast<__nv_bfloat16*>(lf_smem);                        // [rank][vdim + 8]
  float* red = reinterpret_cast<float*>(lf_smem + (size_t)rank * ld * 2);                // [8 warps][8 tokens][vdim]
  __shared__ float share[LF_TOKENS][LD_MAX_SPLITS];
  pdl_trigger();
  const int t0 = blockIdx.x * LF_TOKENS, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2,
            t2 = (lane & 3) * 2;
  const __nv_bfloat16* w = uv + (long long)h * rank * vdim;
  const int pieces = vdim / 8;
  for (int i = tid; i < rank * pieces; i += LD_THREADS) {
    const int r = i / pieces, c = (i - r * pieces) * 8;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(w_s + r * ld + c)),
                 "l"(w + (long long)r * vdim + c) : "memory");
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  pdl_wait();
  if (JOIN && t0 + warp < n_tokens) {      // a warp a token: the splits' shares
    const float* src = part + ((long long)(t0 + warp) * n_heads + h) * n_splits * (rank + 2);
    float m[LD_MAX_SPLITS / 32], l[LD_MAX_SPLITS / 32];
    float top = -INFINITY;
#pragma unroll
    for (int i = 0; i < LD_MAX_SPLITS / 32; ++i) {
      const int s = lane + 32 * i;
      m[i] = s < n_splits ? src[(long long)s * (rank + 2) + rank] : -INFINITY;
      l[i] = s < n_splits ? src[(long long)s * (rank + 2) + rank + 1] : 0.f;
      top = fmaxf(top, m[i]);
    }
    top = warp_max(top);
    float denom = 0.f;
#pragma unroll
    for (int i = 0; i < LD_MAX_SPLITS / 32; ++i) {
      m[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
      denom += l[i] * m[i];
    }
    denom = warp_sum(denom);
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
#pragma unroll
    for (int i = 0; i < LD_MAX_SPLITS / 32; ++i)
      if (lane + 32 * i < n_splits) share[warp][lane + 32 * i] = m[i] * inv;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  const int t = t0 + g;      // this thread's row (the tile's rows 8 to 15 hold nothing)
  const long long unit = (long long)t * n_heads + h;
  float o[8][4] = {}, o_small[8][4] = {};
  for (int k = warp * 16; k < rank; k += LF_WARPS * 16) {
    float2 x[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (t < n_tokens) {
      if (JOIN) {
        const float* src = part + unit * n_splits * (rank + 2) + k + t2;
#pragma unroll 4
        for (int s = 0; s < n_splits; ++s) {
          const float f = share[g][s];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 v = *reinterpret_cast<const float2*>(src + (long long)s * (rank + 2) + 8 * i);
            x[i].x = fmaf(v.x, f, x[i].x);
            x[i].y = fmaf(v.y, f, x[i].y);
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) x[i] = cm_load2(mixed_latent + unit * rank + k + t2 + 8 * i);
      }
    }
    unsigned a[PARTS][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      unsigned parts[PARTS];
      cm_split<PARTS>(x[i].x, x[i].y, parts);
#pragma unroll
      for (int q = 0; q < PARTS; ++q) {
        a[q][2 * i] = parts[q];
        a[q][2 * i + 1] = 0u;
      }
    }
    const __nv_bfloat16* at = w_s + (k + (lane & 15)) * ld + (lane >> 4) * 8;
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      if (8 * j >= vdim) break;
      unsigned b[1][4];
      cm_ldmatrix_t(b[0], at + 8 * j);
      cm_products<PARTS, 1>(o[j], o_small[j], o[j + 1], o_small[j + 1], a, b);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (8 * j < vdim)
      *reinterpret_cast<float2*>(red + (warp * LF_TOKENS + g) * vdim + 8 * j + t2) = make_float2(o[j][0] + o_small[j][0], o[j][1] + o_small[j][1]);
  __syncthreads();
  for (int i = tid; i < LF_TOKENS * vdim; i += LD_THREADS) {
    const int r = i / vdim, j = i - r * vdim, token = t0 + r;
    if (token >= n_tokens) continue;
    float acc = 0.f;
#pragma unroll
    for (int q = 0; q < LF_WARPS; ++q) acc += red[(q * LF_TOKENS + r) * vdim + j];
    if (JOIN && !isfinite(acc)) {      // (an infinity, or a number that bfloat16 rounds to one, has no parts: by multiply-adds)
      const float* src = part + ((long long)token * n_heads + h) * n_splits * (rank + 2);
      acc = 0.f;
#pragma unroll 1
      for (int k = 0; k < rank && !isnan(acc); ++k) {
        float x = 0.f;
#pragma unroll 1
        for (int s = 0; s < n_splits; ++s) x = fmaf(src[(long long)s * (rank + 2) + k], share[r][s], x);
        acc = fmaf(x, to_float(w_s[k * ld + j]), acc);
      }
    }
    if (gate) acc *= 1.f / (1.f + expf(-to_float(gate[(long long)token * gate_row_stride + (gate_per_head ? h : (long long)h * vdim + j)])));
    out[(long long)token * out_row_stride + (long long)h * vdim + j] = from_float<__nv_bfloat16>(acc);
  }
}

}  // namespace bt

// The queries are the channels from `q_off` on of `proj`'s rows; the tokens' latent rows are `latent_rows` (rows
// `latent_row_stride` elements apart), or, when that is null, the channels from `latent_off` on of the same `proj` rows.
extern "C" int bt_latent_decode_prep(const void* proj, long long row_stride, int q_off, int latent_off,
                                     const void* latent_rows, long long latent_row_stride, const void* uk,
                                     const float* norm_weight, float eps, const int* positions, const int* token_seq,
                                     const float* inv_freq, int rot_dims, const int* table, int table_stride,
                                     int table_len, int page_size, void* pool, void* q_latent, int n_tokens, int n_heads,
                                     int dim, int rank, int rot, int owns, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && n_heads <= 65535 && dim > 0 && rank > 0 && rot >= 0 && rot_dims >= 0 && rot_dims <= rot &&
           rot_dims % 2 == 0 && dim <= 8192, "latent_decode_prep: bad sizes heads=%d dim=%d rank=%d rot=%d", n_heads, dim, rank, rot);
  if (n_tokens == 0) return 0;
  const dim3 grid(n_tokens, n_heads), block(LD_THREADS);
  const size_t smem = (size_t)dim * sizeof(float);
  const size_t elem = dtype == kF32 ? 4 : 2;
  if (latent_rows == nullptr) {
    latent_rows = (const char*)proj + (size_t)latent_off * elem;
    latent_row_stride = row_stride;
  }
  if (dtype == kBF16 && dim % 16 == 0 && dim <= 256 && rank % CM_COLS == 0 && rot % 2 == 0 && q_off % 2 == 0 && row_stride % 2 == 0 &&
      ((unsigned long long)uk % 16 | (unsigned long long)proj % 4 | (unsigned long long)q_latent % 4) == 0) {
    const long long product_blocks = (long long)n_heads * (rank / CM_COLS) * ((n_tokens + 63) / 64);
    BT_CHECK(product_blocks + n_tokens <= 0x7fffffffll, "latent_decode_prep: %d tokens of %d heads are too many", n_tokens, n_heads);
    BT_PDL_OK("latent_decode_prep", launch_pdl(latent_decode_prep_mma_kernel, dim3((unsigned)(product_blocks + n_tokens)), dim3(LP_THREADS),
                                               (size_t)dim * CM_ROW * 2, stream, 1, (const __nv_bfloat16*)proj, row_stride, q_off,
                                               (const __nv_bfloat16*)latent_rows, latent_row_stride, (const __nv_bfloat16*)uk,
                                               norm_weight, eps, positions, token_seq, inv_freq, rot_dims, table, table_stride,
                                               table_len, page_size, (__nv_bfloat16*)pool, (__nv_bfloat16*)q_latent, n_tokens, n_heads,
                                               dim, rank, rot, owns, (int)product_blocks));
    return 0;
  }
  if (dtype == kF32)
    BT_PDL_OK("latent_decode_prep", launch_pdl(latent_decode_prep_kernel<float>, grid, block, smem, stream, 1,
                                               (const float*)proj, row_stride, q_off, (const float*)latent_rows,
                                               latent_row_stride, (const float*)uk,
                                               norm_weight, eps, positions, token_seq, inv_freq, rot_dims, table,
                                               table_stride, table_len, page_size, (float*)pool, (float*)q_latent, n_heads,
                                               dim, rank, rot, owns));
  else if (dtype == kBF16)
    BT_PDL_OK("latent_decode_prep", launch_pdl(latent_decode_prep_kernel<__nv_bfloat16>, grid, block, smem, stream, 1,
                                               (const __nv_bfloat16*)proj, row_stride, q_off,
                                               (const __nv_bfloat16*)latent_rows, latent_row_stride,
                                               (const __nv_bfloat16*)uk, norm_weight, eps, positions, token_seq, inv_freq,
                                               rot_dims, table, table_stride, table_len, page_size, (__nv_bfloat16*)pool,
                                               (__nv_bfloat16*)q_latent, n_heads, dim, rank, rot, owns));
  else
    return fail("latent_decode_prep: unknown dtype %d", dtype);
  return 0;
}

extern "C" int bt_latent_decode_finish(const float* part, const void* mixed_latent, int n_splits, const void* uv,
                                       const void* gate, long long gate_row_stride, int gate_per_head, void* out, long long out_row_stride,
                                       int n_tokens, int n_heads, int rank, int vdim, int dtype, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(n_heads > 0 && n_heads <= 65535 && rank > 0 && rank <= 8192 && vdim > 0 && n_splits >= 1 &&
           n_splits <= LD_MAX_SPLITS, "latent_decode_finish: bad sizes heads=%d rank=%d vdim=%d splits=%d", n_heads, rank, vdim, n_splits);
  BT_CHECK(n_splits == 1 ? mixed_latent != nullptr : part != nullptr, "latent_decode_finish: the attention's result is missing");
  if (n_tokens == 0) return 0;
  const size_t smem_mma = (size_t)rank * (vdim + 8) * 2 + (size_t)LF_WARPS * LF_TOKENS * vdim * 4;
  if (dtype == kBF16 && rank % 16 == 0 && vdim % 16 == 0 && vdim <= 64 && smem_mma <= 200 * 1024 &&
      ((unsigned long long)uv % 16 | (unsigned long long)part % 8 | (unsigned long long)mixed_latent % 4) == 0) {
    const dim3 tiles((n_tokens + LF_TOKENS - 1) / LF_TOKENS, n_heads);
    auto kern = n_splits > 1 ? latent_decode_finish_mma_kernel<true> : latent_decode_finish_mma_kernel<false>;
    static SharedMemoryAllowance allowed[2];
    BT_CHECK(allow_shared_memory(allowed[n_splits > 1], kern, smem_mma), "latent_decode_finish: cannot reserve %zu bytes of shared memory", smem_mma);
    BT_PDL_OK("latent_decode_finish", launch_pdl(kern, tiles, dim3(LD_THREADS), smem_mma, stream, 1, part,
                                                 (const __nv_bfloat16*)mixed_latent, n_splits, (const __nv_bfloat16*)uv,
                                                 (const __nv_bfloat16*)gate, gate_row_stride, gate_per_head, (__nv_bfloat16*)out,
                                                 out_row_stride, n_tokens, n_heads, rank, vdim));
    return 0;
  }
  const dim3 grid(n_tokens, n_heads), block(LD_THREADS);
  const size_t smem = (size_t)(rank + LD_MAX_SPLITS) * sizeof(float);
  if (dtype == kF32)
    BT_PDL_OK("latent_decode_finish", launch_pdl(latent_decode_finish_kernel<float>, grid, block, smem, stream, 1, part,
                                                 (const float*)mixed_latent, n_splits, (const float*)uv, (const float*)gate,
                                                 gate_row_stride, gate_per_head, (float*)out, out_row_stride, n_heads, rank, vdim));
  else if (dtype == kBF16)
    BT_PDL_OK("latent_decode_finish",
              launch_pdl(latent_decode_finish_kernel<__nv_bfloat16>, grid, block, smem, stream, 1, part,
                         (const __nv_bfloat16*)mixed_latent, n_splits, (const __nv_bfloat16*)uv, (const __nv_bfloat16*)gate,
                         gate_row_stride, gate_per_head, (__nv_bfloat16*)out, out_row_stride, n_heads, rank, vdim));
  else
    return fail("latent_decode_finish: unknown dtype %d", dtype);
  return 0;
}
