// The products inside a chunk of 64 tokens of a recurrence (lightning.cu, mlstm.cu, gla.cu), on tensor cores with no operand's bits given up:
// a 32-bit number goes in as the sum of three bfloat16 numbers (the residues are exact), a number that bfloat16 holds as itself,
// and the products whose parts' orders add up to two at most are formed; what is left out is below 2^-24 of a product (of a number below
// 2^-110 the parts end at 2^-133, bfloat16's last).
//
// Tensor cores cut their sums where a multiply-add rounds them.  So the products of the first parts begin from zero at every step of
// 16 along the sum and are added in 32-bit registers; those of the smaller parts, 2^-8 and less of the result, share accumulators.
//
// A number that is infinite, or that bfloat16 rounds to infinity, has no parts: its residue is none.  And a weight of zero that stands for a
// later token meets that token's values all the same.  Either way the sum that it meets is no finite number, whatever else is in it; the
// kernels look for such results when they have written them and form them again by multiply-adds (cm_state says whether there are
// any, cm_bad_rows where; cm_plain_row forms a row).
//
// A block is four warps with 16 rows of the result each.  The second operands lie in shared memory, their parts one behind the
// other, in rows of (columns + 8) numbers: eight rows' 16-byte pieces then meet all banks, however they are read.
#pragma once
#include "common.cuh"

namespace bt {

constexpr int CM_CHUNK = 64, CM_THREADS = 128, CM_COLS = 64;
constexpr int CM_ROW = CM_COLS + 8;      // numbers of a row of value channels in shared memory

__device__ __forceinline__ void cm_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same from zero
__device__ __forceinline__ void cm_mma_zero(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// (two sums an instruction)
__device__ __forceinline__ void cm_add(float (&d)[4], const float (&x)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i += 2)
    asm("{\n.reg .b64 a, b;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nadd.rn.f32x2 a, a, b;\nmov.b64 {%0, %1}, a;\n}\n"
        : "+f"(d[i]), "+f"(d[i + 1]) : "f"(x[i]), "f"(x[i + 1]));
}
__device__ __forceinline__ void cm_ldmatrix(unsigned (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void cm_ldmatrix_t(unsigned (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}

// two numbers' parts, each as a pair of bfloat16
template <int PARTS>
__device__ __forceinline__ void cm_split(float x, float y, unsigned (&part)[PARTS]) {
#pragma unroll
  for (int q = 0; q < PARTS; ++q) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    part[q] = *reinterpret_cast<const unsigned*>(&h);
    if (q + 1 < PARTS) {
      // (both differences at once; they are exact)
      asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nmov.b64 c, {%4, %4};\nfma.rn.f32x2 a, b, c, a;\n"
          "mov.b64 {%0, %1}, a;\n}\n" : "+f"(x), "+f"(y) : "r"(part[q] << 16), "r"(part[q] & 0xffff0000u), "r"(0xbf800000u));
    }
  }
}

__device__ __forceinline__ void cm_load8(const float* p, float (&x)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void cm_load8(const __nv_bfloat16* p, float (&x)[8]) { unpack16(*reinterpret_cast<const uint4*>(p), x); }
__device__ __forceinline__ float2 cm_load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 cm_load2(const __nv_bfloat16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }

// Rows of `cols` numbers (whole pieces of 8) into shared memory, part behind part (`part_size` numbers apart), rows `stride` apart:
// load(row, column, x) gives eight numbers.
template <int PARTS, typename Load>
__device__ __forceinline__ void cm_fill(__nv_bfloat16* dst, int rows, int cols, int stride, int part_size, Load load) {
  const int pieces = cols / 8;
#pragma unroll 2
  for (int i = threadIdx.x; i < rows * pieces; i += CM_THREADS) {
    const int r = i / pieces, c = (i - r * pieces) * 8;
    float x[8];
    load(r, c, x);
    unsigned part[4][PARTS];
#pragma unroll
    for (int u = 0; u < 4; ++u) cm_split<PARTS>(x[2 * u], x[2 * u + 1], part[u]);
#pragma unroll
    for (int q = 0; q < PARTS; ++q)
      *reinterpret_cast<uint4*>(dst + q * part_size + r * stride + c) = make_uint4(part[0][q], part[1][q], part[2][q], part[3][q]);
  }
}

// big += a0 b0, small += the other products of the parts, for two neighbouring tiles of eight columns (b: their operands, part by
// part: the first tile's two registers, then the second's)
template <int AP, int BP>
__device__ __forceinline__ void cm_products(float (&big0)[4], float (&small0)[4], float (&big1)[4], float (&small1)[4],
                                            const unsigned (&a)[AP][4], const unsigned (&b)[BP][4]) {
#pragma unroll
  for (int q = AP + BP - 2; q >= 0; --q)
#pragma unroll
    for (int pa = 0; pa < AP; ++pa) {
      const int pb = q - pa;
      if (q > 2 || pb < 0 || pb >= BP) continue;
      if (q > 0) {
        cm_mma(small0, a[pa], b[pb][0], b[pb][1]);
        cm_mma(small1, a[pa], b[pb][2], b[pb][3]);
      } else {
        float x[4], y[4];
        cm_mma_zero(x, a[0], b[0][0], b[0][1]);
        cm_mma_zero(y, a[0], b[0][2], b[0][3]);
        cm_add(big0, x);
        cm_add(big1, y);
      }
    }
}

// One step of 16 along the sum over a second operand whose rows run along the sum (S_in or V: [sum][column]): rows row0.., the tiles
// of columns [0, 8 tiles).
template <int AP, int BP, int TILES>
__device__ __forceinline__ void cm_step_rows(float (&big)[TILES][4], float (&small)[TILES][4], const unsigned (&a)[AP][4],
                                             const __nv_bfloat16* src, int row0, int part_size) {
  const int lane = threadIdx.x & 31;
  const __nv_bfloat16* at = src + (row0 + (lane & 15)) * CM_ROW + (lane >> 4) * 8;
#pragma unroll
  for (int j = 0; j < TILES; j += 2) {
    unsigned b[BP][4];
#pragma unroll
    for (int q = 0; q < BP; ++q) cm_ldmatrix_t(b[q], at + q * part_size + 8 * j);
    cm_products<AP, BP>(big[j], small[j], big[j + 1], small[j + 1], a, b);
  }
}

// The chunk's contribution to the state, rows d of `dim` (16 a warp and round), columns [0, 64):  sum_s K'[s][d] V[s][c], K' and V in
// shared memory ([token][channel]; KP and VP parts).  store(d, c, x, y) gets the numbers of columns c and c + 1.  Whether one of this
// thread's numbers may not be finite.
template <int KP, int VP, typename Store>
__device__ __forceinline__ bool cm_state(const __nv_bfloat16* k, int k_stride, int k_part, const __nv_bfloat16* v, int v_part, int dim,
                                         Store store) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t2 = (lane & 3) * 2;
  float zeros = 0.f;      // (zero times all numbers' sum, which is no finite number if one of them is none)
  for (int d0 = warp * 16; d0 < dim; d0 += 64) {
    float big[8][4] = {}, small[8][4] = {};
#pragma unroll
    for (int s = 0; s < CM_CHUNK; s += 16) {
      unsigned a[KP][4];
      // (matrices: channels d0.. of tokens s.., channels d0 + 8.., then tokens s + 8..)
      const __nv_bfloat16* at = k + (s + (lane & 7) + (lane >> 4) * 8) * k_stride + d0 + (lane >> 3 & 1) * 8;
#pragma unroll
      for (int q = 0; q < KP; ++q) cm_ldmatrix_t(a[q], at + q * k_part);
      cm_step_rows<KP, VP, 8>(big, small, a, v, s, v_part);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) big[j][i] += small[j][i];
      zeros = fmaf((big[j][0] + big[j][1]) + (big[j][2] + big[j][3]), 0.f, zeros);
      store(d0 + g, 8 * j + t2, big[j][0], big[j][1]);
      store(d0 + g + 8, 8 * j + t2, big[j][2], big[j][3]);
    }
  }
  return zeros != 0.f;
}

// Of a warp's 16 rows those with a number that is not finite, a bit each; a, b: whether this thread has one in its rows lane / 4 and lane / 4 + 8.
__device__ __forceinline__ unsigned cm_bad_rows(bool a, bool b) {
  unsigned rows = 0;
  const unsigned all_a = __ballot_sync(0xffffffffu, a), all_b = __ballot_sync(0xffffffffu, b);
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    rows |= (unsigned)((all_a >> (4 * g) & 15u) != 0) << g;
    rows |= (unsigned)((all_b >> (4 * g) & 15u) != 0) << (g + 8);
  }
  return rows;
}

// Columns lane and lane + 32 of a block whose incoming state holds a NaN: so do their results, which need not be formed again (in(d, c) as
// below; a state that has become NaN would bring every later token here).
template <typename In>
__device__ __forceinline__ void cm_nan_columns(int dim, int cols, In in, bool (&nan)[2]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float sum = 0.f;
#pragma unroll 8
    for (int d = 0; d < dim; ++d) {
      const float y = lane + 32 * h < cols ? in(d, lane + 32 * h) : 0.f;
      sum = isnan(y) ? y : sum;
    }
    nan[h] = isnan(sum) || lane + 32 * h >= cols;
  }
}

// The chunk's token t by multiply-adds, a warp together, columns lane and lane + 32 of a block's: x = carry * sum_d q(d) in(d, c) and then, token
// by token, weigh(s, q . k_s) v(s, c), up to 128 channels d.  The sum of the weights is returned.  (Eight channels' or tokens' numbers are asked
// for at once: a state that has become infinite brings every later token here.)
template <typename Q, typename K, typename V, typename In, typename Weigh>
__device__ __forceinline__ float cm_plain_row(int t, int dim, int cols, float carry, Q q, K k, V v, In in, Weigh weigh, float (&x)[2]) {
  const int lane = threadIdx.x & 31;
  float sum = 0.f, own[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) own[i] = lane + 32 * i < dim ? q(lane + 32 * i) : 0.f;
  x[0] = x[1] = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll 1
    for (int d = 32 * i; d < min(dim, 32 * i + 32); d += 8) {      // (dim is whole operand tiles)
      float y[8][2];
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) y[u][h] = lane + 32 * h < cols ? in(d + u, lane + 32 * h) : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float z = __shfl_sync(0xffffffffu, own[i], (d + u) & 31);
        x[0] = fmaf(z, y[u][0], x[0]);
        x[1] = fmaf(z, y[u][1], x[1]);
      }
    }
  x[0] *= carry;
  x[1] *= carry;
#pragma unroll 1
  for (int s = 0; s <= t; s += 8) {
    float w[8], y[8][2];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int token = min(s + u, t);
      w[u] = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (lane + 32 * i < dim) w[u] = fmaf(own[i], k(token, lane + 32 * i), w[u]);
#pragma unroll
      for (int h = 0; h < 2; ++h) y[u][h] = lane + 32 * h < cols ? v(token, lane + 32 * h) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float z = weigh(min(s + u, t), warp_sum(w[u]));
      if (s + u > t) break;
      sum += z;
      x[0] = fmaf(z, y[u][0], x[0]);
      x[1] = fmaf(z, y[u][1], x[1]);
    }
  }
  return sum;
}

}  // namespace bt
