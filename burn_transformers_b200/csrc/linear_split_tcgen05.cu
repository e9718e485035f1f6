// out[M,N] = act(A[M,K] @ W + bias) (+ residual) for 32-bit operands, on the fifth-generation tensor cores without giving up any
// of the operands' bits: every number is the sum of three bfloat16 numbers, x = x1 + x2 + x3 (x1 = bf16(x), x2 = bf16(x - x1),
// x3 = x - x1 - x2, which 8 bits hold: the residues are exact), and
//
//     a b = a1 b1 + (a1 b2 + a2 b1) + (a2 b2 + a1 b3 + a3 b1) + (terms below 2^-24 |a b|, left out)
//
// Products of bfloat16 numbers are exact in 32 bits.  Tensor cores cut their sums where a multiply-add rounds them, so no sum stays
// in them for long: every 64 of K (a k-block) begin from zero, in three accumulators by size, R0 = a1 b1, R1 = a1 b2 + a2 b1, R2 =
// a1 b3 + a2 b2 + a3 b1, and R0 + (R1 + R2) is added in 32-bit registers, in order, to the sum of its eighth of the k-blocks (a
// segment); the segments' sums s0 .. s7 are added as ((s0 + s1) + (s2 + s3)) + ((s4 + s5) + (s6 + s7)).  An element's
// sums depend on K alone, never on the tile, the split or the other rows: a row gives the same bits whatever is in the call.
// A result that is not finite is formed again by multiply-adds (the split of an infinity, or of a number that rounds to one,
// is no number), up to the first NaN, so infinities and NaN come out as they do there.
//
// Against 64 bits the result is closer than that of the multiply-add kernel (linear_simt.cu) at every size measured: 768 x 768 8.7e-8
// and 2.5e-7, 768 x 3072 1.0e-7 and 5.0e-7 (norms, normal operands, 1 to 1,600 rows).
//
// The three parts of W lie one behind the other, so that one product takes all of them: a1 [b1 b2 b3] into [R0 R1 R2], a2 [b1 b2] into
// [R1 R2], a3 b1 into R2.  (A tcgen05.mma takes 45 ns and more however narrow it is: as six products of 64 columns, or of 128 by a
// pair of blocks, a k-block took 1.3 and 1.8 us.)
//
// A block takes tiles of 128 x 64 one after the other, or, where there are few, a cluster of 2, 4 or 8 blocks one tile, each 4, 2 or 1
// of the segments: its sums then go to the block of the cluster that owns their columns (distributed shared memory), which adds them.
// Sixteen warps (128 registers a thread) with fixed jobs:
//   warps 0-7    fetch 32-bit numbers, split them and write the operand tiles (128-byte swizzle; A and W [N,K] K-major, W [K,N] as
//                it lies, MN-major) into one of two stages of 64 along k.  Numbers wait in registers, 32 along k at a time and three
//                of those deep: a fetch takes longer than a split;
//   warps 8-15   add each k-block's three sums from tensor memory (two sets in turn) into registers, and finish the tile (a warp
//                reaches the 32 rows of its quarter; the two warps of a quarter take half of the columns each);
//   warp 8       also issues a k-block's 12 products from one elected lane.
// A k-block takes 1.35 us, in which 216 KB go through shared memory's port, two thirds of what it moves: 96 KB that the products read, 72 KB
// of operand tiles written, 48 KB fetched.  The counters show warps waiting for what they fetched before all else (4.9 of 9 cycles an
// instruction at 804 x 768 x 3,072; issue slots 38 %, tensor pipe 13 %).  (Fetched by the tensor memory accelerator as 32-bit tiles first: 1.75 us, a way more through it; one
// accumulator for all small terms, tiles of 128 columns by pairs of blocks: 2.2.)
// W may be [K,N] with N contiguous or [N,K] with K contiguous.  Every wait is bounded and reports through the status word.
#include "common.cuh"
#include "tcgen05.cuh"

namespace bt {

constexpr int LS_BM = 128, LS_STAGES = 2;
constexpr int LS_SPLIT_WARPS = 8, LS_SUM_WARPS = 8;
constexpr int LS_THREADS = 32 * (LS_SPLIT_WARPS + LS_SUM_WARPS);
constexpr int LS_BN = 64, LS_SEGMENTS = 8;
constexpr int LS_PATCH = 20;                             // floats between rows of a warp's 32 x 16 patch

struct SplitParams {
  const float* a;           // [M, K]
  const float* w;           // [K, N] or [N, K]
  const float* bias;        // [N] or null
  const float* residual;    // [M, N] or null (may be `out`)
  float* out;               // [M, N]
  int* status;
  int M, N, K, act, rows16;
};

// four numbers as three groups of four bfloat16 (the residues two an instruction: h * -1 + x is exact)
__device__ __forceinline__ unsigned long long ls_pair(unsigned lo, unsigned hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
__device__ __forceinline__ unsigned ls_halves(unsigned long long& x, bool last) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x));
  const unsigned h = tc_pack(lo, hi);
  if (!last) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(x) : "l"(ls_pair(h << 16, h & 0xffff0000u)), "l"(ls_pair(0xbf800000u, 0xbf800000u)));
  return h;
}
__device__ __forceinline__ void ls_split(const float4& v, uint2 (&part)[3]) {
  unsigned long long x = ls_pair(__float_as_uint(v.x), __float_as_uint(v.y)), y = ls_pair(__float_as_uint(v.z), __float_as_uint(v.w));
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    part[p].x = ls_halves(x, p == 2);
    part[p].y = ls_halves(y, p == 2);
  }
}

// Behind the stages: what SPLIT blocks of a tile send one another, [block][row][64 / SPLIT], or the warps' patches.
template <int SPLIT>
constexpr size_t ls_smem() {
  return (size_t)LS_STAGES * 3 * (LS_BM + LS_BN) * TC_BK * 2 + 1024 +
         (SPLIT > 1 ? (size_t)LS_BM * LS_BN * 4 : (size_t)LS_SUM_WARPS * 32 * LS_PATCH * 4);
}
// 16 columns of this thread's lane of tensor memory
__device__ __forceinline__ void ls_st16(unsigned taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr), "f"(v[0]),
      "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]),
      "f"(v[13]), "f"(v[14]), "f"(v[15])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// One result by multiply-adds, sixteen numbers asked for at once, up to the first NaN, which nothing behind it changes: of rows that
// are NaN, 804 x 768 x 3,072, 90 us as of any others (1,130 to the end of K).  a: the row; w: the column's first number.
template <bool NK>
__device__ __noinline__ float ls_plain(const float* a, const float* w, int N, int K) {
  float x = 0.f;
#pragma unroll 1
  for (int k = 0; k < K && !isnan(x); k += 16) {
    float av[16], wv[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      av[u] = k + u < K ? a[k + u] : 0.f;
      wv[u] = k + u < K ? w[NK ? (long long)(k + u) : (long long)(k + u) * N] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) x = fmaf(av[u], wv[u], x);
  }
  return x;
}

template <bool NK, int SPLIT>
__global__ void __launch_bounds__(LS_THREADS, 1) linear_split_kernel(SplitParams p) {
  extern __shared__ unsigned char ls_smem_raw[];
  __shared__ __align__(8) unsigned long long full[LS_STAGES], empty[LS_STAGES], sums_full[2], sums_free[2];
  __shared__ unsigned tmem_base;
  __shared__ int failed;
  constexpr int BN = LS_BN;
  constexpr unsigned A_PART = LS_BM * TC_BK * 2, W_PART = BN * TC_BK * 2, STAGE = 3 * (A_PART + W_PART);
  constexpr int TMEM_COLS = 512;      // two sets of R0 R1 R2
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<unsigned long long>(ls_smem_raw) + 1023ull) & ~1023ull);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  pdl_trigger();
  const int tiles_n = (p.N + BN - 1) / BN, n_tiles = ((p.M + LS_BM - 1) / LS_BM) * tiles_n;
  const int all_blocks = (p.K + TC_BK - 1) / TC_BK;
  const int rank = SPLIT > 1 ? (int)tc_rank() : 0, tile0 = (int)blockIdx.x / SPLIT, tile_step = (int)gridDim.x / SPLIT;
  // this block's segments, and their k-blocks
  constexpr int SEGS = LS_SEGMENTS / SPLIT;
  auto segment = [&](int j) { return (int)((long long)j * all_blocks / LS_SEGMENTS); };      // the first k-block of segment j
  const int kb0 = segment(rank * SEGS), k_blocks = segment(rank * SEGS + SEGS) - kb0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < LS_STAGES; ++s) {
      tc_bar_init(&full[s], LS_SPLIT_WARPS);
      tc_bar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc_bar_init(&sums_full[b], 1);
      tc_bar_init(&sums_free[b], LS_SUM_WARPS);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if constexpr (SPLIT > 1) tc_cluster_sync();      // (the others' shared memory may be written from here on)
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem = tmem_base;

  if (warp < LS_SPLIT_WARPS) {
    const int tid = threadIdx.x;                            // 0 .. 255
    constexpr int A_VECS = LS_BM * 32 / 4 / 256, W_VECS = BN * 32 / 4 / 256, VECS = A_VECS + W_VECS;
    // K-major: eight threads a row of 32 numbers; of the two rows that half a warp writes, one has the swizzle's other half
    const int x = tid >> 3, row_a = (x & ~7) | ((x & 1) << 2) | ((x & 7) >> 1), ka = (tid & 7) * 4;      // rows row_a + 32 j
    constexpr int QN = BN / 4;                          // 16-byte pieces of a row of W [K,N]
    const int kw = tid / QN, nw = tid % QN * 4;             // of W [K,N]: rows kw + 256 / QN j, columns nw ..
    // what is fetched next: half a k-block f_h of tile f_tile; this thread's first number of A's and W's there, and which rows exist
    int f_tile = tile0, f_h = 0, rows_a = 0, rows_w = 0;
    const float *at_a = p.a, *at_w = p.w;
    const long long step_a = 32ll * p.K, step_w = NK ? 32ll * p.K : (long long)(256 / QN) * p.N;      // from one piece of a thread to the next
    auto begin = [&]() {
      if (f_tile >= n_tiles || k_blocks == 0) return;
      const int tm = f_tile / tiles_n, n0 = (f_tile - tm * tiles_n) * BN;
      rows_a = max(0, min(A_VECS, (p.M - tm * LS_BM - row_a + 31) / 32));      // pieces j < rows_a lie in A
      at_a = p.a + (long long)(tm * LS_BM + row_a) * p.K + kb0 * TC_BK + ka;
      if (NK) {
        rows_w = max(0, min(W_VECS, (p.N - n0 - row_a + 31) / 32));
        at_w = p.w + (long long)(n0 + row_a) * p.K + kb0 * TC_BK + ka;
      } else {
        rows_w = n0 + nw < p.N ? W_VECS : 0;
        at_w = p.w + (long long)(kb0 * TC_BK + kw) * p.N + n0 + nw;
      }
    };
    auto fetch = [&](float4 (&v)[VECS]) {
      if (f_tile >= n_tiles || k_blocks == 0) return;
      const int left = p.K - kb0 * TC_BK - 32 * f_h;      // of K from here on
#pragma unroll
      for (int j = 0; j < W_VECS; ++j)
        v[A_VECS + j] = j < rows_w && (NK ? ka : kw + (256 / QN) * j) < left ? __ldg(reinterpret_cast<const float4*>(at_w + j * step_w))
                                                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < A_VECS; ++j)
        v[j] = j < rows_a && ka < left ? *reinterpret_cast<const float4*>(at_a + j * step_a) : make_float4(0.f, 0.f, 0.f, 0.f);
      at_a += 32;
      at_w += NK ? 32ll : 32ll * p.N;
      if (++f_h == 2 * k_blocks) {
        f_h = 0;
        f_tile += tile_step;
        begin();
      }
    };
    int tile = k_blocks > 0 ? tile0 : n_tiles, h = 0, i = 0;      // what is split next; k-blocks so far
    int kept_a = max(0, min(A_VECS, (p.M - tile / tiles_n * LS_BM - row_a + 31) / 32));
    bool ok = true;
    auto work = [&](float4 (&v)[VECS]) {
      if (!ok || tile >= n_tiles) return;
      const int s = i % LS_STAGES, second = h & 1;
      if (!second && i >= LS_STAGES && !__all_sync(0xffffffffu, tc_bar_wait(&empty[s], (i / LS_STAGES - 1) & 1))) {
        failed = 1;
        ok = false;
        return;
      }
      unsigned char* at = tiles + (size_t)s * STAGE;
      const int c = second * 4 + (ka >> 3), in_piece = (ka & 4) << 1;      // the 16-byte piece of a K-major row, and where in it
      // (rows of A past M are left as they are: whatever they hold goes to rows of the result that are not written)
#pragma unroll
      for (int j = 0; j < A_VECS; ++j) {
        const int r = row_a + 32 * j;
        if (j < kept_a) {
          uint2 part[3];
          ls_split(v[j], part);
          unsigned char* dst = at + r * 128 + ((c ^ (r & 7)) << 4) + in_piece;
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * A_PART) = part[q];
        }
      }
#pragma unroll
      for (int j = 0; j < W_VECS; ++j) {
        uint2 part[3];
        ls_split(v[A_VECS + j], part);
        unsigned char* dst = at + 3 * A_PART;
        {
          if constexpr (NK) {
            const int r = row_a + 32 * j;
            dst += r * 128 + ((c ^ (r & 7)) << 4) + in_piece;
          } else {
            const int r = second * 32 + kw + (256 / QN) * j;
            dst += r * 128 + (((nw >> 3) ^ (r & 7)) << 4) + ((nw & 4) << 1);
          }
#pragma unroll
          for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(dst + q * W_PART) = part[q];
        }
      }
      if (second) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_bar_arrive(&full[s]);
      }
      fetch(v);
      i += second;
      if (++h == 2 * k_blocks) {
        h = 0;
        tile += tile_step;
        kept_a = max(0, min(A_VECS, (p.M - tile / tiles_n * LS_BM - row_a + 31) / 32));
      }
    };
    float4 r0[VECS], r1[VECS], r2[VECS];
    begin();
    pdl_wait();
    fetch(r0);
    fetch(r1);
    fetch(r2);
    while (ok && tile < n_tiles) {
      work(r0);
      work(r1);
      work(r2);
    }
  } else {
    const int quarter = warp & 3, half = (warp - LS_SPLIT_WARPS) >> 2;
    constexpr int HALF = BN / 2;      // a warp's columns
    float* sums_s = reinterpret_cast<float*>(tiles + (size_t)LS_STAGES * STAGE);      // (SPLIT > 1)
    float* patch = sums_s + (warp - LS_SPLIT_WARPS) * (32 * LS_PATCH);
    const unsigned lanes = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(half * HALF);
    // 32-bit accumulator, bfloat16 operands, A K-major, W K-major or MN-major; the number of columns goes in for each product
    constexpr unsigned IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (NK ? 0u : 1u << 16) | ((unsigned)(LS_BM >> 4) << 24);
    constexpr unsigned long long W_STEP = NK ? 2 : (16 * 128) >> 4;      // 16 of K further: along the row, or 16 rows on
    auto issue = [&](int i) -> bool {
      const int s = i % LS_STAGES, buf = i & 1;
      if (!__all_sync(0xffffffffu, (i < 2 || tc_bar_wait(&sums_free[buf], ((i >> 1) - 1) & 1)) && tc_bar_wait(&full[s], (i / LS_STAGES) & 1)))
        return false;      // (a wait that runs out must not part the warp's lanes)
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      if (tc_elect()) {
        unsigned char* at = tiles + (size_t)s * STAGE;
        const unsigned d = tmem + (unsigned)(buf * 3 * BN);
        unsigned long long dw = tc_desc(at + 3 * A_PART);
        // (MN-major: 8 rows of 64 columns are 1024 bytes, the next 64 columns, the next part, lie W_PART further)
        if (!NK) dw = (dw & ~(0x3FFFull << 16)) | (unsigned long long)(W_PART >> 4) << 16;
#pragma unroll
        for (int k = 0; k < TC_BK / 16; ++k)
#pragma unroll
          for (int q = 0; q < 3; ++q)
            tc_mma(d + (unsigned)(q * BN), tc_desc(at + q * A_PART) + 2ull * k, dw + W_STEP * k, IDESC | (unsigned)((3 - q) * BN >> 3) << 17,
                   (k > 0 || q > 0) ? 1u : 0u);
        tc_commit(&empty[s]);
        tc_commit(&sums_full[buf]);
      }
      __syncwarp();
      return true;
    };
    const bool issuer = warp == LS_SPLIT_WARPS;
    pdl_wait();      // (the residual is read and the output written)
    int i = 0;      // k-blocks so far
    bool ok = true;
    for (int tile = tile0; tile < n_tiles && ok; tile += tile_step) {
      const int m0 = tile / tiles_n * LS_BM, n0 = tile % tiles_n * BN + half * HALF;
      float sum[HALF], even[SPLIT < 8 ? HALF : 1];      // of the segment; of the one before, where it waits for this one
#pragma unroll
      for (int c = 0; c < HALF; ++c) sum[c] = 0.f;
      auto take = [&](int i) -> bool {      // adds the sums of k-block i
        const int buf = i & 1;
        if (!__all_sync(0xffffffffu, tc_bar_wait(&sums_full[buf], (i >> 1) & 1))) return false;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
        for (int c0 = 0; c0 < HALF; c0 += 16) {
          float v[16], w[16];
          const unsigned at = lanes + (unsigned)(buf * 3 * BN + c0);
          tc_ld16(at + BN, v);
          tc_ld16(at + 2 * BN, w);
#pragma unroll
          for (int c = 0; c < 16; ++c) w[c] = v[c] + w[c];
          tc_ld16(at, v);
#pragma unroll
          for (int c = 0; c < 16; ++c) sum[c0 + c] += v[c] + w[c];
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) tc_bar_arrive(&sums_free[buf]);
        __syncwarp();
        return true;
      };
      // a segment's k-blocks: one ahead is issued while the one before is added
      int issued = 0, taken = 0;
      if (issuer && k_blocks > 0) {
        ok = issue(i);
        issued = 1;
      }
      const int row = m0 + quarter * 32 + lane;
#pragma unroll 1
      for (int j = 0; j < SEGS && ok; ++j) {
        const int end = segment(rank * SEGS + j + 1) - kb0;
        for (; taken < end && ok; ++taken) {
          if (issuer && issued < k_blocks) {
            ok = issue(i + issued);
            ++issued;
          }
          ok = ok && take(i + taken);
        }
        if (!ok) break;
        // segments in pairs, pairs in fours, fours together
        if constexpr (SPLIT < 8) {
          if (j % 2 == 0) {
#pragma unroll
            for (int c = 0; c < HALF; ++c) {
              even[c] = sum[c];
              sum[c] = 0.f;
            }
          } else {
            // (sums that wait for their partners do so in tensor memory, behind the accumulators: a pair's, then the first four's)
            const bool quad = SPLIT < 4 && j % 4 == 3, all = SPLIT == 1 && j == 7, last = j == SEGS - 1;
            const unsigned waiting = lanes + 6u * BN;
#pragma unroll
            for (int c0 = 0; c0 < HALF; c0 += 16) {
              float x[16], w[16];
#pragma unroll
              for (int c = 0; c < 16; ++c) x[c] = even[c0 + c] + sum[c0 + c];
              if (quad) {
                tc_ld16(waiting + c0, w);
#pragma unroll
                for (int c = 0; c < 16; ++c) x[c] = w[c] + x[c];
              }
              if (all) {
                tc_ld16(waiting + BN + c0, w);
#pragma unroll
                for (int c = 0; c < 16; ++c) x[c] = w[c] + x[c];
              }
              if (!last) ls_st16(waiting + (quad ? BN : 0) + c0, x);
#pragma unroll
              for (int c = 0; c < 16; ++c) sum[c0 + c] = last ? x[c] : 0.f;
            }
          }
        }
      }
      if constexpr (SPLIT > 1) {      // to the blocks that own these columns
        constexpr int OWN = BN / SPLIT;
#pragma unroll
        for (int c = 0; c < HALF; c += 4) {
          const int col = half * HALF + c;
          unsigned at;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at)
                       : "r"(tc_smem(sums_s + (rank * LS_BM + quarter * 32 + lane) * OWN + col % OWN)), "r"(col / OWN));
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(at), "f"(sum[c]), "f"(sum[c + 1]), "f"(sum[c + 2]),
                       "f"(sum[c + 3]) : "memory");
        }
      }
      i += k_blocks;
      if (!ok) {
        failed = 1;
        break;
      }
      if constexpr (SPLIT == 1) {
      __syncwarp();
      unsigned long long bad = 0;      // columns whose sum is not finite: formed again by multiply-adds
#pragma unroll
      for (int c = 0; c < HALF; ++c) bad |= (unsigned long long)!isfinite(sum[c]) << c;
      if (row >= p.M) bad = 0;
      while (bad) {
        const int c = __ffsll((long long)bad) - 1;
        bad &= bad - 1;
        if (n0 + c >= p.N) continue;
        const float x = ls_plain<NK>(p.a + (long long)row * p.K, p.w + (NK ? (long long)(n0 + c) * p.K : n0 + c), p.N, p.K);
#pragma unroll
        for (int u = 0; u < HALF; ++u) sum[u] = u == c ? x : sum[u];
      }
      __syncwarp();
      const int cq = lane & 3, rq = lane >> 2, row_base = m0 + quarter * 32 + rq;
#pragma unroll
      for (int c0 = 0; c0 < HALF; c0 += 16) {
        const int col0 = n0 + c0;
        if (col0 >= p.N) break;      // (uniform)
        if (p.rows16 && col0 + 16 <= p.N) {
          // rows of 16 columns through the warp's patch, so that four lanes cover 64 contiguous bytes of a row
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(patch + lane * LS_PATCH + 4 * j) = make_float4(sum[c0 + 4 * j], sum[c0 + 4 * j + 1], sum[c0 + 4 * j + 2], sum[c0 + 4 * j + 3]);
          __syncwarp();
          const long long o_base = (long long)row_base * p.N + col0 + 4 * cq;
          float4 res[4], b4 = make_float4(0.f, 0.f, 0.f, 0.f);
          if (p.residual) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (row_base + 8 * k < p.M) res[k] = *reinterpret_cast<const float4*>(p.residual + o_base + (long long)(8 * k) * p.N);
          }
          if (p.bias) b4 = __ldg(reinterpret_cast<const float4*>(p.bias + col0 + 4 * cq));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float4 x = *reinterpret_cast<const float4*>(patch + (rq + 8 * k) * LS_PATCH + 4 * cq);
            x.x = apply_activation(x.x + b4.x, p.act);
            x.y = apply_activation(x.y + b4.y, p.act);
            x.z = apply_activation(x.z + b4.z, p.act);
            x.w = apply_activation(x.w + b4.w, p.act);
            if (row_base + 8 * k < p.M) {
              if (p.residual) { x.x += res[k].x; x.y += res[k].y; x.z += res[k].z; x.w += res[k].w; }
              *reinterpret_cast<float4*>(p.out + o_base + (long long)(8 * k) * p.N) = x;
            }
          }
          __syncwarp();      // the patch is free again
        } else if (row < p.M) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            if (col0 + c >= p.N) break;
            const long long o = (long long)row * p.N + col0 + c;
            float x = apply_activation(sum[c0 + c] + (p.bias ? p.bias[col0 + c] : 0.f), p.act);
            if (p.residual) x += p.residual[o];
            p.out[o] = x;
          }
        }
      }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (failed) let_copies_land();
  if constexpr (SPLIT > 1) {
    tc_cluster_sync();      // every segment's sums have arrived (and nothing is written to another block from here on)
    constexpr int OWN = LS_BN / SPLIT;
    const float* sums_s = reinterpret_cast<const float*>(tiles + (size_t)LS_STAGES * STAGE);
    const int m0 = tile0 / tiles_n * LS_BM, n0 = tile0 % tiles_n * LS_BN + rank * OWN;
    for (int e = threadIdx.x; e < LS_BM * OWN; e += LS_THREADS) {
      const int r = e / OWN, c = e % OWN, row = m0 + r, col = n0 + c;
      if (row >= p.M || col >= p.N) continue;
      float from[SPLIT];
#pragma unroll
      for (int j = 0; j < SPLIT; ++j) from[j] = sums_s[(j * LS_BM + r) * OWN + c];
#pragma unroll
      for (int w = 1; w < SPLIT; w *= 2)      // (pairs, then pairs of pairs: the order of one block)
#pragma unroll
        for (int j = 0; j < SPLIT; j += 2 * w) from[j] += from[j + w];
      float x = from[0];
      if (!isfinite(x)) x = ls_plain<NK>(p.a + (long long)row * p.K, p.w + (NK ? (long long)col * p.K : col), p.N, p.K);
      x = apply_activation(x + (p.bias ? p.bias[col] : 0.f), p.act);
      const long long o = (long long)row * p.N + col;
      if (p.residual) x += p.residual[o];
      p.out[o] = x;
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && failed && p.status) atomicExch(p.status, 2);
}

template <bool NK, int SPLIT>
static int launch_split(const SplitParams& p, cudaStream_t stream) {
  constexpr size_t smem = ls_smem<SPLIT>();
  static_assert(smem <= 227 * 1024, "a multiprocessor's shared memory");
  auto kern = linear_split_kernel<NK, SPLIT>;
  static SharedMemoryAllowance allowed;
  BT_CHECK(allow_shared_memory(allowed, kern, smem), "linear_split: cannot reserve %zu bytes of shared memory", smem);
  const long long n_tiles = (long long)((p.N + LS_BN - 1) / LS_BN) * ((p.M + LS_BM - 1) / LS_BM);
  const int sms = sm_count();
  BT_CHECK(sms > 0 && n_tiles <= 0x7fffffffll / 8 - sms, "linear_split: sizes M=%d N=%d are not supported", p.M, p.N);
  const long long blocks = SPLIT > 1 ? n_tiles * SPLIT : (n_tiles < sms ? n_tiles : sms);      // (a cluster takes one tile)
  BT_PDL_OK("linear_split", launch_pdl(kern, dim3((unsigned)blocks), dim3(LS_THREADS), smem, stream, SPLIT, p));
  return 0;
}

}  // namespace bt

// Which weights take this kernel, whatever the rows (a row's result must not depend on how many there are): those whose K is long
// enough beside N for a cluster to share it, so that few rows fill the GPU as well as many.  Against linear_simt.cu, us at 1 / 130 / 804
// rows: 768 x 768 8.3 / 12.0 / 33.8 and 7.3 / 10.2 / 25.5; 768 x 3072 28 / 41 / 126 and 12 / 22 / 68; 1024 x 4096 36 / 48 / 180 and 23 / 28 /
// 105; 1600 x 6400 56 / 118 / 448 and 33 / 76 / 269; 256 x 768 8.3 / 8.7 / 14.5 and 6.4 / 7.5 / 10.6.  Not 512 x 512 (6.1 / 6.5 / 16 and
// 6.5 / 8.4 / 13), nor wide ones: 2304 x 768 8.2 / 21 / 80 and 13 / 16 / 48, and behind by more where the weights come from memory.
extern "C" int bt_linear_split_supports(int N, int K, int w_is_nk) {
  return K % 4 == 0 && (w_is_nk || N % 4 == 0) && N >= 256 && N <= 2048 && K >= 768 && K >= N;
}

// How many blocks share a tile (1, 2, 4 or 8) on a device of `sms` multiprocessors, by what the tiles take: a k-block 1.35 us, start and end
// 2.5, the exchange 1.5.  Of 4 blocks 32 clusters are resident together on 148 multiprocessors, of 8 blocks 14; a device with too few for
// any by that measure does without.  (Any answer gives the same bits.)
extern "C" int bt_linear_split_blocks(int M, int N, int K, int sms) {
  using namespace bt;
  const long long tiles = (long long)((M + LS_BM - 1) / LS_BM) * ((N + LS_BN - 1) / LS_BN), k_blocks = (K + TC_BK - 1) / TC_BK;
  long long best = -1;
  int split = 1;
  for (const int s : {1, 2, 4, 8}) {
    const long long places = s <= 2 ? sms / s : s == 4 ? sms / 4 - 5 : sms / 8 - 4;
    if (places < 1) continue;
    const long long rounds = (tiles + places - 1) / places;
    const long long cost = 2500 + (s > 1 ? 1500 : 0) + rounds * ((k_blocks + s - 1) / s * 1350 + (s > 1 && rounds > 1 ? 3000 : 0));
    if (best < 0 || cost < best) {
      best = cost;
      split = s;
    }
  }
  return split;
}

// All operands 32-bit, A and W on 16-byte boundaries with rows of such pieces (K, and N of a [K,N] weight, multiples of 4).
// split: 0 by the sizes; 1, 2, 4 or 8 blocks a tile.
extern "C" int bt_linear_split(const float* a, const float* w, const float* bias, const float* residual, float* out, int* status, int M,
                               int N, int K, int w_is_nk, int act, int split, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(M >= 0 && N > 0 && K > 0 && K % 4 == 0 && (w_is_nk || N % 4 == 0) && ((unsigned long long)a | (unsigned long long)w) % 16 == 0,
           "linear_split: sizes or addresses that are not supported (M=%d N=%d K=%d)", M, N, K);
  BT_CHECK(act >= 0 && act <= 2, "linear_split: unknown activation %d", act);
  BT_CHECK(split == 0 || split == 1 || split == 2 || split == 4 || split == 8, "linear_split: %d blocks a tile", split);
  if (M == 0) return 0;
  const int rows16 = N % 4 == 0 && ((unsigned long long)out | (unsigned long long)residual | (unsigned long long)bias) % 16 == 0;
  const SplitParams p{a, w, bias, residual, out, status, M, N, K, act, rows16};
  if (split == 0) {
    const int sms = sm_count();
    BT_CHECK(sms > 0, "linear_split: cannot read the number of multiprocessors of the current device");
    split = bt_linear_split_blocks(M, N, K, sms);
  }
  if (split == 8) return w_is_nk ? launch_split<true, 8>(p, stream) : launch_split<false, 8>(p, stream);
  if (split == 2) return w_is_nk ? launch_split<true, 2>(p, stream) : launch_split<false, 2>(p, stream);
  if (split == 4) return w_is_nk ? launch_split<true, 4>(p, stream) : launch_split<false, 4>(p, stream);
  return w_is_nk ? launch_split<true, 1>(p, stream) : launch_split<false, 1>(p, stream);
}
