// Matrix products for steps with many rows (prefill), bfloat16 operands, 32-bit accumulation, on the
// fifth-generation tensor cores:  out[M,N] = act(A[M,K] @ W[N,K]^T + bias) (+ residual).
//
// A block computes 128 x BN tiles of the output, one after another (one block per SM).  Its ten warps have fixed jobs:
//   warp 0    asks the tensor memory accelerator (TMA) for the next 128 x 64 tile of A and BN x 64 tile of W
//             (cp.async.bulk.tensor, 128-byte swizzle) into a ring of shared-memory stages;
//   warp 1    one elected thread issues tcgen05.mma (M = 128, or 256 for a pair, N = BN, K = 16, four per stage) whose accumulator
//             lives in tensor memory (TMEM), and commits each stage back to the producer when it has been read;
//   warps 2-9 wait for a tile's last commit and read the accumulator with tcgen05.ld (a warp reaches the 32 TMEM lanes
//             of its quarter; the two warps of a quarter take half of the columns each).  A thread then holds 32
//             consecutive columns of one row: it adds the bias, applies GELU and writes the segment with 16-byte
//             stores (bfloat16 or 32-bit); with a 32-bit residual the warp first turns its patch through shared
//             memory, so that four lanes read and write 64 contiguous bytes of a row.  There are two
//             accumulators, so this runs while the next tile's products are already being issued.
// What bounds the loop is the issuer at narrow tiles (0.25 us a k-block alone, 0.17 in a pair, up to 128 columns), the tensor
// cores at wide ones, and for large calls what the whole GPU takes in from L2 and its power.  So two neighbouring blocks (a
// cluster) may work on one tile of 256 x BN as a PAIR: each loads its own 128 rows of A and half of W's rows, and the tensor
// cores of both read both halves of W (cta_group::2, issued by the pair's first block).  A block then takes in 16 KB + BN x
// 64 bytes a k-block for the same products as 16 KB + BN x 128 alone.
// Both operands are K-major (K contiguous): A as the activations are stored, W as [N, K].
// The kernel is launched as a programmatic dependent: it sets itself up (barriers, tensor memory) and asks for its
// first tiles of W while its predecessor still runs, and waits for it only before it touches activations.
// Stages hand over through mbarriers; every wait is bounded, and a wait that runs out marks the call as failed
// (status word) instead of hanging: the block still frees its tensor memory and returns.
// Rows and columns beyond M, N, K are zero-filled by the TMA on the way in and skipped on the way out.
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace bt {

constexpr int TC_BM = 128;
constexpr int TC_EPI_WARPS = 8;                    // two per quarter of the accumulator's rows, half the columns each
constexpr int TC_THREADS = (2 + TC_EPI_WARPS) * 32;
constexpr int TC_PATCH_STRIDE = 20;       // floats between rows of an epilogue warp's 32 x 16 patch in shared memory

struct TcParams {
  const float* bias;        // [N] or null
  const float* residual;    // [M, N] 32-bit or null (may be `out`)
  void* out;                // [M, N] 32-bit or bfloat16
  int* status;              // set to 1 when a bounded wait ran out
  int M, N, K, act, out_is_f32;
  // head_cols > 0 (bfloat16 results only): column c of row r goes to out[(c / head_cols) * head_stride + r * out_row + c % head_cols]
  int head_cols;
  long long out_row, head_stride;
  int band;                 // tiles of rows that go over all columns before the next rows are begun (at least 1)
  // a gated product (bfloat16 results of N / 2 columns): W's first N / 2 rows are the gate's, the others up's
  float limit;
};


// A warp's 32 rows of 32 numbers as bfloat16: a thread's 64-byte row goes into the patch (rows 80 bytes apart: no bank conflicts),
// then lane 4 r + c writes 16 bytes of rows r, r + 8, r + 16, r + 24: four lanes cover a row's 64 bytes, an instruction 8 lines
// instead of 32.  dst: the first column of row 0; rows from row0 on, up to `rows`, are written.
__device__ __forceinline__ void tc_store32(unsigned char* patch, int stride, const float (&v)[32], int lane, __nv_bfloat16* dst,
                                           long long row_stride, int row0, int rows) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4 x;
    x.x = tc_pack(v[8 * j], v[8 * j + 1]);
    x.y = tc_pack(v[8 * j + 2], v[8 * j + 3]);
    x.z = tc_pack(v[8 * j + 4], v[8 * j + 5]);
    x.w = tc_pack(v[8 * j + 6], v[8 * j + 7]);
    *reinterpret_cast<uint4*>(patch + lane * stride + 16 * j) = x;
  }
  __syncwarp();
  const int cq = lane & 3, rq = lane >> 2;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = rq + 8 * k;
    const uint4 x = *reinterpret_cast<const uint4*>(patch + r * stride + 16 * cq);
    if (row0 + r < rows) *reinterpret_cast<uint4*>(dst + (long long)(row0 + r) * row_stride + 8 * cq) = x;
  }
  __syncwarp();      // the patch is free again
}

// Persistent: a block walks over output tiles (tile, tile + grid, ...).  The accumulator is double-buffered in
// tensor memory (2 x BN columns), so the epilogue of one tile runs while the products of the next are issued.
// Shared memory: STAGES x (A tile 128 x 64, W tile BN x 64), each tile 1024-byte aligned, then a 32 x 20 float
// patch per epilogue warp through which accumulator rows are turned into coalesced global rows.
// GATED: half of a tile's BN rows of W are the gate's and half up's, of the same BN / 2 columns of the result (each block of a
// pair loads one of the halves), so that the epilogue has both numbers of a result and writes rule(gate) * up: the rows of 2 N
// numbers between the product and an activation kernel, written and read again, are gone.  2,048 rows of 5,632 x 1,024
// and the activation in a recorded layer: 20 and 12 us as two kernels, 25 as one.
template <int BN, int STAGES, bool PAIR, bool GATED>
__global__ void __launch_bounds__(TC_THREADS)
linear_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, TcParams p) {
  extern __shared__ unsigned char tc_smem_raw[];
  __shared__ __align__(8) unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  __shared__ unsigned tmem_base;
  __shared__ int failed;
  constexpr int W_ROWS = PAIR ? BN / 2 : BN;           // of W that this block loads
  constexpr unsigned A_BYTES = TC_BM * TC_BK * 2, W_BYTES = W_ROWS * TC_BK * 2;
  constexpr unsigned STAGE_BYTES = (A_BYTES + W_BYTES) * (PAIR ? 2 : 1);      // what a stage's barrier counts
  constexpr int BM = PAIR ? 2 * TC_BM : TC_BM;          // rows of a tile
  // columns of tensor memory from one accumulator to the other: a power of two, as the allocation has to be
  constexpr int ACC = BN <= 64 ? 64 : (BN <= 128 ? 128 : 256);
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<unsigned long long>(tc_smem_raw) + 1023ull) & ~1023ull);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (uniform for the compiler too)
  pdl_trigger();     // the next kernel may set itself up (and fetch its weights) while this one runs
  const int rank = PAIR ? (int)tc_rank() : 0;           // (the pair's first block is 0)
  const int tile0 = (int)blockIdx.x / (PAIR ? 2 : 1), tile_step = (int)gridDim.x / (PAIR ? 2 : 1);
  const int tiles_m = (p.M + BM - 1) / BM, tiles_n = (p.N + BN - 1) / BN;
  const int n_tiles = tiles_m * tiles_n;
  const int k_blocks = (p.K + TC_BK - 1) / TC_BK;
  // the first row of W that this block loads for the tn-th tile of columns, of half `h` where it loads two
  auto w_row = [&](int tn, int h) {
    if constexpr (GATED) return tn * (BN / 2) + (PAIR ? rank : h) * (p.N / 2);
    else return tn * BN + rank * W_ROWS;
  };
  // Where a tile lies: bands of `band` tiles of rows, a band's rows first, then its columns (the band's A comes from L2 then)
  auto place = [&](int tile, int& tm, int& tn) {
    const int b = tile / (p.band * tiles_n), first = b * p.band, in_band = tile - first * tiles_n;
    const int rows = min(p.band, tiles_m - first);
    tn = in_band / rows;
    tm = first + in_band - tn * rows;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc_bar_init(&full[s], 1);
      tc_bar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc_bar_init(&acc_full[b], 1);
      tc_bar_init(&acc_empty[b], TC_EPI_WARPS * (PAIR ? 2 : 1));       // one arrival per epilogue warp (of both blocks)
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    // two accumulators of BN 32-bit columns each (the count is a power of two of at least 32)
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&tmem_base)), "r"(2 * ACC) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&tmem_base)), "r"(2 * ACC) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) tc_cluster_sync();      // (the other block's barriers are set up as well)
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_acc = tmem_base;

  if (warp == 0) {
    if (tc_elect()) {
      // The first stages' tiles of W are asked for before the kernel waits for its predecessor (programmatic dependent
      // launch): nothing of a step writes weights, so they travel while the previous kernel finishes.  Their tiles
      // of A follow after the wait.
      const int pre = tile0 < n_tiles ? (k_blocks < STAGES ? k_blocks : STAGES) : 0;
      auto expect = [&](int s) {
        if (rank == 0) tc_bar_expect(&full[s], STAGE_BYTES);      // (a pair's copies all count on its first block's barrier)
      };
      auto load = [&](int s, bool weights, int kb, int row) {
        unsigned char* dst = tiles + (size_t)s * (A_BYTES + W_BYTES) + (weights ? A_BYTES : 0);
        if constexpr (PAIR) tc_tma_load_pair(dst, weights ? &map_w : &map_a, kb * TC_BK, row, tc_first_block(&full[s]));
        else tc_tma_load(dst, weights ? &map_w : &map_a, kb * TC_BK, row, &full[s]);
      };
      auto load_w = [&](int s, int kb, int tn) {
        load(s, true, kb, w_row(tn, 0));
        if constexpr (GATED && !PAIR)
          tc_tma_load(tiles + (size_t)s * (A_BYTES + W_BYTES) + A_BYTES + W_BYTES / 2, &map_w, kb * TC_BK, w_row(tn, 1), &full[s]);
      };
      {
        int tm = 0, tn = 0;
        place(tile0, tm, tn);
        const int m0 = tm * BM + rank * TC_BM;
        for (int kb = 0; kb < pre; ++kb) {
          expect(kb);
          load_w(kb, kb, tn);
        }
        pdl_wait();
        for (int kb = 0; kb < pre; ++kb) load(kb, false, kb, m0);
      }
      // the ring: stage `s`, waited for with the parity of its round (the first round's stages are free)
      int kb = pre, s = pre == STAGES ? 0 : pre;
      unsigned parity = pre == STAGES ? 0u : 1u;      // (of the round before: a fresh barrier's is complete)
      for (int tile = tile0; tile < n_tiles; tile += tile_step, kb = 0) {
        int tm, tn;
        place(tile, tm, tn);
        const int m0 = tm * BM + rank * TC_BM;
        for (; kb < k_blocks; ++kb) {
          if (!tc_bar_wait(&empty[s], parity)) {
            failed = 1;
            tile = n_tiles;
            break;
          }
          expect(s);
          load(s, false, kb, m0);
          load_w(s, kb, tn);
          if (++s == STAGES) {
            s = 0;
            parity ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // (the whole warp walks the ring and one elected lane issues, so that the operands stay in uniform registers: walked by
    // the lane whose number is 0, a k-block cost the issuer 0.34 us whatever its width, and that bounded the loop)
    if (rank == 0) {
      // instruction descriptor: 32-bit accumulator, bfloat16 operands, both K-major, N = BN, M = 128 (256 for a pair)
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
      int s = 0, local = 0;
      unsigned parity = 0;
      bool ok = true;
      for (int tile = tile0; tile < n_tiles && ok; tile += tile_step, ++local) {
        const int buf = local & 1;
        // the epilogue must have emptied this accumulator (it was last used two tiles ago)
        // (a wait that runs out must not part the warp's lanes)
        if (!__all_sync(0xffffffffu, local < 2 || tc_bar_wait(&acc_empty[buf], ((local >> 1) - 1) & 1))) {
          failed = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned d_tmem = tmem_acc + (unsigned)(buf * ACC);
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!__all_sync(0xffffffffu, tc_bar_wait(&full[s], parity))) {
            failed = 1;
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          if (tc_elect()) {
            unsigned char* a_tile = tiles + (size_t)s * (A_BYTES + W_BYTES);
            const unsigned long long da = tc_desc(a_tile), dw = tc_desc(a_tile + A_BYTES);
#pragma unroll
            for (int k = 0; k < TC_BK / 16; ++k) { // 16 bfloat16 = 32 bytes further along the row: +2 in 16-byte units
              const unsigned more = (kb > 0 || k > 0) ? 1u : 0u;
              if constexpr (PAIR) tc_mma_pair(d_tmem, da + 2ull * k, dw + 2ull * k, idesc, more);
              else tc_mma(d_tmem, da + 2ull * k, dw + 2ull * k, idesc, more);
            }
            // arrives when these products have read the stage (in both blocks of a pair)
            if constexpr (PAIR) tc_commit_pair(&empty[s]);
            else tc_commit(&empty[s]);
            // and, behind a tile's last ones, when every product issued so far has finished
            if (kb + 1 == k_blocks) {
              if constexpr (PAIR) tc_commit_pair(&acc_full[buf]);
              else tc_commit(&acc_full[buf]);
            }
          }
          __syncwarp();
          if (++s == STAGES) {
            s = 0;
            parity ^= 1u;
          }
        }
      }
    }
  } else {
    // epilogue: warp w reaches TMEM lanes 32 * (w % 4) .. + 31, i.e. the tile's rows of that quarter; the two warps
    // of a quarter take half of the tile's columns each.  A thread holds 32 consecutive columns of its row: bias,
    // activation and residual are applied there and the row segment is written with 16-byte stores.
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float* patch = reinterpret_cast<float*>(tiles + (size_t)STAGES * (A_BYTES + W_BYTES)) + (warp - 2) * (32 * TC_PATCH_STRIDE);
    // a tile's bias is on its way while the products run (the first tile's while the previous kernel does): a thread asks for it in every
    // chunk of 32 columns, and each time waited for L2, or for memory.  Layers of GPT-2, cold: 2 x 1,024 tokens (small) 84.0 to 81.9
    // us, 8 portions of 129 (medium) 85.5 to 84.2, 64 sequences' decode (XL) 85.8 to 84.9
    auto bias_ahead = [&](int tn) {
      const int col = tn * BN + lane * 32;
      if (p.bias != nullptr && lane * 32 < BN && col < p.N) asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p.bias + col));
    };
    if (tile0 < n_tiles) {
      int tm, tn;
      place(tile0, tm, tn);
      bias_ahead(tn);
    }
    pdl_wait();      // the residual is read and the output written only when the previous kernel has finished
    const bool vec_ok = p.out_is_f32 ? (p.N % 4 == 0) : (p.N % 8 == 0);
    int local = 0;
    for (int tile = tile0; tile < n_tiles; tile += tile_step, ++local) {
      const int buf = local & 1;
      int tm, tn;
      place(tile, tm, tn);
      if (local > 0) bias_ahead(tn);
      const int m0 = tm * BM + rank * TC_BM, n0 = tn * BN;
      if (!__all_sync(0xffffffffu, tc_bar_wait(&acc_full[buf], (local >> 1) & 1))) {      // (what follows is collective)
        failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int row = m0 + quarter * 32 + lane;
      const bool row_ok = row < p.M;
      // (the first warp of a quarter takes the larger part when the 32-column chunks are an odd number)
      constexpr int COLS = GATED ? BN / 2 : BN;      // of the result
      constexpr int SPLIT = (COLS / 32 + 1) / 2 * 32;
#pragma unroll 1
      for (int c0 = half ? SPLIT : 0; c0 < (half ? COLS : SPLIT); c0 += 32) {
        float v[32];
        tc_ld32(tmem_acc + ((unsigned)(quarter * 32) << 16) + (unsigned)(buf * ACC + c0), v);
        if constexpr (GATED) {
          float up[32];
          tc_ld32(tmem_acc + ((unsigned)(quarter * 32) << 16) + (unsigned)(buf * ACC + COLS + c0), up);
          const int cols = p.N / 2, col0 = tn * COLS + c0;
          if (col0 >= cols) continue;
          if (p.act == kActSwish) tc_gated_all<kActSwish>(v, up, p.limit);
          else if (p.act == kActSwishClamp) tc_gated_all<kActSwishClamp>(v, up, p.limit);
          else if (p.act == kActGeluTanh) tc_gated_all<kActGeluTanh>(v, up, p.limit);
          else tc_gated_all<kActGeluErf>(v, up, p.limit);
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out);
          if (cols % 8 == 0 && col0 + 32 <= cols) {
            tc_store32(reinterpret_cast<unsigned char*>(patch), TC_PATCH_STRIDE * 4, v, lane, out + col0, cols, m0 + quarter * 32, p.M);
          } else if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (col0 + i < cols) out[(long long)row * cols + col0 + i] = __float2bfloat16_rn(v[i]);
          }
          continue;
        }
        const int col0 = n0 + c0;
        if (col0 >= p.N) continue;                 // (uniform in the warp; the load above is collective)
        const long long o0 = (long long)row * p.N + col0;
        if (vec_ok && col0 + 32 <= p.N && p.residual != nullptr) {
          // 32-bit output with a residual (the residual stream itself, as a rule): the warp's patch goes through
          // shared memory, 16 columns at a time, so that global memory is reached row by row: a thread writes its
          // row (rows 20 floats apart: no bank conflicts for 16-byte accesses), then lane 4 r + c takes columns
          // 4 c .. 4 c + 3 of rows r, r + 8, ..., so that four lanes cover 64 contiguous bytes of a row of the
          // residual and of the output.  (With a lane per row every instruction touches 32 lines, and the
          // load/store unit takes them one by one: 1.8 us per 32 columns each way.)
          const int cq = lane & 3, rq = lane >> 2;
          const int row_base = m0 + quarter * 32 + rq;
#pragma unroll
          for (int h16 = 0; h16 < 2; ++h16) {
            const long long o_base = (long long)row_base * p.N + col0 + 16 * h16 + 4 * cq;
            float4 res[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (row_base + 8 * k < p.M) res[k] = *reinterpret_cast<const float4*>(p.residual + o_base + (long long)(8 * k) * p.N);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<float4*>(patch + lane * TC_PATCH_STRIDE + 4 * j) =
                  make_float4(v[16 * h16 + 4 * j], v[16 * h16 + 4 * j + 1], v[16 * h16 + 4 * j + 2], v[16 * h16 + 4 * j + 3]);
            __syncwarp();
            float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (p.bias) b4 = __ldg(reinterpret_cast<const float4*>(p.bias + col0 + 16 * h16 + 4 * cq));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float4 x = *reinterpret_cast<const float4*>(patch + (rq + 8 * k) * TC_PATCH_STRIDE + 4 * cq);
              x.x = tc_activation(x.x + b4.x, p.act, true) + res[k].x;
              x.y = tc_activation(x.y + b4.y, p.act, true) + res[k].y;
              x.z = tc_activation(x.z + b4.z, p.act, true) + res[k].z;
              x.w = tc_activation(x.w + b4.w, p.act, true) + res[k].w;
              if (row_base + 8 * k < p.M) *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + o_base + (long long)(8 * k) * p.N) = x;
            }
            __syncwarp();      // the patch is free again
          }
        } else if (vec_ok && col0 + 32 <= p.N) {
          float4 res[8];
          if (p.residual && row_ok) {
            // the whole segment of the residual first, so that the latencies overlap (the output may be the
            // residual itself, which keeps the compiler from moving these loads above the stores on its own)
#pragma unroll
            for (int j = 0; j < 8; ++j) res[j] = *reinterpret_cast<const float4*>(p.residual + o0 + 4 * j);
          }
          if (p.bias) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 b4 = __ldg(reinterpret_cast<const float4*>(p.bias + col0 + 4 * j));
              v[4 * j] += b4.x; v[4 * j + 1] += b4.y; v[4 * j + 2] += b4.z; v[4 * j + 3] += b4.w;
            }
          }
          const bool exact = p.residual != nullptr || p.out_is_f32 != 0;
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = tc_activation(v[i], p.act, exact);
          if (p.out_is_f32) {
            if (!row_ok) continue;
            float* dst = reinterpret_cast<float*>(p.out) + o0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float4 x = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
              if (p.residual) { x.x += res[j].x; x.y += res[j].y; x.z += res[j].z; x.w += res[j].w; }
              *reinterpret_cast<float4*>(dst + 4 * j) = x;
            }
          } else {
            // (a chunk of 32 columns lies in one head)
            const int head = p.head_cols > 0 ? col0 / p.head_cols : 0;
            tc_store32(reinterpret_cast<unsigned char*>(patch), TC_PATCH_STRIDE * 4, v, lane,
                       reinterpret_cast<__nv_bfloat16*>(p.out) + head * p.head_stride + (col0 - head * p.head_cols), p.out_row,
                       m0 + quarter * 32, p.M);
          }
        } else if (row_ok) {
          // a ragged edge, or rows that are no multiple of 16 bytes: one element at a time
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (col0 + i >= p.N) break;
            float x = tc_activation(v[i] + (p.bias ? p.bias[col0 + i] : 0.f), p.act, p.residual != nullptr || p.out_is_f32 != 0);
            if (p.residual) x += p.residual[o0 + i];
            if (p.out_is_f32)
              reinterpret_cast<float*>(p.out)[o0 + i] = x;
            else
              reinterpret_cast<__nv_bfloat16*>(p.out)[o0 + i] = __float2bfloat16_rn(x);
          }
        }
      }
      // this warp has read its part of the accumulator: hand the buffer back to the issuer
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) tc_bar_arrive_at(tc_first_block(&acc_empty[buf]));
        else tc_bar_arrive(&acc_empty[buf]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (failed) let_copies_land();
  if constexpr (PAIR) tc_cluster_sync();      // neither block's memory or barriers are touched by the other from here on
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_acc), "r"(2 * ACC) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_acc), "r"(2 * ACC) : "memory");
  }
  if (threadIdx.x == 0 && failed && p.status) atomicExch(p.status, 2);
}

// A tile's shape, what a call costs beside its k-blocks (start, and the last tile's way out) and what a k-block costs, in ns,
// measured at 1,024 and 2,048 rows with K from 768 to 4,096.  Against the version without pairs, whose issuer a single lane
// walked (us a call, GPT-2's products with bias, GELU or residual): 2,048 rows: 768 x 3072 23.0 to 15.4, 768 x 768 10.2 to
// 8.9, 2304 x 768 11.4 to 10.9, 3072 x 768 14.9 to 13.4; 1024 x 4096 30.3 to 19.0; 16,384 rows: 6400 x 1600 262 to 222,
// 1600 x 6400 364 to 314, 4800 x 1600 201 to 177.
struct TcTile {
  int bn;
  bool pair;
  int once_ns, k_block_ns;
};
constexpr long long TC_BAND = 16ll << 20;
constexpr TcTile TC_TILES[] = {{256, false, 8900, 296}, {192, false, 7600, 265}, {128, false, 6400, 245}, {96, false, 5800, 250},
                               {64, false, 5200, 233}, {256, true, 9400, 294}, {224, true, 8900, 260}, {192, true, 8400, 217},
                               {160, true, 7900, 196}, {128, true, 7400, 170}, {96, true, 6900, 167}, {64, true, 6400, 163}};

template <int BN, int STAGES, bool PAIR, bool GATED = false>
static int launch_tc(const CUtensorMap& ma, const CUtensorMap& mw, const TcParams& p, cudaStream_t stream) {
  constexpr size_t smem = (size_t)STAGES * (TC_BM * TC_BK * 2 + (PAIR ? BN / 2 : BN) * TC_BK * 2) + 1024 + (size_t)TC_EPI_WARPS * 32 * TC_PATCH_STRIDE * 4;
  static_assert(smem <= 227 * 1024, "a multiprocessor's shared memory");
  auto kern = linear_tcgen05_kernel<BN, STAGES, PAIR, GATED>;
  static SharedMemoryAllowance allowed;
  BT_CHECK(allow_shared_memory(allowed, kern, smem), "linear_tcgen05: cannot reserve %zu bytes of shared memory", smem);
  constexpr int GROUP = PAIR ? 2 : 1;
  const int n_tiles = ((p.N + BN - 1) / BN) * ((p.M + GROUP * TC_BM - 1) / (GROUP * TC_BM));
  const int groups = sm_count() / GROUP;
  BT_CHECK(groups > 0, "linear_tcgen05: cannot read the number of multiprocessors of the current device");
  const int blocks = (n_tiles < groups ? n_tiles : groups) * GROUP;     // one persistent block per SM
  BT_PDL_OK("linear_tcgen05", launch_pdl(kern, dim3(blocks), dim3(TC_THREADS), smem, stream, GROUP, ma, mw, p));
  return 0;
}

}  // namespace bt

extern "C" int bt_linear_tcgen05_supports(int M, int N, int K) {
  return M >= 1 && N >= 8 && K >= 8 && K % 8 == 0;   // rows of A and W are 16-byte multiples
}

static int run_linear_tcgen05(const void* a, long long a_row, const void* w, bt::TcParams p, bool gated, cudaStream_t stream) {
  using namespace bt;
  const int M = p.M, N = p.N, K = p.K;
  // The tile: wide ones reuse every loaded row of A for more columns, narrow ones cover the GPU with fewer idle
  // multiprocessors and fewer rounds; a pair takes in less and issues more products at once, a single block starts and ends
  // sooner.  The least of (start and end + rounds of tiles x (k-blocks x their time + 0.4 us)) decides.
  const int sms = sm_count();
  BT_CHECK(sms > 1, "linear_tcgen05: cannot read the number of multiprocessors of the current device");
  int bn = 256;
  bool pair = false;
  long long best = -1;
  const int k_blocks = (K + TC_BK - 1) / TC_BK;
  for (const TcTile& t : TC_TILES) {
    if (gated && t.bn % 64 != 0) continue;      // (half of the tile's columns are whole chunks of the epilogue)
    const long long rows = t.pair ? 2 * TC_BM : TC_BM, groups = t.pair ? sms / 2 : sms;
    const long long tiles = ((M + rows - 1) / rows) * ((N + t.bn - 1) / t.bn), rounds = (tiles + groups - 1) / groups;
    // (more than three rounds: the whole GPU takes in no more than about 85 GB/s a multiprocessor)
    const int taken_in = (TC_BM + (t.pair ? t.bn / 2 : t.bn)) * TC_BK * 2 / 85;
    const long long per_block = rounds > 3 && taken_in > t.k_block_ns ? taken_in : t.k_block_ns;
    const long long cost = t.once_ns + rounds * (k_blocks * per_block + 400);
    if (best < 0 || cost < best) {
      best = cost;
      bn = t.bn;
      pair = t.pair;
    }
  }
  // Tiles of rows whose A is at most TC_BAND bytes go over all columns before the next rows are begun: with all rows first,
  // an A beyond L2 (or in L2 beside a residual that streams through it) came from memory again for every tile of columns.
  // GPT-2 XL's layer at 16 x 1,024 tokens 1,270 to 1,176 us with bands of 16 MB, about 1,200 with 40; no sum changes.
  const long long tile_rows = pair ? 2 * TC_BM : TC_BM, tiles_m = (M + tile_rows - 1) / tile_rows;
  const long long band = TC_BAND / (tile_rows * K * 2);
  p.band = (int)(band < 1 ? 1 : (band < tiles_m ? band : tiles_m));
  CUtensorMap ma, mw;
  if (int rc = tensor_map_2d_bf16(&ma, a, (unsigned long long)M, (unsigned long long)K, (unsigned long long)a_row, TC_BM)) return rc;
  if (int rc = tensor_map_2d_bf16(&mw, w, (unsigned long long)N, (unsigned long long)K, (unsigned long long)K, (unsigned)(pair || gated ? bn / 2 : bn))) return rc;
  if (gated && pair) {
    if (bn == 64) return launch_tc<64, 8, true, true>(ma, mw, p, stream);
    if (bn == 128) return launch_tc<128, 8, true, true>(ma, mw, p, stream);
    if (bn == 192) return launch_tc<192, 7, true, true>(ma, mw, p, stream);
    return launch_tc<256, 6, true, true>(ma, mw, p, stream);
  }
  if (gated) {
    if (bn == 64) return launch_tc<64, 8, false, true>(ma, mw, p, stream);
    if (bn == 128) return launch_tc<128, 6, false, true>(ma, mw, p, stream);
    if (bn == 192) return launch_tc<192, 5, false, true>(ma, mw, p, stream);
    return launch_tc<256, 4, false, true>(ma, mw, p, stream);
  }
  if (pair) {
    if (bn == 64) return launch_tc<64, 8, true>(ma, mw, p, stream);
    if (bn == 96) return launch_tc<96, 8, true>(ma, mw, p, stream);
    if (bn == 128) return launch_tc<128, 8, true>(ma, mw, p, stream);
    if (bn == 160) return launch_tc<160, 7, true>(ma, mw, p, stream);
    if (bn == 192) return launch_tc<192, 7, true>(ma, mw, p, stream);
    if (bn == 224) return launch_tc<224, 6, true>(ma, mw, p, stream);
    return launch_tc<256, 6, true>(ma, mw, p, stream);
  }
  if (bn == 64) return launch_tc<64, 8, false>(ma, mw, p, stream);
  if (bn == 96) return launch_tc<96, 7, false>(ma, mw, p, stream);
  if (bn == 128) return launch_tc<128, 6, false>(ma, mw, p, stream);
  if (bn == 192) return launch_tc<192, 5, false>(ma, mw, p, stream);
  return launch_tc<256, 4, false>(ma, mw, p, stream);
}

// a: [M, K] bfloat16; w: [N, K] bfloat16; out: [M, N] 32-bit (out_is_f32) or bfloat16.
extern "C" int bt_linear_tcgen05(const void* a, const void* w, const float* bias, const float* residual, void* out,
                                 int* status, int M, int N, int K, int act, int out_is_f32, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(bt_linear_tcgen05_supports(M, N, K), "linear_tcgen05: sizes M=%d N=%d K=%d are not supported", M, N, K);
  BT_CHECK(act >= 0 && act <= 2, "linear_tcgen05: unknown activation %d", act);
  BT_CHECK(!(residual && !out_is_f32), "linear_tcgen05: a residual needs a 32-bit output");
  return run_linear_tcgen05(a, K, w, TcParams{bias, residual, out, status, M, N, K, act, out_is_f32, 0, N, 0}, false, stream);
}

// Per-head rows of one product: out[h][t][:] = a[t] @ w[h]^T for heads of N numbers (a multiple of 32), all bfloat16.
// a: [M, K], rows a_row elements apart; w: [heads * N, K]; out: rows out_row apart, heads head_stride.
extern "C" int bt_head_rows_tcgen05_supports(int M, int N, int K, long long a_row, long long out_row, long long head_stride) {
  return M >= 1 && N >= 32 && N % 32 == 0 && K >= 8 && K % 8 == 0 && a_row >= K && a_row % 8 == 0 && out_row % 8 == 0 && head_stride % 8 == 0;
}
extern "C" int bt_head_rows_tcgen05(const void* a, long long a_row, const void* w, void* out, long long out_row, long long head_stride,
                                    int* status, int M, int heads, int N, int K, cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(heads > 0 && bt_head_rows_tcgen05_supports(M, N, K, a_row, out_row, head_stride) &&
               ((unsigned long long)a | (unsigned long long)w | (unsigned long long)out) % 16 == 0,
           "head_rows_tcgen05: sizes or strides that are not supported (M=%d heads=%d N=%d K=%d)", M, heads, N, K);
  return run_linear_tcgen05(a, a_row, w, TcParams{nullptr, nullptr, out, status, M, heads * N, K, 0, 0, N, out_row, head_stride}, false, stream);
}

// out[M, inner] = rule(gate) * up (gated_pair of common.cuh), gate and up the halves of a[M, K] @ w[2 inner, K]^T, all bfloat16;
// both halves and the rule in 32 bits, the result rounded once.  act: an Activation; limit: kActSwishClamp's.
extern "C" int bt_gated_tcgen05_supports(int M, int inner, int K) {
  return M >= 1 && inner >= 8 && inner <= 0x3fffffff && K >= 8 && K % 8 == 0;
}
extern "C" int bt_gated_tcgen05(const void* a, const void* w, void* out, int* status, int M, int inner, int K, int act, float limit,
                                cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(bt_gated_tcgen05_supports(M, inner, K) && ((unsigned long long)a | (unsigned long long)w | (unsigned long long)out) % 16 == 0,
           "gated_tcgen05: sizes or addresses that are not supported (M=%d inner=%d K=%d)", M, inner, K);
  BT_CHECK(act >= kActGeluTanh && act <= kActSwish, "gated_tcgen05: unknown rule %d", act);
  return run_linear_tcgen05(a, K, w, TcParams{nullptr, nullptr, out, status, M, 2 * inner, K, act, 0, 0, inner, 0, 0, limit}, true, stream);
}
