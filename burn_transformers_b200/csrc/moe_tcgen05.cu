// The routed experts' products for many rows an expert (prompts), bfloat16, on the fifth-generation tensor cores: rows of
// `a` sorted by expert (bt_moe_sort; for the first product gathered by bt_moe_gather), each expert's rows times its weights.
//
// The blocks are linear_tcgen05.cu's, one a multiprocessor, with a tile of 128 rows of ONE expert by 128 rows of its weights
// (for experts with a gate 64 of the gate's and the 64 of the up's beside them, so that both numbers of a pair lie in one
// accumulator): warp 0 copies by TMA into a ring of six stages, warp 1 walks the ring and an elected lane issues tcgen05.mma,
// warps 2-9 take one of two accumulators out of tensor memory (pair rule, activation or the pair's weight) while the next
// tile's products run.  How many tiles there are only the device knows: every block counts them from the experts' offsets.
// A tile's rows past its expert's last one are the next expert's: computed and not stored.
// 8,192 pairs over 16 experts of 512 x 1,024, the most popular with four times the mean (us, first / second product): 110 / 79
// with mma.sync on 32 x 64 tiles (moe.cu), about 33 / 30 here and 8 for the gathered rows (in a recorded layer, beside a
// recurrence's kernels).
#include "api.h"
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace bt {

constexpr int ME_BM = 128, ME_BN = 128;
constexpr int ME_STAGES = 6;
constexpr int ME_EPI_WARPS = 8;
constexpr int ME_THREADS = (2 + ME_EPI_WARPS) * 32;
constexpr int ME_PATCH = 20;                      // floats between rows of a warp's 32 x 16 patch
constexpr int ME_MAX_EXPERTS = 256;
constexpr unsigned ME_TILE_BYTES = ME_BM * TC_BK * 2;
constexpr size_t ME_SMEM = (size_t)ME_STAGES * 2 * ME_TILE_BYTES + 1024 + (size_t)ME_EPI_WARPS * 32 * ME_PATCH * 4;
constexpr int kMeOut = 0, kMePair = 1, kMePlain = 2;      // as in moe.cu

struct MeParams {
  const int* offsets;          // [E + 1]
  const int* order;            // kMeOut: the pair in each sorted row
  const float* pair_weight;    // kMeOut: [pairs]
  void* out;                   // [pairs, N]: 32-bit (kMeOut) or bfloat16
  int* status;
  int E, N, K, act;
  float limit;
};

template <int MODE>
__global__ void __launch_bounds__(ME_THREADS)
moe_expert_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, MeParams p) {
  constexpr bool PAIR = MODE == kMePair;
  constexpr int COLS = PAIR ? ME_BN / 2 : ME_BN;          // output columns of a tile
  extern __shared__ unsigned char me_raw[];
  __shared__ __align__(8) unsigned long long full[ME_STAGES], empty[ME_STAGES], acc_full[2], acc_empty[2];
  __shared__ unsigned tmem_base;
  __shared__ int failed;
  __shared__ int first_row[ME_MAX_EXPERTS + 1], first_tile[ME_MAX_EXPERTS + 1];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<unsigned long long>(me_raw) + 1023ull) & ~1023ull);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < ME_STAGES; ++s) {
      tc_bar_init(&full[s], 1);
      tc_bar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc_bar_init(&acc_full[b], 1);
      tc_bar_init(&acc_empty[b], ME_EPI_WARPS);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(&tmem_base)), "r"(2 * ME_BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  pdl_wait();      // (the sorting and the rows are results of the kernels before)
  for (int e = threadIdx.x; e <= p.E; e += ME_THREADS) first_row[e] = p.offsets[e];
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  if (warp == 0) {      // row tiles before each expert's first: a scan over the experts, 32 at a time
    int before = 0;
    for (int e0 = 0; e0 < p.E; e0 += 32) {
      const int e = e0 + lane;
      const int own = e < p.E ? (first_row[e + 1] - first_row[e] + ME_BM - 1) / ME_BM : 0;
      int sum = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += x;
      }
      if (e < p.E) first_tile[e] = before + sum - own;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) first_tile[p.E] = before;
  }
  __syncthreads();
  const unsigned tmem_acc = tmem_base;
  const int tiles_n = (p.N + COLS - 1) / COLS;
  const int n_tiles = first_tile[p.E] * tiles_n;
  const int k_blocks = (p.K + TC_BK - 1) / TC_BK;
  // which expert, which of the sorted rows (from row0 to row1) and which output columns tile `tile` is
  auto find = [&](int tile, int& expert, int& row0, int& row1, int& n0) {
    const int mt = tile / tiles_n;
    int lo = 0, hi = p.E - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first_tile[mid] <= mt) lo = mid; else hi = mid - 1;
    }
    expert = lo;
    row0 = first_row[lo] + (mt - first_tile[lo]) * ME_BM;
    row1 = min(row0 + ME_BM, first_row[lo + 1]);
    n0 = (tile - mt * tiles_n) * COLS;
  };

  if (warp == 0) {
    if (tc_elect()) {
      int s = 0;
      unsigned parity = 1;                // (of the round before: a fresh barrier's is complete)
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        int expert, row0, row1, n0;
        find(tile, expert, row0, row1, n0);
        const int w_row = expert * (PAIR ? 2 : 1) * p.N + n0;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!tc_bar_wait(&empty[s], parity)) {
            failed = 1;
            ok = false;
            break;
          }
          tc_bar_expect(&full[s], 2 * ME_TILE_BYTES);
          unsigned char* at = tiles + (size_t)s * 2 * ME_TILE_BYTES;
          // (boxes of 64 rows: 8 KB each)
          tc_tma_load(at, &map_a, kb * TC_BK, row0, &full[s]);
          tc_tma_load(at + ME_TILE_BYTES / 2, &map_a, kb * TC_BK, row0 + 64, &full[s]);
          tc_tma_load(at + ME_TILE_BYTES, &map_w, kb * TC_BK, w_row, &full[s]);
          tc_tma_load(at + ME_TILE_BYTES * 3 / 2, &map_w, kb * TC_BK, PAIR ? w_row + p.N : w_row + 64, &full[s]);
          if (++s == ME_STAGES) {
            s = 0;
            parity ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(ME_BN >> 3) << 17) | ((unsigned)(ME_BM >> 4) << 24);
    int s = 0, local = 0;
    unsigned parity = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++local) {
      const int buf = local & 1;
      // (a wait that runs out must not part the warp's lanes)
      if (!__all_sync(0xffffffffu, local < 2 || tc_bar_wait(&acc_empty[buf], ((local >> 1) - 1) & 1))) {
        failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const unsigned d_tmem = tmem_acc + (unsigned)(buf * ME_BN);
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!__all_sync(0xffffffffu, tc_bar_wait(&full[s], parity))) {
          failed = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (tc_elect()) {
          unsigned char* at = tiles + (size_t)s * 2 * ME_TILE_BYTES;
          const unsigned long long da = tc_desc(at), dw = tc_desc(at + ME_TILE_BYTES);
#pragma unroll
          for (int k = 0; k < TC_BK / 16; ++k) tc_mma(d_tmem, da + 2ull * k, dw + 2ull * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          tc_commit(&empty[s]);
          if (kb + 1 == k_blocks) tc_commit(&acc_full[buf]);
        }
        __syncwarp();
        if (++s == ME_STAGES) {
          s = 0;
          parity ^= 1u;
        }
      }
    }
  } else {
    // warp w reaches TMEM lanes 32 (w % 4) .. + 31; the two warps of a quarter take half of the output columns each
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float* patch = reinterpret_cast<float*>(tiles + (size_t)ME_STAGES * 2 * ME_TILE_BYTES) + (warp - 2) * (32 * ME_PATCH);
    const unsigned lanes = (unsigned)(quarter * 32) << 16;
    const bool vec = p.N % (MODE == kMeOut ? 4 : 8) == 0;
    int local = 0;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++local) {
      const int buf = local & 1;
      int expert, row0, row1, n0;
      find(tile, expert, row0, row1, n0);
      if (!__all_sync(0xffffffffu, tc_bar_wait(&acc_full[buf], (local >> 1) & 1))) {
        failed = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int first = row0 + quarter * 32;              // the warp's rows
      const bool row_ok = first + lane < row1;
      const float weight = MODE == kMeOut && row_ok ? p.pair_weight[p.order[first + lane]] : 1.f;
#pragma unroll 1
      for (int c0 = half * (COLS / 2); c0 < (half + 1) * (COLS / 2); c0 += 32) {
        float v[32];
        tc_ld32(tmem_acc + lanes + (unsigned)(buf * ME_BN + c0), v);
        if constexpr (PAIR) {
          float u[32];
          tc_ld32(tmem_acc + lanes + (unsigned)(buf * ME_BN + COLS + c0), u);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = gated_pair(v[i], u[i], p.act, p.limit);
        } else if constexpr (MODE == kMePlain) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = apply_activation(v[i], p.act);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] *= weight;
        }
        const int col0 = n0 + c0;
        if (col0 >= p.N) continue;                        // (uniform in the warp; the loads above are collective)
        if (vec && col0 + 32 <= p.N) {
          // through the patch, so that four lanes write 64 contiguous bytes of a row
          const int cq = lane & 3, rq = lane >> 2;
          if constexpr (MODE == kMeOut) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(patch + lane * ME_PATCH + 4 * j) =
                    make_float4(v[16 * h + 4 * j], v[16 * h + 4 * j + 1], v[16 * h + 4 * j + 2], v[16 * h + 4 * j + 3]);
              __syncwarp();
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int r = first + rq + 8 * k;
                if (r < row1)
                  *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (long long)r * p.N + col0 + 16 * h + 4 * cq) =
                      *reinterpret_cast<const float4*>(patch + (rq + 8 * k) * ME_PATCH + 4 * cq);
              }
              __syncwarp();
            }
          } else {
            unsigned char* patch8 = reinterpret_cast<unsigned char*>(patch);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 x;
              x.x = tc_pack(v[8 * j], v[8 * j + 1]);
              x.y = tc_pack(v[8 * j + 2], v[8 * j + 3]);
              x.z = tc_pack(v[8 * j + 4], v[8 * j + 5]);
              x.w = tc_pack(v[8 * j + 6], v[8 * j + 7]);
              *reinterpret_cast<uint4*>(patch8 + lane * (ME_PATCH * 4) + 16 * j) = x;
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int r = first + rq + 8 * k;
              const uint4 x = *reinterpret_cast<const uint4*>(patch8 + (rq + 8 * k) * (ME_PATCH * 4) + 16 * cq);
              if (r < row1) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (long long)r * p.N + col0 + 8 * cq) = x;
            }
            __syncwarp();
          }
        } else if (row_ok) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (col0 + i >= p.N) break;
            const long long o = (long long)(first + lane) * p.N + col0 + i;
            if constexpr (MODE == kMeOut) reinterpret_cast<float*>(p.out)[o] = v[i];
            else reinterpret_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(v[i]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_bar_arrive(&acc_empty[buf]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (failed) let_copies_land();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_acc), "r"(2 * ME_BN) : "memory");
  }
  if (threadIdx.x == 0 && failed && p.status) atomicExch(p.status, 8);
}

// out[r] = x[order[r] / top], 16 bytes a thread.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const uint4* __restrict__ x, long long row_pieces, const int* __restrict__ order, int top, uint4* __restrict__ out,
                  long long pieces, int per_row) {
  pdl_trigger();
  pdl_wait();
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < pieces; i += (long long)gridDim.x * 256) {
    const long long r = i / per_row;
    out[i] = __ldg(x + (long long)(order[r] / top) * row_pieces + (i - r * per_row));
  }
}

}  // namespace bt

extern "C" int bt_moe_expert_tcgen05_supports(int pairs, int E, int K, int N) {
  return pairs >= 1 && E >= 1 && E <= bt::ME_MAX_EXPERTS && K >= 8 && K % 8 == 0 && N >= 8;
}

// x: [tokens, K] bfloat16 (rows x_row_stride apart); out: [pairs, K]: the row of each sorted pair's token.
extern "C" int bt_moe_gather(const void* x, long long x_row_stride, const int* order, int top, void* out, int pairs, int K,
                             cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(pairs >= 0 && top > 0 && K > 0 && K % 8 == 0 && x_row_stride % 8 == 0 && ((unsigned long long)x | (unsigned long long)out) % 16 == 0,
           "moe_gather: rows must be whole 16-byte pieces (K=%d)", K);
  if (pairs == 0) return 0;
  const long long pieces = (long long)pairs * (K / 8);
  const long long blocks = (pieces + 255) / 256, most = 148 * 16;
  BT_PDL_OK("moe_gather", launch_pdl(moe_gather_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, stream, 1,
                                     (const uint4*)x, x_row_stride / 8, order, top, (uint4*)out, pieces, K / 8));
  return 0;
}

// mode as bt_moe_expert's `first`; a: [pairs, K] bfloat16, sorted by expert; the rest as bt_moe_expert.
extern "C" int bt_moe_expert_tcgen05(int mode, const void* a, const void* w, void* out, const int* offsets, const int* order,
                                     const float* pair_weight, int* status, int pairs, int E, int K, int N, int act, float limit,
                                     cudaStream_t stream) {
  using namespace bt;
  BT_CHECK(mode >= 0 && mode <= 2 && bt_moe_expert_tcgen05_supports(pairs, E, K, N),
           "moe_expert_tcgen05: sizes pairs=%d experts=%d K=%d N=%d are not supported", pairs, E, K, N);
  BT_CHECK(((unsigned long long)a | (unsigned long long)w | (unsigned long long)out) % 16 == 0,
           "moe_expert_tcgen05: operands must lie on 16-byte boundaries");
  const int sms = sm_count();
  BT_CHECK(sms > 0, "moe_expert_tcgen05: cannot read the number of multiprocessors of the current device");
  const unsigned long long w_rows = (unsigned long long)E * (mode == kMePair ? 2 : 1) * N;
  CUtensorMap ma, mw;
  if (int rc = tensor_map_2d_bf16(&ma, a, (unsigned long long)pairs, (unsigned long long)K, (unsigned long long)K, 64)) return rc;
  if (int rc = tensor_map_2d_bf16(&mw, w, w_rows, (unsigned long long)K, (unsigned long long)K, 64)) return rc;
  const MeParams p{offsets, order, pair_weight, out, status, E, N, K, act, limit};
  const int cols = mode == kMePair ? ME_BN / 2 : ME_BN;
  const long long most = ((long long)pairs / ME_BM + E) * ((N + cols - 1) / cols);      // no more tiles than this
  const int blocks = most < sms ? (int)most : sms;
  auto launch = [&](auto kern) -> int {
    BT_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ME_SMEM) == cudaSuccess,
             "moe_expert_tcgen05: cannot reserve %zu bytes of shared memory", ME_SMEM);
    BT_PDL_OK("moe_expert_tcgen05", launch_pdl(kern, dim3(blocks), dim3(ME_THREADS), ME_SMEM, stream, 1, ma, mw, p));
    return 0;
  };
  if (mode == kMePair) return launch(moe_expert_tcgen05_kernel<kMePair>);
  if (mode == kMePlain) return launch(moe_expert_tcgen05_kernel<kMePlain>);
  return launch(moe_expert_tcgen05_kernel<kMeOut>);
}
