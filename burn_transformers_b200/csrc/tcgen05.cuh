// Wrappers of the instructions that the tcgen05 matrix products share: mbarriers with bounded waits, tensor-map
// copies, shared-memory operand descriptors, tcgen05.mma / commit / ld, and the epilogue's activation.
#pragma once
#include "common.cuh"
#include "tma.cuh"

namespace bt {

constexpr int TC_BK = 64;                 // bfloat16 per stage row: 128 bytes, the swizzle span
constexpr int TC_WAIT_LIMIT = 1 << 22;    // polls of an mbarrier before giving up

__device__ __forceinline__ unsigned tc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void tc_bar_init(unsigned long long* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(tc_smem(bar)), "r"(count));
}
__device__ __forceinline__ void tc_bar_expect(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(tc_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tc_bar_wait(unsigned long long* bar, unsigned parity) {
  for (int i = 0; i < TC_WAIT_LIMIT; ++i) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(tc_smem(bar)), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void tc_tma_load(void* dst, const CUtensorMap* map, int col, int row, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          tc_smem(dst)),
      "l"(map), "r"(col), "r"(row), "r"(tc_smem(bar))
      : "memory");
}
// Shared-memory operand descriptor: K-major tile of 128-byte rows, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ unsigned long long tc_desc(const void* tile) {
  unsigned long long d = 0;
  d |= (unsigned long long)((tc_smem(tile) & 0x3FFFFu) >> 4);   // start address, 16-byte units
  d |= (unsigned long long)1 << 16;                             // leading byte offset (unused with this swizzle)
  d |= (unsigned long long)(1024 >> 4) << 32;                   // stride byte offset: next group of 8 rows
  d |= (unsigned long long)1 << 46;                             // descriptor version of this architecture
  d |= (unsigned long long)2 << 61;                             // 128-byte swizzle
  return d;
}
__device__ __forceinline__ void tc_mma(unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(tc_smem(bar)) : "memory");
}
// True for one lane of a converged warp, in a way that the compiler knows to be one lane.
__device__ __forceinline__ bool tc_elect() {
  unsigned one;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one != 0;
}

// ---- pairs of blocks (clusters of two, cta_group::2): the first block of the pair issues the products of both ----
__device__ __forceinline__ unsigned tc_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
// the address, in the pair, of what lies at `p` in this block's shared memory, but in the pair's first block
__device__ __forceinline__ unsigned tc_first_block(const void* p) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(a) : "r"(tc_smem(p)));
  return a;
}
__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
// a copy into this block's shared memory that counts its bytes on a barrier of the pair's first block (`bar`: tc_first_block)
__device__ __forceinline__ void tc_tma_load_pair(void* dst, const CUtensorMap* map, int col, int row, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          tc_smem(dst)),
      "l"(map), "r"(col), "r"(row), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_mma_pair(unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives at the barrier of both blocks when every product issued so far has finished
__device__ __forceinline__ void tc_commit_pair(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(tc_smem(bar)),
               "h"((unsigned short)3)
               : "memory");
}
__device__ __forceinline__ void tc_bar_arrive_at(unsigned bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_ld16(unsigned taddr, float (&v)[16]) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tc_ld32(unsigned taddr, float (&v)[32]) {
  unsigned r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
// GELU of the epilogue.  When the result is rounded to bfloat16 anyway, the tanh form uses the hardware's tanh
// (relative error about 2^-11, below that rounding); a 32-bit result gets the full-precision functions.
__device__ __forceinline__ unsigned tc_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ float tc_activation(float x, int act, bool exact) {
  if (exact) return apply_activation(x, act);
  if (act == kActGeluTanh) {
    float t;
    asm("tanh.approx.f32 %0, %1;\n" : "=f"(t) : "f"(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    return 0.5f * x * (1.f + t);
  }
  if (act == kActGeluErf) return gelu_erf(x);
  return x;
}
// gated_pair (common.cuh) for results that are rounded to bfloat16: the same rules with the special-function unit's exponential and
// reciprocal (a few units of 2^-23, more where the exponential is small; the tanh form as x sigmoid(2 z)).  Where 1 + e^x is too large for
// the reciprocal both sides of the division are taken down by 2^32.
template <int ACT>
__device__ __forceinline__ float tc_gated(float g, float u, float limit) {
  if (ACT == kActGeluErf) return gelu_erf(g) * u;
  float e = g;
  if (ACT == kActSwishClamp) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit) + 1.f;
    e = 1.702f * g;
  } else if (ACT == kActGeluTanh) {
    e = 2.f * 0.7978845608028654f * (g + 0.044715f * g * g * g);
  }
  const float y = 1.f + __expf(-e), down = y > 0x1p125f ? 0x1p-32f : 1.f;
  return __fdividef(g * down, y * down) * u;
}
// v = rule(v) * up
template <int ACT>
__device__ __forceinline__ void tc_gated_all(float (&v)[32], const float (&up)[32], float limit) {
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = tc_gated<ACT>(v[i], up[i], limit);
}
__device__ __forceinline__ void tc_bar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc_smem(bar)) : "memory");
}

}  // namespace bt
