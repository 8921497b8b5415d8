// tcgen05 (5th-generation tensor core), tensor-memory and TMA wrappers shared by the
// tensor-core GEMM and convolution kernels.  Everything here is inline PTX for sm_100a;
// every load is CTA-local.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "device_utils.cuh"

namespace b200 {

// One lane of a converged warp (the same one every time).  The warps that issue tcgen05.mma stay
// converged -- every lane runs the loops and the waits, and only the instruction itself is left to
// the elected lane -- because descriptors and addresses then live in uniform registers, which the
// instruction wants: issued from an `if (lane == 0)` branch, every MMA first moves its operands
// there, 120 - 145 cycles an instruction whatever its width; issued this way the tensor pipe is the
// limit (measured back to back on TF32, M = 128: 48 cycles at N = 64, 64 at 128, 96 at 192, 128 at 256).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}
// the warp's number, known to the compiler to be the same in all of its lanes
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// bounded wait of a whole warp: the same answer in every lane
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
}
// The same for roles that can be late by SLEEP_NS: a warp that polls takes issue slots from the working
// warps of its SM (with sixteen pollers, most of them), one that sleeps between polls does not.
template <int SLEEP_NS>
__device__ __forceinline__ bool mbar_wait_warp_sleep(uint64_t *bar, uint32_t parity,
                                                     unsigned long long limit_ns = 2000000000ull) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t0));
    do {
#pragma unroll 1
      for (int i = 0; i < 64 && !ok; ++i) {
        __nanosleep(SLEEP_NS);
        ok = mbar_try_wait(bar, parity);
      }
      asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t1));
    } while (!ok && t1 - t0 < limit_ns);
  }
  return __all_sync(0xffffffffu, ok);
}

// instruction descriptor: TF32 x TF32 -> F32, both operands K-major, M x N tile
__host__ __device__ constexpr uint32_t umma_idesc_tf32(int M, int N) {
  return (1u << 4)                    // D format F32
         | (2u << 7)                  // A format TF32
         | (2u << 10)                 // B format TF32
         | ((uint32_t)(N >> 3) << 17) // N / 8
         | ((uint32_t)(M >> 4) << 24); // M / 16
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                 smem_u32(bar))
               : "memory");
}

// 3D tiled load (coordinates innermost first) into this CTA's shared memory that counts its bytes on `bar`, a
// shared::cluster address: a pair's second CTA names the first one's barrier (leader_bar), on which the MMA that reads both
// CTAs' rows waits.  The innermost coordinate must be a multiple of 16 bytes; coordinates outside the tensor read zero.
template <int CG>
__device__ __forceinline__ void tma_load_3d_cg(void *dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t bar) {
  if constexpr (CG == 1)
    asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n" ::"r"(
        smem_u32(dst)),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
  else
    asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n" ::"r"(
        smem_u32(dst)),
      "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// the barrier of a pair's first CTA, or this CTA's own
template <int CG>
__device__ __forceinline__ uint32_t leader_bar(const uint64_t *bar) {
  uint32_t at = smem_u32(bar);
  if constexpr (CG == 2) asm("mapa.shared::cluster.u32 %0, %0, 0;\n" : "+r"(at));
  return at;
}

__device__ __forceinline__ void tma_load_4d(void *smem_dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, int c3, uint64_t *bar) {
  asm volatile(
    "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n" ::"r"(
      smem_u32(smem_dst)),
    "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
    : "memory");
}

// General shared-memory matrix descriptor.  `layout`: 2 = 128-byte swizzle of 16-byte chunks
// (K-major operands: rows of 32 floats, `sbo` bytes between groups of 8 rows), 1 = 128-byte
// swizzle of 32-byte chunks (the form 32-bit MN-major operands need: rows are 32 floats along
// M/N, one row per k; `lbo` bytes between successive 32-wide M/N blocks, `sbo` bytes between
// groups of 4 k-rows).  The swizzle is a function of the absolute shared address, so a start
// address offset by whole 128-byte rows addresses the rows that follow.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo,
                                              uint32_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffff) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)layout << 61;
  return d;
}

// round to the nearest TF32 (10 explicit mantissa bits, ties away from zero); lo = x - hi is exact
// in fp32.  Integer form of cvt.rna.tf32.f32 (same bits for every finite input): that instruction
// issues on the conversion pipe, a quarter-rate unit that a kernel converting an im2col tile in
// its inner loop saturates, while an add and a mask run at full rate.
__device__ __forceinline__ void split_tf32_rn(float x, float &hi, float &lo) {
  hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  lo = x - hi;
}

__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                 smem_u32(slot)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(cols)
               : "memory");
}

// ---- forms for one CTA (CG = 1) or a pair of CTAs on neighbouring SMs (CG = 2) ----------------------
// In a pair the CTA of even rank (the leader) issues the MMAs for both: A rows and accumulator rows are
// split between the CTAs, each holds half of B's rows, and a commit signals the barrier of both.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;\n" ::: "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_alloc_cg(uint32_t *slot, uint32_t cols) {
  if constexpr (CG == 1) {
    tmem_alloc(slot, cols);
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc_cg(uint32_t base, uint32_t cols) {
  if constexpr (CG == 1)
    tmem_dealloc(base, cols);
  else
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(cols) : "memory");
}
// instruction descriptor: bf16 x bf16 -> F32, both operands K-major, M x N tile
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// bf16 operands, A from tensor memory: two k's per 32-bit column, 8 columns (16 k's) per instruction
template <int CG>
__device__ __forceinline__ void umma_bf16_ta_cg(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                                uint32_t accumulate) {
  if constexpr (CG == 1)
    asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
  else
    asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// the same value in every lane, known as such to the compiler
__device__ __forceinline__ uint32_t uni(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }

// The six products of one step of 16 k's of operands split by split_bf16x3, small ones first: the largest
// to the accumulator dm, the others to dl.  A's parts lie 16 columns apart, B's P descriptor units.
template <int CG>
__device__ __forceinline__ void umma_6(uint32_t dm, uint32_t dl, uint32_t a1, uint64_t b1, uint32_t P, uint32_t idesc,
                                       uint32_t more) {
  const uint32_t a2 = a1 + 16, a3 = a1 + 32;
  const uint64_t b2 = b1 + P, b3 = b2 + P;
  umma_bf16_ta_cg<CG>(dl, a3, b1, idesc, more);
  umma_bf16_ta_cg<CG>(dl, a1, b3, idesc, 1);
  umma_bf16_ta_cg<CG>(dl, a2, b2, idesc, 1);
  umma_bf16_ta_cg<CG>(dl, a2, b1, idesc, 1);
  umma_bf16_ta_cg<CG>(dl, a1, b2, idesc, 1);
  umma_bf16_ta_cg<CG>(dm, a1, b1, idesc, more);
}

// the same into one accumulator
template <int CG>
__device__ __forceinline__ void umma_6one(uint32_t d, uint32_t a1, uint64_t b1, uint32_t P, uint32_t idesc, uint32_t more) {
  const uint32_t a2 = a1 + 16, a3 = a1 + 32;
  const uint64_t b2 = b1 + P, b3 = b2 + P;
  umma_bf16_ta_cg<CG>(d, a3, b1, idesc, more);
  umma_bf16_ta_cg<CG>(d, a1, b3, idesc, 1);
  umma_bf16_ta_cg<CG>(d, a2, b2, idesc, 1);
  umma_bf16_ta_cg<CG>(d, a2, b1, idesc, 1);
  umma_bf16_ta_cg<CG>(d, a1, b2, idesc, 1);
  umma_bf16_ta_cg<CG>(d, a1, b1, idesc, 1);
}

template <int CG>
__device__ __forceinline__ void umma_commit_cg(uint64_t *bar) {
  if constexpr (CG == 1)
    umma_commit(bar);
  else
    asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(
        smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
// Arrival at the leader's barrier (this CTA's own one without a pair) that hands over tensor memory only,
// after tcgen05.wait and tcgen05.fence::before_thread_sync.  Relaxed: a releasing arrival also waits for the
// thread's global stores, a microsecond in an epilogue (conv 3->32 5x5, 32x32, batch 256: 31 -> 24 us).
template <int CG>
__device__ __forceinline__ void mbar_arrive_leader(uint64_t *bar) {
  if constexpr (CG == 1) {
    asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
  } else {
    asm volatile(
      "{\n .reg .b32 ra;\n mapa.shared::cluster.u32 ra, %0, 0;\n"
      " mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [ra];\n}\n" ::"r"(smem_u32(bar))
      : "memory");
  }
}
// bounded wait of a whole warp for arrivals that may come from the other CTA of a pair
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
    "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
    " selp.u32 %0, 1, 0, p;\n}\n"
    : "=r"(ok)
    : "r"(smem_u32(bar)), "r"(parity)
    : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_warp_cluster(uint64_t *bar, uint32_t parity,
                                                       unsigned long long limit_ns = 2000000000ull) {
  bool ok = mbar_try_wait_cluster(bar, parity);
  if (!ok) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t0));
    do {
#pragma unroll 1
      for (int i = 0; i < 64 && !ok; ++i) ok = mbar_try_wait_cluster(bar, parity);
      asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t1));
    } while (!ok && t1 - t0 < limit_ns);
  }
  return __all_sync(0xffffffffu, ok);
}
template <int CG>
__device__ __forceinline__ bool mbar_wait_warp_cg(uint64_t *bar, uint32_t parity) {
  return CG == 1 ? mbar_wait_warp(bar, parity) : mbar_wait_warp_cluster(bar, parity);
}

// ---- shared-memory reads by address -----------------------------------
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
// Predicated loads, zero where !ok.  Straight-line code on purpose: loads inside branches are waited for where
// the branches meet, and a batch of them would then cost one memory latency each instead of one together.
__device__ __forceinline__ uint32_t ldg_if(const float *p, bool ok) {
  uint32_t v;
  asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n mov.b32 %0, 0;\n @q ld.global.nc.b32 %0, [%1];\n}\n"
               : "=r"(v)
               : "l"(p), "r"((int)ok));
  return v;
}
__device__ __forceinline__ void ldg4_if(const float *p, bool ok, uint32_t *v) {
  asm volatile(
    "{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n mov.b32 %2, 0;\n mov.b32 %3, 0;\n"
    " @q ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];\n}\n"
    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
    : "l"(p), "r"((int)ok));
}
// N = 1, 2 or 4 words of shared memory by address; the same to shared memory
template <int N>
__device__ __forceinline__ void lds_words(uint32_t addr, uint32_t *v) {
  if constexpr (N == 1)
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v[0]) : "r"(addr));
  else if constexpr (N == 2)
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v[0]), "=r"(v[1]) : "r"(addr));
  else
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
template <int N>
__device__ __forceinline__ void sts_words(uint8_t *p, const uint32_t *v) {
  if constexpr (N == 1)
    *reinterpret_cast<uint32_t *>(p) = v[0];
  else if constexpr (N == 2)
    *reinterpret_cast<uint2 *>(p) = make_uint2(v[0], v[1]);
  else
    *reinterpret_cast<uint4 *>(p) = make_uint4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
  uint32_t r[16];
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
      "=r"(r[15])
    : "r"(taddr)
    : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// the same load without the wait: issue several, then tmem_ld_wait() once before the values are used
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t *r) {
  asm volatile(
    "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
      "=r"(r[15])
    : "r"(taddr)
    : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// A operand from tensor memory (lanes = rows of A, 8 columns per TF32 instruction)
__device__ __forceinline__ void umma_tf32_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
    " tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
    "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
    : "memory");
}

// Two fp32 values as three words of packed bf16 pairs (x in the low halves): x = p1 + p2 + p3 exactly for
// every x whose parts stay above the subnormal range.  The first part is rounded to nearest, so that the
// rest is symmetric and at most 2^-8 of x; the others are truncated (what is left then fits 8 bits).
__device__ __forceinline__ void split_bf16x3(uint32_t x, uint32_t y, uint32_t &p1, uint32_t &p2, uint32_t &p3) {
  const uint32_t tx = x + 0x8000u, ty = y + 0x8000u;
  p1 = __byte_perm(tx, ty, 0x7632);
  const float rx = __uint_as_float(x) - __uint_as_float(tx & 0xffff0000u);
  const float ry = __uint_as_float(y) - __uint_as_float(ty & 0xffff0000u);
  p2 = __byte_perm(__float_as_uint(rx), __float_as_uint(ry), 0x7632);
  const float sx = rx - __uint_as_float(__float_as_uint(rx) & 0xffff0000u);
  const float sy = ry - __uint_as_float(__float_as_uint(ry) & 0xffff0000u);
  p3 = __byte_perm(__float_as_uint(sx), __float_as_uint(sy), 0x7632);
}

// 16 consecutive TMEM columns of the warp's 32 lanes; complete with tcgen05.wait::st
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r) {
  asm volatile(
    "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
    "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
    "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
    "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
    : "memory");
}

// Cycle counter of the role-timing diagnostics.  They exist only in a build with
// -DB200_TC_TIMING (python -m tiny_cnn_b200.build --tc-timing); otherwise this is a constant and
// every counter update folds away.
__device__ __forceinline__ long long tc_clock() {
#ifdef B200_TC_TIMING
  return clock64();
#else
  return 0;
#endif
}

// Role counters of that build: total cycles of a role and up to three kinds of waits (a.dbg: 16 per block).
#ifdef B200_TC_TIMING
#define CV_TIMING(ROLE, COND)                                          \
  if (a.dbg && (COND) && lane == 0) {                                  \
    long long *d = a.dbg + (size_t)blockIdx.x * 16 + (ROLE) * 4;       \
    d[0] = tc_clock() - t0, d[1] = w0, d[2] = w1, d[3] = w2;           \
  }
#else
#define CV_TIMING(ROLE, COND) (void)w0, (void)w1, (void)w2, (void)t0, (void)tq;
#endif

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}


// ---- host side: tensor-map encoder obtained from the driver at run time ----------------

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

}  // namespace b200
