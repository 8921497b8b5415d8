// Convolution on the 5th-generation tensor cores (tcgen05) with the im2col operand made in tensor
// memory, fp32-accurate.  Replaces the loops of kernels::conv2d_op_internal and
// kernels::conv2d_grad_op_internal (tiny_dnn/core/kernels/conv2d_op_internal.h:13-74 forward, :91-127 dX).
//
// Arithmetic: every fp32 operand is the exact sum of three bf16 numbers (8 + 8 + 8 significant bits),
// and the six products down to 2^-16 of the largest are accumulated in fp32; what is dropped is below
// 2^-22.  This costs the tensor pipe the same as three TF32 products (bf16 runs at twice the rate), but
// an instruction covers 16 k's, so an accumulator is added to half as often -- and the five small
// products go to an accumulator of their own, so the large one is added to once per 16 k's.  The tensor
// core truncates when it adds to an accumulator: the length of that chain is what decides the error.
//
// GEMM form of one pass: D[pixel][n] = sum_k A[pixel][k] * F[n][k], k = (channel slab, tap, channel).
//   M = 128 consecutive output pixels of the flattened (image, row, column) index per TMEM lane set --
//       every lane is an output pixel whatever the map size, and a warp's stores are consecutive;
//       a tile is S such sets per CTA, and a pair of CTAs (cta_group::2) works on two tiles at once
//   N = output channels (up to 128 at a time), so the filter is the B operand
//   K = taps x channels in steps of 16
// A exists only in tensor memory.  Loader warps read the input rows a tile needs straight from the CHW
// tensor (zero outside the image), split each value once and leave it in shared memory the way an MMA
// wants it: the bf16 parts of V neighbouring channels of a place side by side (V = 8: 16 bytes).  Gather
// warps then collect each pixel's words for 32 k's at a time (an offset table gives the place of every V
// k's relative to the pixel) and store them into the pixel's TMEM lane; a value is gathered once per tap,
// but converted once per tile, and a load instruction moves V channels.  Stride,
// dilation, window size, map size and padding are therefore addresses only.  The dX pass of a strided
// layer is one such problem per residue of the input coordinate modulo the stride ("phase"): each has
// its own taps, so no product with an inserted zero is formed.
// F streams from global memory, where conv_gather_prep leaves it split and pre-swizzled, through a
// ring of 64-k blocks; each block serves the S pixel sets of a tile.
//
// What bounds it: at N = 128 the tensor pipe (an MMA of width N takes N / 2 cycles with A in tensor memory, 24 at least).
// At N = 64 no unit by itself (56x56, 64 -> 64, 3x3, 256 samples: pipe 55 % busy, instruction issue 57 %, shared memory 38 %):
// gather and issuers hand over every 32 k's, a barrier's round trip and 450 to 900 cycles of instructions each, and wait for
// one another.  Below that the same, with an MMA that costs its least however narrow it is.
// Warp roles: 0-7 epilogue, 8-15 gather (two groups of one warp per TMEM lane quadrant, taking 32-k units
// in turn), 16-23 loaders, 24 filter producer, 25-26 MMA issuers (each takes every other pixel set: one
// warp's instructions take longer, about 900 cycles a unit, than the MMAs of a narrow unit; of a tile of one set
// each takes every other unit: 8x8, 64 -> 32 channels, 5x5, 256 samples 29.0 us, with the split 21.6 us).
// Every wait is bounded; a timeout sets the context's error word, frees tensor memory and returns.
#include <limits.h>
#include <stdio.h>
#include <stdlib.h>

#include "tc_utils.cuh"

namespace b200 {

namespace {

constexpr int CV_EPI_WARPS = 8;
constexpr int CV_GROUPS = 2;                                // gather groups of four warps
constexpr int CV_W_CONV = CV_EPI_WARPS, CV_CONV_WARPS = 4 * CV_GROUPS;
constexpr int CV_W_LOAD = CV_W_CONV + CV_CONV_WARPS, CV_LOAD_WARPS = 8, CV_LOAD_THREADS = CV_LOAD_WARPS * 32;
constexpr int CV_LOAD_DEPTH = 2;                            // places (V channels each) in flight per loader thread
constexpr int CV_W_FILT = CV_W_LOAD + CV_LOAD_WARPS, CV_W_MMA = CV_W_FILT + 1, CV_ISSUERS = 2;
constexpr int CV_THREADS = (CV_W_MMA + CV_ISSUERS) * 32;
constexpr int CV_ABUFS = 4;        // 32-k units of A in tensor memory: two per gather group
constexpr int CV_A_COLS = 48;      // columns of one: three parts, two k's per column
constexpr int CV_D_COLS = 256;     // columns of the accumulators; the A units take the other 256
constexpr int CV_MAX_D = 8;        // accumulators (large and small products) at N = 16
constexpr int CV_NAP_EPI = 60, CV_NAP_GATHER = 20, CV_NAP_LOAD = 150;  // ns asleep between looks at a barrier
constexpr int CV_MAX_PHASES = 16;
constexpr int CV_MAX_F = 12;       // filter ring stages

struct ConvPhase {
  int PH, PW;          // output pixels of the phase: PH x PW per image
  int oy0, ox0;        // output row of pixel row y: y * oys + oy0
  int nky, nkx;        // taps
  int iy0, ix0;        // input row of (pixel row y, tap row j): y * iys + iy0 + j * tdy
  int pitch;           // places per input row in shared memory
  int kslab;           // k's per channel slab (taps * CS, padded to 16)
  int koff0;           // first entry of the phase in the offset table
  int tile0;           // first tile of the phase
  long long filt;      // word offset of the phase's filter blocks
};

struct ConvGatherArgs {
  const float *in, *bias;
  const uint32_t *filt;
  float *out;
  int *err;
  int B, C, IH, IW;    // images, contracted channels, input plane
  int N, OHf, OWf;     // output channels, full output plane
  int iys, ixs, oys, oxs, tdy, tdx;
  int CS, nslab, cstr; // channels per slab (a multiple of V), slabs, places per V channels in shared memory
  int S, NP, ngroups, ND, nf;
  int Z;               // blocks that share a tile's k's (kernels with SPLIT)
  int ks;              // 2: tiles of one pixel set whose k's are split between the issuers, an accumulator each
  int nphases, ntiles, koff_len;
  int resident;        // the whole filter fits the ring: loaded once
  int act;
  long long *dbg;      // [blocks][16] cycle counters in a build with -DB200_TC_TIMING, else nullptr
  ConvPhase ph[CV_MAX_PHASES];
  CUtensorMap map;     // pairs: the filter blocks as [block * 3 + part][NP rows][32 words]
};

// input rows of one CTA tile: pixels [g0, g0 + n) of a phase
struct TileRows {
  int b0, y0, first, full, nrows;
  __device__ __forceinline__ void init(const ConvPhase &p, const ConvGatherArgs &a, int g0, int n) {
    const int plane = p.PH * p.PW, span = (p.nky - 1) * a.tdy + 1;
    b0 = g0 / plane;
    y0 = (g0 - b0 * plane) / p.PW;
    const int gl = g0 + n - 1, b1 = gl / plane, y1 = (gl - b1 * plane) / p.PW;
    full = (p.PH - 1) * a.iys + span;
    if (b1 == b0) {
      first = nrows = (y1 - y0) * a.iys + span;
    } else {
      first = (p.PH - 1 - y0) * a.iys + span;
      nrows = first + (b1 - b0 - 1) * full + y1 * a.iys + span;
    }
  }
  // shared-memory row of tap 0 of pixel row (b, y)
  __device__ __forceinline__ int slot(const ConvGatherArgs &a, int b, int y) const {
    return b == b0 ? (y - y0) * a.iys : first + (b - b0 - 1) * full + y * a.iys;
  }
};

__device__ __forceinline__ const ConvPhase &phase_of(const ConvGatherArgs &a, int tile) {
  int i = 0;
  while (i + 1 < a.nphases && tile >= a.ph[i + 1].tile0) ++i;
  return a.ph[i];
}

__device__ __forceinline__ void add_bias_act(float *v, const float *bias, int act) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 b = *reinterpret_cast<const float4 *>(bias + 4 * q);
    v[4 * q] += b.x;
    v[4 * q + 1] += b.y;
    v[4 * q + 2] += b.z;
    v[4 * q + 3] += b.w;
  }
  if (act == B200_ACT_RELU) {
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = fmaxf(0.f, v[q]);
  } else if (act == B200_ACT_TANH) {
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = tanhf(v[q]);
  }
}

// 64-k blocks of a tile that a block takes, and the 32-k units that these are
struct KRange {
  int i0, i1, u0, u1;
  __device__ __forceinline__ void init(const ConvGatherArgs &a, const ConvPhase &p, int rank) {
    const int nfb = (p.kslab + 63) >> 6, nkb = (p.kslab + 31) >> 5, n = a.nslab * nfb;
    i0 = n * rank / a.Z;
    i1 = n * (rank + 1) / a.Z;
    u0 = i0 / nfb * nkb + i0 % nfb * 2;
    u1 = i1 / nfb * nkb + i1 % nfb * 2;
  }
};

// SPLIT: a cluster of Z blocks takes one tile of 128 pixels, each a share of its k's, and adds up the sums over distributed
// shared memory, in the order of the blocks.  For passes whose tiles leave most SMs idle, where the chain over k is what
// takes the time (9x11, 220 -> 31 channels, 3x3, 5 samples: three tiles of 2000 k's, 32 us, in shares of 256 12 us).
template <int CG, int V, bool SPLIT>
__global__ void __launch_bounds__(CV_THREADS, 1) conv_gather_kernel(const __grid_constant__ ConvGatherArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t PB = (uint32_t)a.NP * 128u / CG;        // this CTA's rows of one part of a filter block
  const uint32_t FB = 3u * PB;
  const uint32_t RP = ((uint32_t)a.CS * a.cstr * 2u + 15u) & ~15u;   // one part of a slab
  const uint32_t RB = 3u * RP;
  uint8_t *filt = smem;
  uint8_t *raw = filt + (size_t)a.nf * FB;
  int *koff = reinterpret_cast<int *>(raw + 2 * (size_t)RB);
  int *pixtab = koff + a.koff_len;                       // [2][S * 128]
  int *postab = pixtab + 2 * a.S * 128;                  // [cstr rounded to 32] source offset of every place, -1: zero
  float *bias_s = reinterpret_cast<float *>(postab + ((a.cstr + 31) & ~31));
  uint64_t *raw_full = reinterpret_cast<uint64_t *>(bias_s + a.ngroups * a.NP);
  uint64_t *raw_empty = raw_full + 2;
  uint64_t *a_full = raw_empty + 2;
  uint64_t *a_empty = a_full + CV_ABUFS;
  uint64_t *acc_full = a_empty + CV_ABUFS;
  uint64_t *acc_empty = acc_full + CV_MAX_D;
  uint64_t *filt_full = acc_empty + CV_MAX_D;
  uint64_t *filt_empty = filt_full + CV_MAX_F;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(filt_empty + CV_MAX_F);

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  static_assert(!SPLIT || CG == 1, "a tile is split or a pair's");
  const uint32_t rank = CG == 2 ? cluster_rank() : 0;
  const int zrank = SPLIT ? (int)cluster_rank() : 0;
  const int cluster = SPLIT ? blockIdx.x / a.Z : blockIdx.x / CG, nclusters = SPLIT ? gridDim.x / a.Z : gridDim.x / CG;
  const int nunits = a.ntiles * a.ngroups;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&raw_full[i], CV_LOAD_WARPS);
      mbar_init(&raw_empty[i], CV_CONV_WARPS);
    }
    for (int i = 0; i < CV_ABUFS; ++i) {
      mbar_init(&a_full[i], 4 * CG);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < CV_MAX_D; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], CV_EPI_WARPS * CG);
    }
    for (int i = 0; i < a.nf; ++i) {
      mbar_init(&filt_full[i], 1);
      mbar_init(&filt_empty[i], min(a.S * a.ks, CV_ISSUERS));
    }
    mbar_fence_init();
  }
  // place of every V k's of a slab relative to the pixel's first ones, in bytes.  Entries that only pad the
  // slab to a multiple of 16 k's repeat the last real one: their filter entries are zero.
  for (int i = 0; i < a.nphases; ++i) {
    const ConvPhase &p = a.ph[i];
    const int np = (p.kslab + 63) / 64 * (64 / V), cg = a.CS / V;
    for (int k = tid; k < np; k += CV_THREADS) {
      const int kk = min(k, p.nky * p.nkx * cg - 1), tap = kk / cg, c = kk - tap * cg;
      const int jy = tap / p.nkx, jx = tap - jy * p.nkx;
      koff[p.koff0 + k] = (c * a.cstr + jy * a.tdy * p.pitch + jx * a.tdx) * (2 * V);
    }
  }
  wait_for_previous_kernel();
  for (int n = tid; n < a.ngroups * a.NP; n += CV_THREADS) bias_s[n] = (a.bias && n < a.N) ? a.bias[n] : 0.f;
  if (warp == CV_W_FILT) tmem_alloc_cg<CG>(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();
  tc_fence_after();
  // All 512 columns are this CTA's, so they start at 0: with a constant base every tensor-memory address is
  // arithmetic on loop counters and stays in uniform registers (see elect_one).
  constexpr uint32_t tmem_base = 0, tmem_a = tmem_base + CV_D_COLS;
  bool failed = __any_sync(0xffffffffu, *tmem_slot != tmem_base);

  if (SPLIT && warp < CV_EPI_WARPS) {
    // ---- epilogue of a share: the sums to shared memory, [channel][pixel], where the filter blocks were ----
    const ConvPhase &p = phase_of(a, cluster / a.ngroups);
    KRange kr;
    kr.init(a, p, zrank);
    const int nu = kr.u1 - kr.u0, quad = warp & 3;
    float *part = reinterpret_cast<float *>(filt) + quad * 32 + lane;
    bool have[2];  // with two accumulators the units go to them by parity
    for (int e = 0; e < 2; ++e) {
      have[e] = e < a.ks && (a.ks == 1 ? nu >= 1 : nu >= 2 || (nu == 1 && (kr.u0 & 1) == e));
      if (have[e] && !failed && !mbar_wait_warp_sleep<CV_NAP_EPI>(&acc_full[e], 0)) failed = true;
    }
    tc_fence_after();
    const uint32_t tq0 = tmem_base + ((uint32_t)(quad * 32) << 16);
    for (int c = (warp >> 2) * 16; c < a.NP; c += 32) {
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0.f;
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (have[e] && !failed) {
          uint32_t x[16], y[16];
          tmem_ld16_nowait(tq0 + (uint32_t)(e * 2 * a.NP + c), x);
          tmem_ld16_nowait(tq0 + (uint32_t)(e * 2 * a.NP + a.NP + c), y);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(x[j]) + __uint_as_float(y[j]);
        }
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(c + j) * 128] = v[j];
    }
  } else if (warp < CV_EPI_WARPS) {
    // ---- epilogue: two warps per TMEM lane quadrant, each takes every other 16 channels -------------
    const size_t plane_o = (size_t)a.OHf * a.OWf;
    const int quad = warp & 3;
    uint32_t q = 0;
    long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
    for (int unit = cluster; unit < nunits && !failed; unit += nclusters) {
      const int tile = unit / a.ngroups, grp = unit - tile * a.ngroups;
      const ConvPhase &p = phase_of(a, tile);
      const int PHW = p.PH * p.PW, total = a.B * PHW;
      const int g0 = ((tile - p.tile0) * CG + (int)rank) * a.S * 128;
      const int n0 = grp * a.NP;
      for (int s = 0; s < a.S; ++s, q += a.ks) {
        const uint32_t db = q % a.ND, db2 = (q + 1) % a.ND;
        const int g = g0 + s * 128 + quad * 32 + lane;
        const int b = g / PHW, r = g - b * PHW, y = r / p.PW, x = r - y * p.PW;
        float *obase = a.out + ((size_t)b * a.N + n0) * plane_o + (size_t)(y * a.oys + p.oy0) * a.OWf +
                       (x * a.oxs + p.ox0);
        tq = tc_clock();
        if (!mbar_wait_warp_sleep<CV_NAP_EPI>(&acc_full[db], (q / a.ND) & 1) ||
            (a.ks == 2 && !mbar_wait_warp_sleep<CV_NAP_EPI>(&acc_full[db2], ((q + 1) / a.ND) & 1))) {
          failed = true;
          break;
        }
        w0 += tc_clock() - tq;
        tc_fence_after();
        const uint32_t tq0 = tmem_base + ((uint32_t)(quad * 32) << 16), tacc = tq0 + db * 2u * (uint32_t)a.NP,
                       tacc2 = tq0 + db2 * 2u * (uint32_t)a.NP;
        const int cfirst = (warp >> 2) * 16;
        for (int c = cfirst; c < a.NP || c == cfirst; c += 32) {
          float v[16];
          if (c < a.NP) {
            uint32_t x[16], y[16];
            tmem_ld16_nowait(tacc + (uint32_t)c, x);
            tmem_ld16_nowait(tacc + (uint32_t)(a.NP + c), y);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(x[j]) + __uint_as_float(y[j]);
            if (a.ks == 2) {
              tmem_ld16_nowait(tacc2 + (uint32_t)c, x);
              tmem_ld16_nowait(tacc2 + (uint32_t)(a.NP + c), y);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(x[j]) + __uint_as_float(y[j]);
            }
          }
          if (c + 32 >= a.NP) {  // this warp has read its share: the last stores need not hold up the next tile
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive_leader<CG>(&acc_empty[db]);
              if (a.ks == 2) mbar_arrive_leader<CG>(&acc_empty[db2]);
            }
          }
          if (g < total && c < a.NP) {
            add_bias_act(v, bias_s + n0 + c, a.act);
            float *dst = obase + (size_t)c * plane_o;
            const int n = min(a.N - n0, a.NP) - c;
#pragma unroll
            for (int j = 0; j < 16; ++j, dst += plane_o)
              if (j < n) *dst = v[j];
          }
        }
      }
    }
    CV_TIMING(0, warp == 0)
  } else if (warp < CV_W_LOAD) {
    // ---- gather -----------------------------------------------------------------------------------
    const int group = (warp - CV_W_CONV) >> 2, quad = warp & 3;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    uint32_t v = 0, slabs = 0, it = 0;   // v: units this group has made
    long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
    for (int unit = cluster; unit < nunits && !failed; unit += nclusters, ++it) {
      const ConvPhase &p = phase_of(a, unit / a.ngroups);
      const int nkb = (p.kslab + 31) >> 5;
      const int *tab = pixtab + (it & 1) * a.S * 128 + quad * 32 + lane;
      KRange kr;
      if (SPLIT) kr.init(a, p, zrank);
      const int slab1 = SPLIT ? (kr.u1 + nkb - 1) / nkb : a.nslab;
      for (int slab = SPLIT ? kr.u0 / nkb : 0; slab < slab1 && !failed; ++slab, ++slabs) {
        const uint32_t rb = slabs & 1;
        tq = tc_clock();
        if (!mbar_wait_warp_sleep<CV_NAP_GATHER>(&raw_full[rb], (slabs >> 1) & 1)) {
          failed = true;
          break;
        }
        w0 += tc_clock() - tq;
        const uint32_t rbase = smem_u32(raw + rb * (size_t)RB);
        const int kb1 = SPLIT ? min(nkb, kr.u1 - slab * nkb) : nkb;
        for (int kb = SPLIT ? max(0, kr.u0 - slab * nkb) : 0; kb < kb1 && !failed; ++kb) {
          const uint32_t ko = smem_u32(koff + p.koff0 + kb * (32 / V));
          // A group and its two unit buffers serve the pixel sets of their own parity (alternate units when
          // there is one set): group, buffers and issuer are one pipeline that sees every phase of its barriers.
          const int first = a.S > 1 ? group : ((slab * nkb + kb) & 1) != group;
          for (int s = first; s < a.S; s += CV_GROUPS, ++v) {
            const uint32_t ab = group * 2 + (v & 1);
            tq = tc_clock();
            if (v >= 2 && !mbar_wait_warp_sleep<CV_NAP_GATHER>(&a_empty[ab], ((v >> 1) - 1) & 1)) {
              failed = true;
              break;
            }
            w1 += tc_clock() - tq;
            tc_fence_after();
            const uint32_t px1 = rbase + (uint32_t)tab[s * 128], px2 = px1 + RP, px3 = px2 + RP;
            const uint32_t ta = tmem_a + ab * CV_A_COLS + lane_base;
            uint32_t b1[16], b2[16], b3[16];
#pragma unroll
            for (int j = 0; j < 8 / V; ++j) {
              const uint4 o = lds_u4(ko + j * 16);
              const uint32_t oo[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int w = (4 * j + e) * (V / 2);
                lds_words<V / 2>(px1 + oo[e], b1 + w);
                lds_words<V / 2>(px2 + oo[e], b2 + w);
                lds_words<V / 2>(px3 + oo[e], b3 + w);
              }
            }
            tmem_st16(ta, b1);
            tmem_st16(ta + 16, b2);
            tmem_st16(ta + 32, b3);
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader<CG>(&a_full[ab]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[rb]);
      }
    }
    CV_TIMING(1, warp == CV_W_CONV)
  } else if (warp < CV_W_FILT) {
    // ---- loaders: the input rows of every slab, split, zero filled; the pixels' places ------------------
    const int lt = tid - CV_W_LOAD * 32, lw = warp - CV_W_LOAD;
    const int plane = a.IH * a.IW, ncg = a.CS / V;   // 1, 2 or 4 groups of V channels, the warps dealt to them
    const int cgrp = lw % ncg, chunk0 = lw / ncg, chunk_step = CV_LOAD_WARPS / ncg;
    uint32_t slabs = 0, it = 0;
    long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
    for (int unit = cluster; unit < nunits; unit += nclusters, ++it) {
      const int tile = unit / a.ngroups;
      const ConvPhase &p = phase_of(a, tile);
      const int PHW = p.PH * p.PW, total = a.B * PHW;
      const int g0 = ((tile - p.tile0) * CG + (int)rank) * a.S * 128;
      const int npx = min(a.S * 128, total - g0);
      TileRows tr = {};
      if (npx > 0) tr.init(p, a, g0, npx);
      const int npos = npx > 0 ? tr.nrows * p.pitch : 0, nchunks = (npos + 31) / 32;
      // every loader warp takes part in this barrier (the table below is shared), so leave together
      {
        int any;
        asm volatile(
          "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
          : "=r"(any)
          : "r"((int)failed), "n"(CV_LOAD_THREADS)
          : "memory");
        if (any) {
          failed = true;
          break;
        }
      }
      for (int pos = lt; pos < (npos + 31 & ~31); pos += CV_LOAD_THREADS) {
        int row = pos / p.pitch;
        const int ix = p.ix0 + (pos - row * p.pitch);
        int b = 0, iy = tr.y0 * a.iys + p.iy0 + row;
        if (row >= tr.first) {
          row -= tr.first;
          const int e = row / tr.full;
          b = 1 + e;
          iy = p.iy0 + row - e * tr.full;
        }
        const bool inside = pos < npos && iy >= 0 && iy < a.IH && ix >= 0 && ix < a.IW;
        postab[pos] = inside ? b * a.C * plane + iy * a.IW + ix : -1;
      }
      asm volatile("bar.sync 1, %0;\n" ::"n"(CV_LOAD_THREADS) : "memory");
      KRange kr;
      if (SPLIT) kr.init(a, p, zrank);
      const int nkb = (p.kslab + 31) >> 5, slab0 = SPLIT ? kr.u0 / nkb : 0, slab1 = SPLIT ? (kr.u1 + nkb - 1) / nkb : a.nslab;
      for (int slab = slab0; slab < slab1 && !failed; ++slab, ++slabs) {
        const uint32_t rb = slabs & 1;
        tq = tc_clock();
        if (slabs >= 2 && !mbar_wait_warp_sleep<CV_NAP_LOAD>(&raw_empty[rb], ((slabs >> 1) - 1) & 1)) {
          failed = true;
          break;
        }
        w0 += tc_clock() - tq;
        if (slab == slab0) {
          int *tab = pixtab + (it & 1) * a.S * 128;
          for (int i = lt; i < a.S * 128; i += CV_LOAD_THREADS) {
            int off = 0;
            if (i < npx) {
              const int g = g0 + i, b = g / PHW, r = g - b * PHW, y = r / p.PW, x = r - y * p.PW;
              off = (tr.slot(a, b, y) * p.pitch + x * a.ixs) * (2 * V);
            }
            tab[i] = off;
          }
        }
        const int c0 = slab * a.CS + cgrp * V, nc = min(V, a.C - c0);   // real channels of this warp's group
        const float *src = a.in + ((size_t)tr.b0 * a.C + c0) * plane;
        uint8_t *dst = raw + rb * (size_t)RB + (size_t)(cgrp * a.cstr) * (2 * V);
        for (int ch = chunk0; ch < nchunks; ch += chunk_step * CV_LOAD_DEPTH) {
          uint32_t x[CV_LOAD_DEPTH][V];
#pragma unroll
          for (int j = 0; j < CV_LOAD_DEPTH; ++j) {
            const int pos = (ch + j * chunk_step) * 32 + lane;
            const int off = pos < npos ? postab[pos] : -1;
            const float *q = src + off;
#pragma unroll
            for (int c = 0; c < V; ++c, q += plane) x[j][c] = ldg_if(q, off >= 0 && c < nc);
          }
#pragma unroll
          for (int j = 0; j < CV_LOAD_DEPTH; ++j) {
            const int pos = (ch + j * chunk_step) * 32 + lane;
            uint32_t p1[V / 2], p2[V / 2], p3[V / 2];
#pragma unroll
            for (int c = 0; c < V / 2; ++c) split_bf16x3(x[j][2 * c], x[j][2 * c + 1], p1[c], p2[c], p3[c]);
            if (pos < npos) {
              uint8_t *d = dst + pos * (2 * V);
              sts_words<V / 2>(d, p1);
              sts_words<V / 2>(d + RP, p2);
              sts_words<V / 2>(d + 2 * RP, p3);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_full[rb]);
      }
    }
    CV_TIMING(2, warp == CV_W_LOAD)
  } else if (warp == CV_W_FILT) {
    // ---- filter producer --------------------------------------------------------------------------------
    uint32_t f = 0;
    for (int unit = cluster; unit < nunits && !failed; unit += nclusters) {
      const int tile = unit / a.ngroups, grp = unit - tile * a.ngroups;
      const ConvPhase &p = phase_of(a, tile);
      const int nblk = a.nslab * ((p.kslab + 63) >> 6);
      const uint32_t *src = a.filt + p.filt + (size_t)grp * nblk * a.NP * 96;
      const int block = (int)(p.filt / (a.NP * 96)) + grp * nblk;
      KRange kr;
      if (SPLIT) kr.init(a, p, zrank);
      for (int i = SPLIT ? kr.i0 : 0; i < (SPLIT ? kr.i1 : nblk); ++i, ++f) {
        const uint32_t st = f % a.nf, use = f / a.nf;
        if (use > 0 && !mbar_wait_warp_sleep<CV_NAP_LOAD>(&filt_empty[st], (use - 1) & 1)) {
          failed = true;
          break;
        }
        if (elect_one()) {
          uint8_t *d = filt + (size_t)st * FB;
          if (rank == 0) mbar_expect_tx(&filt_full[st], FB * CG);
          if (CG == 1)
            bulk_copy_g2s(d, src + (size_t)i * a.NP * 96, FB, &filt_full[st]);
          else
            tma_load_3d_cg<CG>(d, &a.map, 0, (int)rank * (a.NP / 2), (block + i) * 3, leader_bar<CG>(&filt_full[st]));
        }
        __syncwarp();
      }
      if (a.resident) break;
    }
  } else if (rank == 0) {
    // ---- MMA issuers (the whole warp stays converged: see elect_one) ---
    const int me = warp - CV_W_MMA;
    const uint32_t idesc = umma_idesc_bf16(128 * CG, a.NP);
    const uint64_t f0 = umma_desc(smem_u32(filt), 16, 1024, 2);
    const uint32_t P = PB >> 4;   // one part further, in descriptor units
    const uint64_t f0hi = f0 & 0xffffffff00000000ull;
    uint32_t st = 0, fpar = 0;                 // filter ring: stage, parity of its current use
    uint32_t v = 0, v1 = 0;                    // units taken (from the two groups, where one issuer serves both)
    uint32_t db0 = 0, dpar0 = 1;               // accumulator of the tile's first pixel set, parity of its last release
    bool first = true, fresh = true;           // first tile of this CTA; accumulators not yet used before
    long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
    // No loop ends early on a failed wait: what follows it neither waits nor issues, and the trip counts
    // depend on the arguments alone, which keeps the loop state in uniform registers.  An issuer steps through
    // its own pixel sets only: its instructions, not the tensor pipe, bound layers of 64 outputs and fewer.
    const int nsets = a.S * a.ks;
    const bool paired = nsets > 1;             // a gather group and its two buffers belong to one issuer
    for (int unit = cluster; unit < nunits && me < nsets; unit += nclusters) {
      const ConvPhase &p = phase_of(a, unit / a.ngroups);
      KRange kr;
      if (SPLIT) kr.init(a, p, zrank);
      const int kslab = p.kslab, nfb = (kslab + 63) >> 6, nblk = SPLIT ? kr.i1 : a.nslab * nfb,
                nku = SPLIT ? kr.u1 : a.nslab * ((kslab + 31) >> 5), ubeg = SPLIT ? kr.u0 : 0;
      int u0 = ubeg;                           // units of the tile before this block
      for (int i = SPLIT ? kr.i0 : 0, fb = SPLIT ? kr.i0 % nfb : 0; i < nblk; ++i, fb = fb + 1 == nfb ? 0 : fb + 1) {
        tq = tc_clock();
        if ((!a.resident || first) && !failed) {
          failed = !mbar_wait_warp_cg<CG>(&filt_full[st], fpar);
        }
        w0 += tc_clock() - tq;
        const int k16 = min(4, (kslab - fb * 64) >> 4);  // steps of this block, two per unit
        const uint32_t fst = (uint32_t)f0 + ((st * FB) >> 4);
        const int nh = (k16 + 1) >> 1;
        for (int h = a.ks == 2 ? (u0 ^ me) & 1 : 0; h < nh; h += a.ks) {
          const bool last = u0 + h + a.ks >= nku, both = k16 - h * 2 >= 2;
          const uint32_t more = u0 + h - ubeg >= a.ks;
          const uint64_t b1 = f0hi | uni(fst + (uint32_t)(h * 4));
          for (int s = me; s < nsets; s += CV_ISSUERS) {
            uint32_t db = db0 + s;
            const bool wrapped = db >= (uint32_t)a.ND;
            if (wrapped) db -= a.ND;
            tq = tc_clock();
            if (more == 0 && !(fresh && !wrapped) && !failed)
              failed = !mbar_wait_warp_cg<CG>(&acc_empty[db], dpar0 ^ (uint32_t)wrapped);
            w1 += tc_clock() - tq;
            tq = tc_clock();
            // one issuer alone takes the groups in turn, from group 0 in every tile
            const bool second = !paired && ((u0 + h) & 1);  // by the unit's number in the tile, as the groups count
            const uint32_t turn = second ? v1++ : v++, ab = (paired ? me : (int)second) * 2 + (turn & 1);
            if (!failed) failed = !mbar_wait_warp_cg<CG>(&a_full[ab], (turn >> 1) & 1);
            w2 += tc_clock() - tq;
            tc_fence_after();
            const uint32_t dm = uni(tmem_base + db * 2u * (uint32_t)a.NP), dl = dm + (uint32_t)a.NP;
            const uint32_t a1 = uni(tmem_a + ab * CV_A_COLS);
            if (!failed && elect_one()) {
              umma_6<CG>(dm, dl, a1, b1, P, idesc, more);
              if (both) umma_6<CG>(dm, dl, a1 + 8, b1 + 2, P, idesc, 1);
              umma_commit_cg<CG>(&a_empty[ab]);
              if (last) umma_commit_cg<CG>(&acc_full[db]);
            }
            __syncwarp();
          }
        }
        u0 += nh;
        if (!failed && !a.resident && elect_one()) umma_commit_cg<CG>(&filt_empty[st]);
        __syncwarp();
        if (++st == (uint32_t)a.nf) st = 0, fpar ^= 1;
      }
      first = false;
      db0 += nsets;
      if (db0 >= (uint32_t)a.ND) db0 -= a.ND, dpar0 ^= 1, fresh = false;
    }
    CV_TIMING(3, warp == CV_W_MMA)
  }
  if (failed && a.err) atomicExch(a.err, 3);
  tc_fence_before();
  __syncthreads();
  if (CG == 2 || SPLIT) cluster_sync();
  if (warp == CV_W_FILT) tmem_dealloc_cg<CG>(tmem_base, 512);
  if (SPLIT) {
    // every block adds up each Z-th channel of the tile, a warp 32 pixels of a channel
    const int tile = cluster / a.ngroups, n0 = (cluster - tile * a.ngroups) * a.NP, n = min(a.N - n0, a.NP);
    const ConvPhase &p = phase_of(a, tile);
    const int PHW = p.PH * p.PW, total = a.B * PHW;
    const size_t plane_o = (size_t)a.OHf * a.OWf;
    const uint32_t part = smem_u32(filt);
    for (int e = warp; e < (n - zrank + a.Z - 1) / a.Z * 4; e += CV_THREADS / 32) {
      const int c = e / 4 * a.Z + zrank, px = e % 4 * 32 + lane, g = (tile - p.tile0) * 128 + px;
      float v[8];
#pragma unroll
      for (int z = 0; z < 8; ++z)
        if (z < a.Z) {
          uint32_t ra;
          asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(part + (uint32_t)(c * 128 + px) * 4u), "r"(z));
          asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v[z]) : "r"(ra) : "memory");
        }
#pragma unroll
      for (int z = 1; z < 8; ++z)
        if (z < a.Z) v[0] += v[z];
      if (g >= total) continue;
      const int b = g / PHW, r = g - b * PHW, y = r / p.PW, x = r - y * p.PW;
      a.out[((size_t)b * a.N + n0 + c) * plane_o + (size_t)(y * a.oys + p.oy0) * a.OWf + (x * a.oxs + p.ox0)] =
        apply_act(v[0] + bias_s[n0 + c], a.act);
    }
    cluster_sync();  // nobody leaves while others read its sums
  }
}

// ---- filter blocks ---------------------------------------------------------------------------------
//
// [phase][group][slab][64-k block][part]: NP rows of 64 k's as bf16 (128 bytes, 128-byte swizzle).
// Forward: row n is output channel n, k = (tap, input channel).  dX: row n is input channel n, k = (tap,
// output channel), and tap j of a phase is the filter row phase + stride * (nky - 1 - j).
struct FilterSet {
  uint32_t *dst;
  int for_dx, NP, ngroups, CS, nslab, nphases, SH, SW;
  long long total;                 // words of one part: (row, pair of k's)
  int nky[CV_MAX_PHASES], nkx[CV_MAX_PHASES], fy[CV_MAX_PHASES], fx[CV_MAX_PHASES], kslab[CV_MAX_PHASES];
  long long first[CV_MAX_PHASES];  // first (row, pair) of the phase
};

__global__ void __launch_bounds__(256) conv_gather_prep_kernel(const float *__restrict__ W, const uint8_t *__restrict__ tbl,
                                                               int C, int OC, int KH, int KW,
                                                               const __grid_constant__ FilterSet s0,
                                                               const __grid_constant__ FilterSet s1) {
  after_previous_kernel();
  const FilterSet &s = blockIdx.y == 0 ? s0 : s1;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < s.total; i += gridDim.x * 256ll) {
    int ph = 0;
    while (ph + 1 < s.nphases && i >= s.first[ph + 1]) ++ph;
    const uint32_t r0 = (uint32_t)(i - s.first[ph]);
    const int kp = r0 & 31;
    const uint32_t r1 = r0 >> 5, blk = r1 / s.NP;
    const int n = r1 - blk * s.NP;
    const int nfb = (s.kslab[ph] + 63) >> 6;
    const uint32_t r2 = blk / nfb, grp = r2 / s.nslab;
    const int fb = blk - r2 * nfb, slab = r2 - grp * s.nslab, nn = grp * s.NP + n;
    uint32_t v[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int kk = fb * 64 + kp * 2 + e, tap = kk / s.CS, c = slab * s.CS + kk - tap * s.CS;
      float x = 0.f;
      if (tap < s.nky[ph] * s.nkx[ph]) {
        int ky = tap / s.nkx[ph], kx = tap - ky * s.nkx[ph];
        if (s.for_dx) {
          ky = s.fy[ph] + s.SH * (s.nky[ph] - 1 - ky);
          kx = s.fx[ph] + s.SW * (s.nkx[ph] - 1 - kx);
        }
        const int o = s.for_dx ? c : nn, inc = s.for_dx ? nn : c;
        if (o < OC && inc < C && ky < KH && kx < KW && (tbl == nullptr || tbl[inc * OC + o]))
          x = W[((size_t)(o * C + inc) * KH + ky) * KW + kx];
      }
      v[e] = __float_as_uint(x);
    }
    uint32_t *d = s.dst + 3 * s.first[ph] + (size_t)blk * s.NP * 96 + n * 32 + ((((kp >> 2) ^ (n & 7)) << 2) | (kp & 3));
    split_bf16x3(v[0], v[1], d[0], d[s.NP * 32], d[s.NP * 64]);
  }
}

// ---- host side ----------------------------------------------------------------------------------------

// Tiling of one pass.  Nothing here depends on the batch except what launch_conv_gather decides, so the
// filter blocks serve every batch size.
struct GatherPlan {
  bool ok;
  int Cc, Nn;                 // contracted channels, output channels
  int NP, ngroups, ND;
  int V, S, CS, nslab, cstr;  // S: the most pixel sets per CTA tile
  int koff_len;
  long long filt_words;       // words of one of the three parts of the filter blocks
  ConvPhase ph[CV_MAX_PHASES];
  int fy[CV_MAX_PHASES], fx[CV_MAX_PHASES];
  int nphases;
  int iys, ixs, oys, oxs, tdy, tdx;
};

// channels side by side in shared memory
int gather_vec(int channels) { return channels <= 2 ? 2 : channels <= 4 ? 4 : 8; }

// rows of input a tile of n consecutive pixels needs at most
int rows_needed(const ConvPhase &p, const GatherPlan &g, int n) {
  const long long plane = (long long)p.PH * p.PW;
  const int span = (p.nky - 1) * g.tdy + 1;
  long long orows = n % p.PW == 0 ? n / p.PW : (n + p.PW - 2) / p.PW + 1;
  long long imgs = plane % n == 0 ? 1 : n % plane == 0 ? n / plane : (n + plane - 2) / plane + 1;
  if (orows < imgs) orows = imgs;
  const int extra = span > g.iys ? span - g.iys : 0;
  return (int)(g.iys * orows + imgs * extra);
}

size_t gather_fixed_smem(const GatherPlan &p) {
  return 1024 + (size_t)p.koff_len * 4 + 2 * (size_t)p.S * 128 * 4 + align_up(p.cstr, 32) * 4 + (size_t)p.ngroups * p.NP * 4 +
         (4 + 2 * CV_ABUFS + 2 * CV_MAX_D + 2 * CV_MAX_F) * 8 + 64;
}

GatherPlan gather_plan(const b200_ctx *ctx, const ConvGeom &g, int for_dx) {
  GatherPlan p = {};
  p.Cc = for_dx ? g.OC : g.C;
  p.Nn = for_dx ? g.C : g.OC;
  p.iys = for_dx ? 1 : g.SH;
  p.ixs = for_dx ? 1 : g.SW;
  p.oys = for_dx ? g.SH : 1;
  p.oxs = for_dx ? g.SW : 1;
  p.tdy = for_dx ? 1 : g.DH;
  p.tdx = for_dx ? 1 : g.DW;
  if (g.pad_t < 0 || g.pad_l < 0) return p;
  if (for_dx) {
    if (g.SH * g.SW > CV_MAX_PHASES) return p;
    for (int fy = 0; fy < g.SH; ++fy)
      for (int fx = 0; fx < g.SW; ++fx) {
        ConvPhase q = {};
        q.oy0 = ((fy - g.pad_t) % g.SH + g.SH) % g.SH;   // first input row of this residue
        q.ox0 = ((fx - g.pad_l) % g.SW + g.SW) % g.SW;
        q.PH = g.HI > q.oy0 ? (g.HI - q.oy0 + g.SH - 1) / g.SH : 0;
        q.PW = g.WI > q.ox0 ? (g.WI - q.ox0 + g.SW - 1) / g.SW : 0;
        if (q.PH == 0 || q.PW == 0) continue;
        q.nky = g.KH > fy ? (g.KH - fy + g.SH - 1) / g.SH : 1;  // no tap reaches the residue: one zero tap
        q.nkx = g.KW > fx ? (g.KW - fx + g.SW - 1) / g.SW : 1;
        q.iy0 = (q.oy0 + g.pad_t) / g.SH - (q.nky - 1);
        q.ix0 = (q.ox0 + g.pad_l) / g.SW - (q.nkx - 1);
        p.fy[p.nphases] = fy;
        p.fx[p.nphases] = fx;
        p.ph[p.nphases++] = q;
      }
  } else {
    ConvPhase q = {};
    q.PH = g.OH;
    q.PW = g.OW;
    q.nky = g.KH;
    q.nkx = g.KW;
    q.iy0 = -g.pad_t;
    q.ix0 = -g.pad_l;
    p.ph[p.nphases++] = q;
  }
  int taps = 0;
  for (int i = 0; i < p.nphases; ++i) {
    ConvPhase &q = p.ph[i];
    q.pitch = (q.PW - 1) * p.ixs + (q.nkx - 1) * p.tdx + 1;
    if (q.nky * q.nkx > taps) taps = q.nky * q.nkx;
  }
  const int n16 = (p.Nn + 15) / 16 * 16;
  p.ngroups = (n16 + 127) / 128;
  p.NP = ((n16 + p.ngroups - 1) / p.ngroups + 15) / 16 * 16;
  p.ND = CV_D_COLS / (2 * p.NP) < CV_MAX_D ? CV_D_COLS / (2 * p.NP) : CV_MAX_D;
  // Largest S with slabs of at least 16 channels (or all): a filter block is then used S times per
  // refill.  Two ring stages must fit beside two slabs.
  const size_t ring = (size_t)2 * p.NP * 384;
  p.V = gather_vec(p.Cc);
  const int cv = (p.Cc + p.V - 1) / p.V * p.V;
  int best_cs = 0;
  for (int S = p.ND; S >= 1; S /= 2) {  // powers of two, so that the two pipelines share evenly
    int cstr = 0;
    bool near = true;  // a place's source offset from the tile's first image fits 32 bits
    for (int i = 0; i < p.nphases; ++i) {
      const long long need = (long long)rows_needed(p.ph[i], p, S * 128) * p.ph[i].pitch;
      if (need > 1 << 20) return p;
      if (need > cstr) cstr = (int)need;
      const long long pixels = (long long)p.ph[i].PH * p.ph[i].PW, images = (S * 128 + pixels - 2) / pixels + 1;
      near = near && images * p.Cc * (for_dx ? (long long)g.OH * g.OW : (long long)g.HI * g.WI) <= INT_MAX;
    }
    if (!near) continue;
    // the table of one slab grows with CS as well: 4 bytes per pair of k's (+ padding per phase)
    const long long fixed = 1024 + 2ll * S * 512 + 4ll * align_up(cstr, 32) + (long long)p.ngroups * p.NP * 4 + 2048 + p.nphases * 256ll + (long long)ring;
    long long room = (long long)ctx->smem_optin - fixed;
    int ktaps = 0;
    for (int i = 0; i < p.nphases; ++i) ktaps += p.ph[i].nky * p.ph[i].nkx;
    long long cs = room > 0 ? room / (12ll * cstr + 4ll * ktaps / p.V + 1) / p.V * p.V : 0;
    if (cs > 32) cs = 32;
    if (cs > cv) cs = cv;
    if (cs < p.V) continue;
    const bool enough = cs >= (cv < 16 ? cv : 16);
    if (enough || cs > best_cs) {
      p.S = S;
      p.cstr = cstr;
      best_cs = (int)cs;
      if (enough) break;
    }
  }
  if (best_cs == 0) return p;
  // channels per slab: a power of two, so that the loader warps divide evenly, with the fewest k's after
  // padding (each slab's k's are padded to 16)
  long long least = -1;
  for (int cs = 32; cs >= p.V; cs /= 2) {
    if (cs > best_cs || cs > 4 * p.V) continue;
    long long k = 0;
    for (int i = 0; i < p.nphases; ++i) k += (long long)((p.Cc + cs - 1) / cs) * ((p.ph[i].nky * p.ph[i].nkx * cs + 15) / 16 * 16);
    if (least < 0 || k < least) {
      least = k;
      p.CS = cs;
    }
  }
  p.nslab = (p.Cc + p.CS - 1) / p.CS;
  for (int i = 0; i < p.nphases; ++i) {
    ConvPhase &q = p.ph[i];
    q.kslab = (q.nky * q.nkx * p.CS + 15) / 16 * 16;
    const int nfb = (q.kslab + 63) / 64;
    q.koff0 = p.koff_len;
    p.koff_len += nfb * (64 / p.V);
    q.filt = 3 * p.filt_words;
    p.filt_words += (long long)p.ngroups * p.nslab * nfb * p.NP * 32;
  }
  p.ok = gather_fixed_smem(p) + 6 * align_up((size_t)p.CS * p.cstr * 2, 16) + ring <= ctx->smem_optin;
  return p;
}

FilterSet filter_set(const GatherPlan &p, const ConvGeom &g, int for_dx, float *dst) {
  FilterSet s = {};
  s.dst = reinterpret_cast<uint32_t *>(dst);
  s.for_dx = for_dx;
  s.NP = p.NP;
  s.ngroups = p.ngroups;
  s.CS = p.CS;
  s.nslab = p.nslab;
  s.nphases = p.nphases;
  s.SH = g.SH;
  s.SW = g.SW;
  s.total = p.filt_words;
  for (int i = 0; i < p.nphases; ++i) {
    s.nky[i] = p.ph[i].nky;
    s.nkx[i] = p.ph[i].nkx;
    s.kslab[i] = p.ph[i].kslab;
    s.fy[i] = p.fy[i];
    s.fx[i] = p.fx[i];
    s.first[i] = p.ph[i].filt / 3;
  }
  return s;
}

// 32-k units of the phase with the fewest
int least_units(const GatherPlan &p) {
  int n = 1 << 30;
  for (int i = 0; i < p.nphases; ++i) {
    const int u = p.nslab * ((p.ph[i].kslab + 31) / 32);
    if (u < n) n = u;
  }
  return n;
}

// CTA pair or single CTAs, and S: the least time of the busiest SM, tile after tile, a tile taking the
// longer of its MMAs (N / 2 cycles each, with a floor; pairs measured 1.2 x as fast) and its loads (about
// 40 cycles for 32 places of a channel pair).
// Tiles that leave most SMs idle are split over clusters of Z blocks; as many clusters as surely run at once, however the SMs are
// grouped; about 2500 cycles for the exchange.  A block has two blocks of 64 k's or more in the phase with the most of them.  In a
// strided dX the phases with fewer taps then get shares of one or of none; with the bound on the phase with the fewest, Z is smaller and the
// phase with the most takes the time (14x14, 128 -> 64, 3x3, stride 2, two samples: 11.4 us so, 14.4 with that bound; of 108
// strided passes 24 were 6 to 22 % slower with it, none faster).
struct GatherShape {
  int CG, S, ks, Z, blocks;
};

GatherShape gather_shape(const b200_ctx *ctx, const GatherPlan &p, int B) {
  GatherShape sh = {1, 1, 1, 1, 0};
  long long best = -1;
  for (int cg = 2; cg >= 1; --cg) {
    for (int S = p.S; S >= 1; S /= 2) {
      const int ks = S == 1 && p.ND >= 2 && least_units(p) >= 2 ? 2 : 1;
      const long long slots = ctx->sm_count / cg;
      for (int Z = 1; Z <= (cg * S == 1 ? 8 : 1); Z *= 2) {
        long long tiles = 0, tile_cost = 0, blocks = 0;
        for (int i = 0; i < p.nphases; ++i) {
          const ConvPhase &q = p.ph[i];
          tiles += ((long long)B * q.PH * q.PW + cg * S * 128 - 1) / (cg * S * 128);
          const long long units = ((long long)p.nslab * ((q.kslab + 31) / 32) * S + Z - 1) / Z;
          blocks = max(blocks, (long long)p.nslab * ((q.kslab + 63) / 64));
          // about 900 cycles of an issuer's instructions a unit
          const long long issue = S * ks > 1 ? 450 : 900;
          const long long mma = units * (p.NP * 6 > issue ? p.NP * 6 : issue) * (cg == 2 ? 5 : 6) / 5;
          const long long load = (long long)((p.nslab + Z - 1) / Z) * ((p.CS + 1) / 2) * ((rows_needed(q, p, S * 128) * q.pitch + 31) / 32) * 40;
          tile_cost += mma > load ? mma : load;
        }
        if (Z > 1 && (blocks < 2 * Z || tiles * p.ngroups > ctx->sm_count / Z * 7 / 8)) break;
        const long long cost = (tiles * p.ngroups + slots - 1) / slots * (tile_cost / p.nphases + 2000 + (Z > 1 ? 2500 : 0));
        if (best < 0 || cost < best) {
          best = cost;
          sh = {cg, S, ks, Z, (int)min(tiles * p.ngroups, slots) * cg * Z};
        }
      }
    }
  }
  return sh;
}

int launch_conv_gather(b200_ctx *ctx, const GatherPlan &p, const ConvGeom &g, int for_dx, const float *in, const float *filt,
                       const float *bias, float *out, int B, int act) {
  // the kernel counts pixels and tiles in 32 bits
  long long plane = 1;
  for (int i = 0; i < p.nphases; ++i) plane = max(plane, (long long)p.ph[i].PH * p.ph[i].PW);
  const int most = (int)max(1ll, (1ll << 30) / plane);
  if (B > most) {
    const size_t in_len = (size_t)p.Cc * (for_dx ? g.OH * g.OW : g.HI * g.WI),
                 out_len = (size_t)p.Nn * (for_dx ? g.HI * g.WI : g.OH * g.OW);
    for (int b = 0; b < B; b += most)
      B200_TRY(launch_conv_gather(ctx, p, g, for_dx, in + b * in_len, filt, bias, out + b * out_len, min(most, B - b), act));
    return 0;
  }
  ConvGatherArgs a = {};
  a.in = in;
  a.filt = reinterpret_cast<const uint32_t *>(filt);
  a.bias = bias;
  a.out = out;
  a.err = ctx->dev_err;
  a.B = B;
  a.C = p.Cc;
  a.N = p.Nn;
  a.IH = for_dx ? g.OH : g.HI;
  a.IW = for_dx ? g.OW : g.WI;
  a.OHf = for_dx ? g.HI : g.OH;
  a.OWf = for_dx ? g.WI : g.OW;
  a.iys = p.iys;
  a.ixs = p.ixs;
  a.oys = p.oys;
  a.oxs = p.oxs;
  a.tdy = p.tdy;
  a.tdx = p.tdx;
  a.CS = p.CS;
  a.nslab = p.nslab;
  a.cstr = p.cstr;
  a.NP = p.NP;
  a.ngroups = p.ngroups;
  a.ND = p.ND;
  a.nphases = p.nphases;
  a.koff_len = p.koff_len;
  a.act = act;
  const GatherShape sh = gather_shape(ctx, p, B);
  const int CG = sh.CG;
  a.S = sh.S;
  a.ks = sh.ks;
  a.Z = sh.Z;
  int tile0 = 0;
  for (int i = 0; i < p.nphases; ++i) {
    a.ph[i] = p.ph[i];
    a.ph[i].tile0 = tile0;
    tile0 += (int)(((long long)B * p.ph[i].PH * p.ph[i].PW + CG * a.S * 128 - 1) / (CG * a.S * 128));
  }
  a.ntiles = tile0;
  const size_t base = gather_fixed_smem(p) + 6 * align_up((size_t)p.CS * p.cstr * 2, 16), FB = (size_t)p.NP * 384 / CG;
  int nf = (int)((ctx->smem_optin - base) / FB);
  if (nf > CV_MAX_F) nf = CV_MAX_F;
  const int nblk = p.nslab * ((p.ph[0].kslab + 63) / 64);
  if (p.nphases == 1 && p.ngroups == 1 && nblk <= nf && sh.Z == 1) {
    a.resident = 1;
    nf = nblk;
  }
  a.nf = nf;
  const size_t smem = base + nf * FB;
  const int units = a.ntiles * a.ngroups, grid = sh.blocks;
#ifdef B200_TC_TIMING
  static const bool timing = getenv("B200_TC_TIMING") != nullptr;
  if (timing) B200_CUDA(cudaMalloc(&a.dbg, (size_t)grid * 16 * sizeof(long long)));
  if (timing) B200_CUDA(cudaMemset(a.dbg, 0, (size_t)grid * 16 * sizeof(long long)));
#endif
  if (CG == 2) {
    EncodeTiledFn fn = encode_fn();
    B200_REQUIRE(fn != nullptr, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[3] = {32, (cuuint64_t)p.NP, (cuuint64_t)(3 * p.filt_words / (p.NP * 32))};
    const cuuint64_t strides[2] = {128, 128 * (cuuint64_t)p.NP};
    const cuuint32_t box[3] = {32, (cuuint32_t)p.NP / 2, 3}, estr[3] = {1, 1, 1};
    const CUresult r = fn(&a.map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<float *>(filt), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d) for the filter blocks", (int)r);
  }
  auto launch = [&](auto one, auto pair, auto split) -> int {
    auto kernel = CG == 2 ? pair : sh.Z > 1 ? split : one;
    B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch_kernel(ctx, kernel, dim3((unsigned)grid), CV_THREADS, smem, CG * sh.Z, a);
  };
  if (p.V == 2)
    B200_TRY(launch(conv_gather_kernel<1, 2, false>, conv_gather_kernel<2, 2, false>, conv_gather_kernel<1, 2, true>));
  else if (p.V == 4)
    B200_TRY(launch(conv_gather_kernel<1, 4, false>, conv_gather_kernel<2, 4, false>, conv_gather_kernel<1, 4, true>));
  else
    B200_TRY(launch(conv_gather_kernel<1, 8, false>, conv_gather_kernel<2, 8, false>, conv_gather_kernel<1, 8, true>));
#ifdef B200_TC_TIMING
  if (timing) {  // diagnostic: cycles of the roles and of their waits, averaged over blocks
    std::vector<long long> h((size_t)grid * 16);
    B200_CUDA(cudaStreamSynchronize(ctx->stream));
    B200_CUDA(cudaMemcpy(h.data(), a.dbg, h.size() * sizeof(long long), cudaMemcpyDeviceToHost));
    B200_CUDA(cudaFree(a.dbg));
    double s[16] = {0};
    for (int i = 0; i < grid; ++i)
      for (int k = 0; k < 16; ++k) s[k] += (double)h[(size_t)i * 16 + k] / grid * (k >= 12 ? CG : 1);
    int pairs = 0;
    for (int i = 0; i < p.nphases; ++i) pairs += p.ph[i].kslab;
    fprintf(stderr,
            "[tc-timing] gather %s CG %d S %d Z %d NP %d groups %d CS %d slabs %d k/slab %d ring %d grid %d units %d | mma %.0f (filter %.0f "
            "acc %.0f A %.0f) | converter %.0f (raw %.0f A %.0f) | loader %.0f (raw %.0f) | epilogue %.0f (wait %.0f)\n",
            for_dx ? "dx" : "fwd", CG, a.S, a.Z, a.NP, a.ngroups, a.CS, a.nslab, pairs, a.nf, grid, units, s[12], s[13], s[14], s[15],
            s[4], s[5], s[6], s[8], s[9], s[0], s[1]);
  }
#endif
  return 0;
}

}  // namespace

bool conv_gather_ok(const b200_ctx *ctx, const ConvGeom &g, int for_dx) {
  if (for_dx && (long long)g.HI * g.WI > 1 << 24) return false;
  return gather_plan(ctx, g, for_dx).ok;
}

size_t conv_gather_filter_floats(const b200_ctx *ctx, const ConvGeom &g, int for_dx) {
  return 3 * (size_t)gather_plan(ctx, g, for_dx).filt_words;
}

// filter blocks of the forward pass (wt_fwd) and / or of the dX pass (wt_dx) in one launch
int conv_gather_prep(b200_ctx *ctx, const ConvGeom &g, const float *W, float *wt_fwd, float *wt_dx) {
  if (!wt_fwd && !wt_dx) return 0;
  FilterSet s[2] = {};
  int n = 0;
  if (wt_fwd) s[n++] = filter_set(gather_plan(ctx, g, 0), g, 0, wt_fwd);
  if (wt_dx) s[n++] = filter_set(gather_plan(ctx, g, 1), g, 1, wt_dx);
  const long long total = s[0].total > s[1].total ? s[0].total : s[1].total;
  long long blocks = (total + 255) / 256;
  if (blocks > ctx->sm_count * 8) blocks = ctx->sm_count * 8;
  B200_TRY(launch_kernel(ctx, conv_gather_prep_kernel, dim3((unsigned)blocks, n), dim3(256), 0, 1, W, g.tbl, g.C, g.OC, g.KH,
                         g.KW, s[0], s[1]));
  return 0;
}

int conv_gather_fwd(b200_ctx *ctx, const ConvGeom &g, const float *in, const float *wt, const float *bias, float *out, int B,
                    int act) {
  return launch_conv_gather(ctx, gather_plan(ctx, g, 0), g, 0, in, wt, g.has_bias ? bias : nullptr, out, B, act);
}

int conv_gather_dx(b200_ctx *ctx, const ConvGeom &g, const float *dout, const float *wt, float *din, int B) {
  return launch_conv_gather(ctx, gather_plan(ctx, g, 1), g, 1, dout, wt, nullptr, din, B, B200_ACT_NONE);
}

int conv_gather_dx_blocks(const b200_ctx *ctx, const ConvGeom &g, int B) {
  return gather_shape(ctx, gather_plan(ctx, g, 1), B).blocks;
}

// Which kernels take the passes of a layer.  The gather kernels take what they can: on layers of 3 to 256
// channels, 7 to 64 pixels and 1 to 256 samples they were the fastest for 120 of 132 passes timed against the
// FFMA and general kernels; the others were narrow layers.  Two kinds of layer stay with other kernels:
//   dX into at most 4 channels: an MMA is 16 columns wide and would be three quarters padding, while
//     the FFMA kernel for few outputs reads each gradient once (32x32, 32 -> 3 channels, 5x5, 256 samples:
//     42 us against 104 us);
//   forward and dW of layers whose whole window has at most 96 / 128 values: the im2col kernels keep all
//     taps of a pixel in one operand row (same layer: forward 24 us against 32, dW with its sums 42 us against 44
//     with the window's columns folded into the channels).
ConvTcUse conv_tc_use(const b200_ctx *ctx, const ConvGeom &g, int algo) {
  ConvTcUse u = {false, false, false, false, false, false};
  if (algo == 1 || algo == 2 || (algo != 3 && ctx->conv_tensor_cores == 0)) return u;
  if (g.HI == g.KH && g.WI == g.KW && g.OH == 1 && g.OW == 1 && g.pad_t == 0 && g.pad_l == 0 && !g.tbl) {
    // one output pixel: nothing to gather, and 128 of them would be the inputs of 128 samples
    u.fc = true;
    return u;
  }
  const bool all = algo == 3 || ctx->conv_tensor_cores >= 2;
  const char *env = algo == 3 ? nullptr : getenv("B200_CONV_TC");
  const int m = env ? atoi(env) : 31;  // bit 0 forward, 1 dX, 2 dW, 3 im2col dW, 4 im2col forward
  u.fwd = (m & 1) && conv_gather_ok(ctx, g, 0);
  u.dx = (m & 2) && conv_gather_ok(ctx, g, 1) && (all || g.C > 4 || !conv_tiled_ok(g));
  u.dw = (m & 4) && conv_gather_dw_ok(ctx, g);
  if ((m & 8) && (!u.dw || g.C < 16) && conv_dw_small_ok(ctx, g)) {
    u.dw = false;
    u.dw_small = true;
  }
  if ((m & 16) && (!u.fwd || g.C < 16) && conv_fwd_small_ok(ctx, g)) {
    u.fwd = false;
    u.fwd_small = true;
  }
  return u;
}

}  // namespace b200
