// Forward convolution of layers with few input channels on the 5th-generation tensor cores
// (tcgen05), fp32-accurate through the 3xTF32 split.  Replaces the loops of
// kernels::conv2d_op_internal (tiny_dnn/core/kernels/conv2d_op_internal.h:13-74) for the first layer
// of a network (3 x 5 x 5 = 75 taps), where a 32-channel slab per tap would be almost all padding.
//
// GEMM form: D[pixel][o] = sum_k A[pixel][k] * W[o][k], k = (c*KH + ky)*KW + kx -- the reference's
// own weight order, so the filter needs no reordering, only the hi / lo split.
//   M = 128 pixels: 4 output rows x 32 columns of one image
//   N = out channels (padded to 16); hi and lo rows of the filter are neighbours in shared memory,
//       so A_hi x [W_hi | W_lo] is one instruction of width 2N; A_lo x W_hi is the second
//   K = taps in steps of 8; the filter K-major with the 128-byte swizzle, 32 taps per row
// A (the im2col rows of the tile) exists only in tensor memory: one TMA load brings the raw
// (4 + KH - 1) input rows of every channel (zero filled outside the image) into shared memory,
// sixteen converter warps gather each pixel's taps from them, split them and write the hi / lo
// values into the pixel's TMEM lane (tcgen05.st), from where the MMAs take their A operand -- the
// im2col matrix never passes through shared memory, whose bandwidth bounded the first form of this
// kernel.  The filter is split once per CTA and stays resident in shared memory.
// Warp roles: 0-7 epilogue (one TMEM lane = one pixel per thread, two warps share a lane quadrant and
// split the channels), 8-23 converters, 24 TMA producer + TMEM allocation, 25 MMA issuer.  Accumulators and A buffers are double buffered in tensor memory.
// Every load is CTA-local; every wait is bounded and a timeout sets the context's error word,
// frees tensor memory and returns.
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "tc_utils.cuh"

namespace b200 {

namespace {

constexpr int TFS_ROWS = 4;          // output rows per step
constexpr int TFS_PX = 32;           // output columns per step
constexpr int TFS_CONV_WARPS = 16;         // four warps per tile row: each takes every fourth quad of taps
constexpr int TFS_EPI_WARPS = 8;           // two per TMEM lane quadrant: each takes every other 16 channels
constexpr int TFS_THREADS = (TFS_EPI_WARPS + TFS_CONV_WARPS + 2) * 32;
constexpr int TFS_STAGES = 4;        // raw input tiles in flight
constexpr int TFS_MAX_KB = 3;        // 128-byte K blocks (32 taps each): 96 taps at most
constexpr size_t TFS_MIN_SMEM = 120 * 1024;  // ask for more than half an SM's shared memory: the kernel
                                             // takes all 512 TMEM columns, a second CTA would only wait

struct TcFwdSmallArgs {
  const float *W, *bias;
  const uint8_t *tbl;
  float *out;
  int *err;
  int C, OC, OCp, KH, KW, pad_t, pad_l;
  int OH, OW, nxb, nyb;
  int Kreal;    // C * KH * KW
  int ksteps;   // MMA steps of 8 taps
  int nkb;      // K blocks of 32 taps
  int bw, rows; // raw tile: floats per row, rows per channel
  int nsteps, nblocks;
  int act;
  int tmem_cols;
  long long *dbg;  // optional [blocks][12] cycle counters (B200_TC_TIMING=1), else nullptr
};

// four consecutive TMEM columns of the warp's 32 lanes
__device__ __forceinline__ void tmem_st4(uint32_t taddr, float a, float b, float c, float d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(taddr),
               "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(__float_as_uint(d))
               : "memory");
}

// tile coordinates of consecutive steps without a division per step
struct StepPos {
  int xb, yb, b;
  __device__ __forceinline__ void init(int s, int nxb, int nyb) {
    xb = s % nxb;
    const int t = s / nxb;
    yb = t % nyb;
    b = t / nyb;
  }
  __device__ __forceinline__ void next(int nxb, int nyb) {
    if (++xb == nxb) {
      xb = 0;
      if (++yb == nyb) {
        yb = 0;
        ++b;
      }
    }
  }
};

// 16 channels of one pixel: hi + lo parts, bias, activation, one store per channel plane
template <int ACT>
__device__ __forceinline__ void store16(float *dst, size_t plane, int n, const uint32_t *v, const uint32_t *w,
                                        const float *bv) {
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    float r = (__uint_as_float(v[q]) + __uint_as_float(w[q])) + bv[q];
    if (ACT == B200_ACT_RELU) r = fmaxf(0.f, r);
    if (ACT == B200_ACT_TANH) r = tanhf(r);
    if (q < n) dst[(size_t)q * plane] = r;
  }
}

__global__ void __launch_bounds__(TFS_THREADS, 1)
  conv_fwd_small_tc_kernel(const __grid_constant__ CUtensorMap x_map, const TcFwdSmallArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t WT = 2u * (uint32_t)a.OCp * 128u;               // one K block of the filter: hi rows, lo rows
  const uint32_t XBYTES = (uint32_t)(a.C * a.rows * a.bw * 4);
  const uint32_t XB = (XBYTES + 1023u) & ~1023u;
  const uint32_t STAGE = XB;                                     // one raw input tile
  uint8_t *wt = smem;                                            // [nkb][2*OCp][128 B]
  uint8_t *stage0 = smem + (size_t)a.nkb * WT;
  int *koff = reinterpret_cast<int *>(stage0 + (size_t)TFS_STAGES * STAGE);  // [ksteps*8]
  uint64_t *tma_full = reinterpret_cast<uint64_t *>(koff + TFS_MAX_KB * 32);
  uint64_t *raw_empty = tma_full + TFS_STAGES;
  uint64_t *a_full = raw_empty + TFS_STAGES;   // [2] A buffers in tensor memory
  uint64_t *a_empty = a_full + 2;
  uint64_t *acc_full = a_empty + 2;
  uint64_t *acc_empty = acc_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
  float *bias_s = reinterpret_cast<float *>(tmem_slot + 4);      // [OCp], zeros without a bias

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int s_begin = (int)((long long)blockIdx.x * a.nsteps / a.nblocks);
  const int s_end = (int)((long long)(blockIdx.x + 1) * a.nsteps / a.nblocks);
  constexpr int W_TMA = TFS_EPI_WARPS + TFS_CONV_WARPS, W_MMA = W_TMA + 1;
  if (tid == 0) {
    for (int s = 0; s < TFS_STAGES; ++s) {
      mbar_init(&tma_full[s], 1);
      mbar_init(&raw_empty[s], TFS_CONV_WARPS);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&a_full[s], TFS_CONV_WARPS);
      mbar_init(&a_empty[s], 1);
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], TFS_EPI_WARPS);
    }
    mbar_fence_init();
  }
  wait_for_previous_kernel();
  for (int o = tid; o < a.OCp; o += TFS_THREADS) bias_s[o] = (a.bias && o < a.OC) ? a.bias[o] : 0.f;
  if (warp == W_TMA) tmem_alloc(tmem_slot, (uint32_t)a.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // tensor memory columns: two accumulators of 2*OCp, then two A buffers of (hi | lo) x Kp
  const uint32_t Kp = (uint32_t)a.ksteps * 8u, tmem_a = tmem_base + 4u * (uint32_t)a.OCp;
  bool failed = false;

  if (warp == W_TMA && lane == 0) {
    // ---- TMA producer: the raw input rows of each step -------------------------------------------
    long long w = 0, t0 = tc_clock(), tq;
    StepPos pos;
    pos.init(s_begin, a.nxb, a.nyb);
    for (int s = s_begin; s < s_end; ++s, pos.next(a.nxb, a.nyb)) {
      const uint32_t i = s - s_begin, st = i % TFS_STAGES, use = i / TFS_STAGES;
      tq = tc_clock();
      if (use > 0 && !mbar_wait_bounded(&raw_empty[st], (use - 1) & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      if (a.dbg && s == s_end - 1) {
        a.dbg[blockIdx.x * 12 + 0] = tc_clock() - t0;
        a.dbg[blockIdx.x * 12 + 1] = w;
      }
      const int xs = (pos.xb * TFS_PX - a.pad_l) & ~3;  // aligned start column (floor to a multiple of 4)
      mbar_expect_tx(&tma_full[st], XBYTES);
      tma_load_4d(stage0 + (size_t)st * STAGE, &x_map, xs, pos.yb * TFS_ROWS - a.pad_t, 0, pos.b,
                  &tma_full[st]);
    }
  } else if (warp == W_MMA) {
    // ---- MMA issuer (the whole warp stays converged: see elect_one) ---
    const uint32_t idesc1 = umma_idesc_tf32(128, a.OCp), idesc2 = umma_idesc_tf32(128, 2 * a.OCp);
    const uint64_t b0 = umma_desc(smem_u32(wt), 16, 1024, 2);
    long long w = 0, w2 = 0, t0 = tc_clock(), tq;
    for (int s = s_begin; s < s_end; ++s) {
      const uint32_t i = s - s_begin, ab = i & 1;
      tq = tc_clock();
      if (!mbar_wait_warp(&a_full[ab], (i >> 1) & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      tq = tc_clock();
      if (i >= 2 && !mbar_wait_warp(&acc_empty[ab], ((i >> 1) - 1) & 1)) {
        failed = true;
        break;
      }
      w2 += tc_clock() - tq;
      if (a.dbg && lane == 0 && s == s_end - 1) {
        a.dbg[blockIdx.x * 12 + 2] = tc_clock() - t0;
        a.dbg[blockIdx.x * 12 + 3] = w;
        a.dbg[blockIdx.x * 12 + 4] = w2;
      }
      tc_fence_after();
      const uint32_t acc = tmem_base + ab * 2u * (uint32_t)a.OCp;
      const uint32_t ahi = tmem_a + ab * 2u * Kp, alo = ahi + Kp;
      // the descriptor of K step ks is the first one plus its byte offset / 16 in the address field
      if (elect_one()) {
#pragma unroll 4
        for (int ks = 0; ks < a.ksteps; ++ks) {
          const uint64_t b = b0 + (uint64_t)(((uint32_t)(ks >> 2) * WT + (uint32_t)(ks & 3) * 32u) >> 4);
          umma_tf32_ta(acc, ahi + ks * 8, b, idesc2, ks != 0);
          umma_tf32_ta(acc, alo + ks * 8, b, idesc1, 1);
        }
        umma_commit(&a_empty[ab]);
        umma_commit(&acc_full[ab]);
      }
      __syncwarp();
    }
  } else if (warp >= TFS_EPI_WARPS && warp < W_TMA) {
    // ---- converters ------------------------------------------------------------------------------
    const int ct = tid - TFS_EPI_WARPS * 32;
    constexpr int NCT = TFS_CONV_WARPS * 32;
    const int KK = a.KH * a.KW, nk = a.ksteps * 8;
    // tap -> offset in the raw tile (-1: padding tap)
    for (int k = ct; k < nk; k += NCT) {
      int off = -1;
      if (k < a.Kreal) {
        const int c = k / KK, r = k - c * KK, ky = r / a.KW, kx = r - ky * a.KW;
        off = (c * a.rows + ky) * a.bw + kx;
      }
      koff[k] = off;
    }
    // the filter: W[o][k] split into hi rows and lo rows of every K block
    for (int idx = ct; idx < a.OCp * a.nkb * 32; idx += NCT) {
      const int o = idx / (a.nkb * 32), k = idx - o * (a.nkb * 32);
      float v = 0.f;
      if (o < a.OC && k < a.Kreal && (!a.tbl || a.tbl[(k / KK) * a.OC + o])) v = a.W[(size_t)o * a.Kreal + k];
      float h, l;
      split_tf32_rn(v, h, l);
      const uint32_t kb = k >> 5, kk = k & 31;
      const uint32_t rh = o, rl = a.OCp + o;
      uint8_t *tile = wt + (size_t)kb * WT;
      *reinterpret_cast<float *>(tile + rh * 128u + (((kk >> 2) ^ (rh & 7)) << 4) + (kk & 3) * 4u) = h;
      *reinterpret_cast<float *>(tile + rl * 128u + (((kk >> 2) ^ (rl & 7)) << 4) + (kk & 3) * 4u) = l;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("bar.sync 1, %0;\n" ::"n"(NCT) : "memory");
    const int p = ct & 127, part = ct >> 7;                // pixel of the tile, which share of the tap quads
    const int pixoff = (p >> 5) * a.bw + (p & 31);
    const uint32_t lane_base = (uint32_t)(warp & 3) << 21;   // this warp's TMEM lanes: 32 * (warp % 4), in bits 16..
    const int nkq = a.ksteps * 2, nfull = a.Kreal >> 2;
    constexpr int NPART = TFS_CONV_WARPS / 4, NQ = (TFS_MAX_KB * 8 + NPART - 1) / NPART;
    int4 ko[NQ];  // raw-tile offsets of the tap quads this thread converts, the same in every step
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
      const int kq = part + j * NPART;
      ko[j] = kq < nkq ? *reinterpret_cast<const int4 *>(koff + kq * 4) : make_int4(-1, -1, -1, -1);
    }
    long long w = 0, w2 = 0, t0 = tc_clock(), tq;
    int xb = s_begin % a.nxb;
    for (int s = s_begin; s < s_end; ++s, xb = (xb + 1 == a.nxb) ? 0 : xb + 1) {
      const uint32_t i = s - s_begin, st = i % TFS_STAGES, use = i / TFS_STAGES, ab = i & 1;
      tq = tc_clock();
      if (!mbar_wait_bounded(&tma_full[st], use & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      tq = tc_clock();
      if (i >= 2 && !mbar_wait_bounded(&a_empty[ab], ((i >> 1) - 1) & 1)) {
        failed = true;
        break;
      }
      w2 += tc_clock() - tq;
      tc_fence_after();
      uint8_t *sp = stage0 + (size_t)st * STAGE;
      const int x0 = xb * TFS_PX;
      const int d = (x0 - a.pad_l) - ((x0 - a.pad_l) & ~3);
      const float *xr = reinterpret_cast<const float *>(sp) + d + pixoff;
      const uint32_t thi = tmem_a + ab * 2u * Kp + lane_base, tlo = thi + Kp;
#pragma unroll
      for (int j = 0; j < NQ; ++j) {
        const int kq = part + j * NPART;
        if (kq < nkq) {
          const int4 o4 = ko[j];
          float h[4], l[4];
          if (kq < nfull) {  // all four taps exist (uniform over the warp)
            split_tf32_rn(xr[o4.x], h[0], l[0]);
            split_tf32_rn(xr[o4.y], h[1], l[1]);
            split_tf32_rn(xr[o4.z], h[2], l[2]);
            split_tf32_rn(xr[o4.w], h[3], l[3]);
          } else {
            split_tf32_rn(o4.x >= 0 ? xr[o4.x] : 0.f, h[0], l[0]);
            split_tf32_rn(o4.y >= 0 ? xr[o4.y] : 0.f, h[1], l[1]);
            split_tf32_rn(o4.z >= 0 ? xr[o4.z] : 0.f, h[2], l[2]);
            split_tf32_rn(o4.w >= 0 ? xr[o4.w] : 0.f, h[3], l[3]);
          }
          tmem_st4(thi + (uint32_t)kq * 4u, h[0], h[1], h[2], h[3]);
          tmem_st4(tlo + (uint32_t)kq * 4u, l[0], l[1], l[2], l[3]);
        }
      }
      // the stores have landed in tensor memory: hand the A buffer over, give the raw tile back
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&a_full[ab]);
        mbar_arrive(&raw_empty[st]);
      }
    }
    if (a.dbg && ct == 0) {
      a.dbg[blockIdx.x * 12 + 5] = tc_clock() - t0;
      a.dbg[blockIdx.x * 12 + 6] = w;
      a.dbg[blockIdx.x * 12 + 7] = w2;
    }
  } else if (warp < TFS_EPI_WARPS) {
    // ---- epilogue: hi + lo parts, bias, activation, store ------------------------------------------
    const size_t plane = (size_t)a.OH * a.OW;
    long long w = 0, wl = 0, t0 = tc_clock(), tq;
    StepPos pos;
    pos.init(s_begin, a.nxb, a.nyb);
    for (int s = s_begin; s < s_end; ++s, pos.next(a.nxb, a.nyb)) {
      const uint32_t i = s - s_begin, ab = i & 1;
      tq = tc_clock();
      if (!mbar_wait_bounded(&acc_full[ab], (i >> 1) & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      if (a.dbg && tid == 0 && s == s_end - 1) {
        a.dbg[blockIdx.x * 12 + 8] = tc_clock() - t0;
        a.dbg[blockIdx.x * 12 + 9] = w;
      }
      tc_fence_after();
      const int b = pos.b;
      const int y = pos.yb * TFS_ROWS + (warp & 3), x = pos.xb * TFS_PX + lane;
      const bool inside = y < a.OH && x < a.OW;
      float *obase = a.out + (size_t)b * a.OC * plane + (size_t)y * a.OW + x;
      const uint32_t tacc = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + ab * 2u * (uint32_t)a.OCp;
      const int cfirst = (warp >> 2) * 16;
      if (cfirst >= a.OCp) {  // no channels for this warp: it only keeps step with the barrier
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[ab]);
      }
      for (int c0 = cfirst; c0 < a.OCp; c0 += 32) {
        uint32_t v[16], w[16];
        tq = tc_clock();
        tmem_ld16_nowait(tacc + (uint32_t)c0, v);
        tmem_ld16_nowait(tacc + (uint32_t)(a.OCp + c0), w);
        tmem_ld_wait();
        if (c0 + 32 >= a.OCp) {  // the buffer is read: the next step but one may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[ab]);
        }
        wl += tc_clock() - tq;
        float bv[16];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<float4 *>(bv + 4 * q) = *reinterpret_cast<const float4 *>(bias_s + c0 + 4 * q);
        if (inside) {  // one branch on the activation per 16 channels, not per element
          float *dst = obase + (size_t)c0 * plane;
          const int n = a.OC - c0;
          if (a.act == B200_ACT_RELU)
            store16<B200_ACT_RELU>(dst, plane, n, v, w, bv);
          else if (a.act == B200_ACT_TANH)
            store16<B200_ACT_TANH>(dst, plane, n, v, w, bv);
          else
            store16<B200_ACT_NONE>(dst, plane, n, v, w, bv);
        }
      }
      if (a.dbg && tid == 0 && s == s_end - 1) a.dbg[blockIdx.x * 12 + 10] = wl;
    }
  }
  if (failed && a.err) atomicExch(a.err, 6);
  tc_fence_before();
  __syncthreads();
  if (warp == W_TMA) tmem_dealloc(tmem_base, (uint32_t)a.tmem_cols);
}

int fwd_small_bw(const ConvGeom &g) { return (TFS_PX + g.KW - 1 + 3 + 3) & ~3; }

size_t fwd_small_smem(const ConvGeom &g, int OCp) {
  const int K = g.C * g.KH * g.KW, nkb = (K + 31) / 32;
  const size_t XB = ((size_t)g.C * (TFS_ROWS + g.KH - 1) * fwd_small_bw(g) * 4 + 1023) & ~(size_t)1023;
  const size_t need = 1024 + (size_t)nkb * 2 * OCp * 128 + TFS_STAGES * XB + TFS_MAX_KB * 32 * 4 +
                      (2 * TFS_STAGES + 8) * 8 + 16 + (size_t)OCp * 4 + 64;
  return need > TFS_MIN_SMEM ? need : TFS_MIN_SMEM;
}

// tensor memory columns: two accumulators (hi | lo parts) and two A buffers (hi | lo)
int fwd_small_tmem(const ConvGeom &g, int OCp) {
  const int Kp = (g.C * g.KH * g.KW + 7) / 8 * 8;
  return 4 * OCp + 4 * Kp;
}

int pow2_cols(int v) {
  int p = 32;
  while (p < v) p <<= 1;
  return p;
}

}  // namespace

// true when the im2col tensor-core forward kernel applies
bool conv_fwd_small_ok(const b200_ctx *ctx, const ConvGeom &g) {
  if (g.SH != 1 || g.SW != 1 || g.DH != 1 || g.DW != 1) return false;
  const int K = g.C * g.KH * g.KW;
  if (K > TFS_MAX_KB * 32 || g.OC > 64) return false;
  if (g.WI & 3) return false;                               // TMA strides are multiples of 16 bytes
  if (((size_t)g.HI * g.WI) & 3) return false;
  if (g.pad_t < 0 || g.pad_l < 0) return false;
  const int OCp = (g.OC + 15) / 16 * 16;
  if (fwd_small_tmem(g, OCp) > 512) return false;
  return fwd_small_smem(g, OCp) <= (size_t)ctx->smem_optin;
}

// forward (+ bias, activation) from the CHW input; no scratch
int conv_fwd_small(b200_ctx *ctx, const ConvGeom &g, const float *in, const float *W, const float *bias, float *out,
                   int B, int act) {
  if (B == 0) return 0;
  const int OCp = (g.OC + 15) / 16 * 16, bw = fwd_small_bw(g);
  EncodeTiledFn fn = encode_fn();
  B200_REQUIRE(fn != nullptr, "cuTensorMapEncodeTiled is not available from the driver");
  TcFwdSmallArgs a;
  a.rows = TFS_ROWS + g.KH - 1;
  CUtensorMap x_map;
  {
    cuuint64_t dims[4] = {(cuuint64_t)g.WI, (cuuint64_t)g.HI, (cuuint64_t)g.C, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)g.WI * 4, (cuuint64_t)g.HI * g.WI * 4, (cuuint64_t)g.C * g.HI * g.WI * 4};
    cuuint32_t box[4] = {(cuuint32_t)bw, (cuuint32_t)a.rows, (cuuint32_t)g.C, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(&x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(in), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d) for the input rows", (int)r);
  }
  a.W = W;
  a.bias = g.has_bias ? bias : nullptr;
  a.tbl = g.tbl;
  a.out = out;
  a.err = ctx->dev_err;
  a.C = g.C;
  a.OC = g.OC;
  a.OCp = OCp;
  a.KH = g.KH;
  a.KW = g.KW;
  a.pad_t = g.pad_t;
  a.pad_l = g.pad_l;
  a.OH = g.OH;
  a.OW = g.OW;
  a.nxb = ceil_div(g.OW, TFS_PX);
  a.nyb = ceil_div(g.OH, TFS_ROWS);
  a.Kreal = g.C * g.KH * g.KW;
  a.ksteps = (a.Kreal + 7) / 8;
  a.nkb = (a.Kreal + 31) / 32;
  a.bw = bw;
  a.nsteps = B * a.nyb * a.nxb;
  a.nblocks = a.nsteps < ctx->sm_count ? a.nsteps : ctx->sm_count;
  a.act = act;
  a.tmem_cols = pow2_cols(fwd_small_tmem(g, OCp));
  const size_t smem = fwd_small_smem(g, OCp);
  B200_REQUIRE(smem <= (size_t)ctx->smem_optin, "conv_fwd_small: the tiles do not fit shared memory");
  B200_CUDA(cudaFuncSetAttribute(conv_fwd_small_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  a.dbg = nullptr;
#ifdef B200_TC_TIMING
  static const bool timing = getenv("B200_TC_TIMING") != nullptr;
  if (timing) B200_CUDA(cudaMalloc(&a.dbg, (size_t)a.nblocks * 12 * sizeof(long long)));
#endif
  B200_TRY(launch_kernel(ctx, conv_fwd_small_tc_kernel, dim3(a.nblocks), dim3(TFS_THREADS), smem, 1, x_map, a));
#ifdef B200_TC_TIMING
  if (timing) {  // diagnostic: cycles of the four roles and of their waits, averaged over blocks
    std::vector<long long> h((size_t)a.nblocks * 12);
    B200_CUDA(cudaStreamSynchronize(ctx->stream));
    B200_CUDA(cudaMemcpy(h.data(), a.dbg, h.size() * sizeof(long long), cudaMemcpyDeviceToHost));
    B200_CUDA(cudaFree(a.dbg));
    double s[12] = {0};
    for (int i = 0; i < a.nblocks; ++i)
      for (int k = 0; k < 12; ++k) s[k] += (double)h[(size_t)i * 12 + k] / a.nblocks;
    fprintf(stderr,
            "[tc-timing] fwd small: steps/block %.1f: producer %.0f clk (wait raw %.0f), mma %.0f (wait operands %.0f, "
            "accumulator %.0f), converter %.0f (wait tma %.0f, tile free %.0f), epilogue %.0f (wait %.0f, tmem loads %.0f)\n",
            (double)a.nsteps / a.nblocks, s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8], s[9], s[10]);
  }
#endif
  return 0;
}

// ---- dW of layers with few input channels: explicit transposed im2col operand -----------------
//
// When in_c * KH * KW <= 128 (the first layer of a network: 3 x 5 x 5 = 75) a 32-channel slab would
// be almost all padding.  Here the contraction still runs over pixels, but both operands are
// K-major with 32 consecutive pixels of one output row per 128-byte row:
//   B[o][p]  = dY[b][o][y][x0 + p]                  a TMA tile straight from the CHW gradient
//   A[k][p]  = Xpad[b][c][y + ky][x0 + p + kx]      k = (c*KH + ky)*KW + kx: a converter thread owns
//              tap k, gathers its pixels from the raw input rows (one TMA tile), splits them and
//              writes hi / lo into TMEM lane k (tcgen05.st); the MMAs take A from tensor memory, so
//              the im2col rows never pass through shared memory
//   D[k][o] += A * B^T                              M = 128 (k padded), N = out channels, 4 k-steps
// so dW needs 8 MMAs per 32 pixels.  The converter warps also split B into hi / lo in place and
// keep the bias-gradient sums.  Per-CTA partial results are merged in fixed order afterwards.

namespace {

// Arguments of the finishing pass of conv_dw_small_tc_kernel: sums the partial rows in fixed order and
// stores the totals in the reference layout.  Elements [0, row_w) are weight-gradient entries [k][o];
// the bias-gradient sums come from `bsrc` (bs_rows rows of bs_stride floats, entry bs_off + o of each).
// Unconnected pairs get no gradient.
struct DwFinishArgs {
  const float *part;
  long long part_stride;
  int splits;
  const float *bsrc;
  long long bs_stride, bs_off;
  int bs_rows;
  float *dW, *db;
  int row_w;
  int C, OC, OCp, KH, KW;
  const uint8_t *tbl;
  int accumulate;
};

// One block of the finishing pass (DwFinishArgs): 8 row lanes per
// element, lane k adds rows k, k+8, ... in order, lanes combined in order.
__device__ __forceinline__ void dw_finish_block(const DwFinishArgs &a, const int block) {
  constexpr int RL = 8;  // row lanes
  __shared__ float lanes[RL][33];
  __shared__ float tree[256];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int wblocks = (a.row_w + 31) / 32;
  if (block >= wblocks) {
    // bias gradient: one block per output channel; its many short partial rows are spread over
    // all 256 threads (thread k adds rows k, k+256, ... in order), combined by a fixed tree
    const int o = block - wblocks, t = ty * 32 + tx;
    if (a.db == nullptr || o >= a.OC) return;
    const float *src = a.bsrc + a.bs_off + o;
    float s = 0.f;
    for (int r = t; r < a.bs_rows; r += 256) s += src[(size_t)r * a.bs_stride];
    tree[t] = s;
    __syncthreads();
#pragma unroll
    for (int w = 128; w > 0; w >>= 1) {
      if (t < w) tree[t] += tree[t + w];
      __syncthreads();
    }
    if (t == 0) a.db[o] = a.accumulate ? a.db[o] + tree[0] : tree[0];
    return;
  }
  const int e = block * 32 + tx;
  float s0 = 0.f, s1 = 0.f;
  if (e < a.row_w) {
    const float *src = a.part + e;
    int r = ty;
    for (; r + RL < a.splits; r += 2 * RL) {
      s0 += src[(size_t)r * a.part_stride];
      s1 += src[(size_t)(r + RL) * a.part_stride];
    }
    if (r < a.splits) s0 += src[(size_t)r * a.part_stride];
  }
  lanes[ty][tx] = s0 + s1;
  __syncthreads();
  if (ty == 0 && e < a.row_w) {
    float s = lanes[0][tx];
#pragma unroll
    for (int k = 1; k < RL; ++k) s += lanes[k][tx];
    const int k = e / a.OCp, KK = a.KH * a.KW, o = e - k * a.OCp, inc = k / KK;
    const int t = k - inc * KK, ky = t / a.KW, kx = t - ky * a.KW;
    if (o < a.OC && inc < a.C) {
      if (a.tbl && !a.tbl[inc * a.OC + o]) s = 0.f;
      float *d = a.dW + (((size_t)o * a.C + inc) * a.KH + ky) * a.KW + kx;
      *d = a.accumulate ? *d + s : s;
    }
  }
}

__global__ void __launch_bounds__(256) dw_finish_kernel(const DwFinishArgs a) {
  after_previous_kernel();
  dw_finish_block(a, (int)blockIdx.x);
}

int dw_finish_blocks(const DwFinishArgs &a) { return (a.row_w + 31) / 32 + (a.db != nullptr ? a.OC : 0); }

int launch_dw_finish(b200_ctx *ctx, const DwFinishArgs &a) {
  B200_TRY(launch_kernel(ctx, dw_finish_kernel, dim3(dw_finish_blocks(a)), dim3(32, 8), 0, 1, a));
  return 0;
}

}  // namespace

namespace {

constexpr int TCS_MAX_STAGES = 4;     // gradient tile + raw input rows per stage: a few KB each
constexpr int TCS_PX = 32;          // pixels per step (one 128-byte operand row)
constexpr int TCS_GROUPS = 2;       // converter groups; group g converts the steps i with i % 2 == g
constexpr int TCS_GROUP_WARPS = 8;
static_assert(TCS_GROUPS <= 2, "a group's first step must be the first use of its stage: stages >= groups");
constexpr int TCS_CONV_WARPS = TCS_GROUPS * TCS_GROUP_WARPS;  // then one TMA warp and one MMA warp
constexpr int TCS_THREADS = (TCS_CONV_WARPS + 2) * 32;

struct TcDwSmallArgs {
  float *part;          // [ksplits][row] with row = 128 * OCp (D[k][o]) + OCp (bias sums)
  int *err;
  int C, OC, OCp, KH, KW, pad_t, pad_l;
  int OH, OW, nxb;      // output extent, 32-pixel blocks per output row
  int Kreal;            // C * KH * KW
  int bw;               // floats per raw input row in shared memory
  int nsteps, ksplits;
  int nst;              // pipeline stages
  int tmem_cols;        // accumulator 2*OCp, then two A buffers of 32 hi + 32 lo columns
  long long row;
  long long *dbg;       // [blocks][8] cycle counters in a build with -DB200_TC_TIMING, else nullptr
};

__global__ void __launch_bounds__(TCS_THREADS, 1)
  conv_dw_small_tc_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap dy_map,
                          const TcDwSmallArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t BB = (uint32_t)a.OCp * 128u;           // B tile (hi or lo)
  const uint32_t XB = ((uint32_t)(a.C * a.KH * a.bw * 4) + 1023u) & ~1023u;  // raw input rows
  const uint32_t STAGE = 2 * BB + XB;
  uint64_t *tma_full = reinterpret_cast<uint64_t *>(smem + (size_t)a.nst * STAGE);
  uint64_t *op_full = tma_full + TCS_MAX_STAGES;
  uint64_t *op_empty = op_full + TCS_MAX_STAGES;
  uint64_t *a_empty = op_empty + TCS_MAX_STAGES;   // [2] A buffers in tensor memory, one per converter group
  uint64_t *accum = a_empty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum + 1);
  float *bsum_s = reinterpret_cast<float *>(tmem_slot + 4);   // [group][8 pixel quads][OCp] bias partials

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int s_begin = (int)((long long)blockIdx.x * a.nsteps / a.ksplits);
  const int s_end = (int)((long long)(blockIdx.x + 1) * a.nsteps / a.ksplits);
  if (tid == 0) {
    for (int s = 0; s < a.nst; ++s) {
      mbar_init(&tma_full[s], 1);
      mbar_init(&op_full[s], TCS_CONV_WARPS);
      mbar_init(&op_empty[s], 1);
    }
    mbar_init(&a_empty[0], 1);
    mbar_init(&a_empty[1], 1);
    mbar_init(accum, 1);
    mbar_fence_init();
  }
  wait_for_previous_kernel();
  if (warp == TCS_CONV_WARPS) tmem_alloc(tmem_slot, (uint32_t)a.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_a = tmem_base + 2u * (uint32_t)a.OCp;   // A buffer of group g: 64 columns from tmem_a + 64 g
  bool failed = false;

  if (warp == TCS_CONV_WARPS && lane == 0) {
    // ---- TMA producer: raw input rows and the gradient tile of each step ----------------------
    long long w = 0, t0 = tc_clock(), tq;
    for (int s = s_begin; s < s_end; ++s) {
      const uint32_t i = s - s_begin, st = i % a.nst, use = i / a.nst;
      tq = tc_clock();
      if (use > 0 && !mbar_wait_bounded(&op_empty[st], (use - 1) & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      if (a.dbg && s == s_end - 1) {
        a.dbg[blockIdx.x * 8 + 0] = tc_clock() - t0;
        a.dbg[blockIdx.x * 8 + 1] = w;
      }
      const int xb = s % a.nxb, by = s / a.nxb, y = by % a.OH, b = by / a.OH;
      const int x0 = xb * TCS_PX;
      const int xs = (x0 - a.pad_l) & ~3;  // aligned start column of the raw rows (floor to 4)
      uint8_t *p = smem + (size_t)st * STAGE;
      mbar_expect_tx(&tma_full[st], BB + (uint32_t)(a.C * a.KH * a.bw * 4));
      tma_load_4d(p, &dy_map, x0, 0, y, b, &tma_full[st]);
      tma_load_4d(p + 2 * BB, &x_map, xs, y - a.pad_t, 0, b, &tma_full[st]);
    }
  } else if (warp == TCS_CONV_WARPS + 1) {
    // ---- MMA issuer (the whole warp stays converged: see elect_one) ---
    // the hi and lo gradient tiles are neighbours in shared memory: A_hi * [B_hi | B_lo] is one
    // instruction of width 2*OCp (columns OCp.. hold the A_hi*B_lo part, added in the epilogue)
    const uint32_t idesc1 = umma_idesc_tf32(128, a.OCp), idesc2 = umma_idesc_tf32(128, 2 * a.OCp);
    long long w = 0, t0 = tc_clock(), tq;
    for (int s = s_begin; s < s_end && !failed; ++s) {
      const uint32_t i = s - s_begin, st = i % a.nst;
      tq = tc_clock();
      if (!mbar_wait_warp(&op_full[st], (i / a.nst) & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      if (a.dbg && lane == 0 && s == s_end - 1) {
        a.dbg[blockIdx.x * 8 + 2] = tc_clock() - t0;
        a.dbg[blockIdx.x * 8 + 3] = w;
      }
      tc_fence_after();
      const uint64_t b0 = umma_desc(smem_u32(smem + (size_t)st * STAGE), 16, 1024, 2);
      const uint32_t ta = tmem_a + (i & 1u) * 64u;
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          umma_tf32_ta(tmem_base, ta + k4 * 8, b0 + k4 * 2, idesc2, (i | k4) != 0);
          umma_tf32_ta(tmem_base, ta + 32 + k4 * 8, b0 + k4 * 2, idesc1, 1);
        }
        umma_commit(&op_empty[st]);
        umma_commit(&a_empty[i & 1u]);
      }
      __syncwarp();
    }
    if (!failed && elect_one()) umma_commit(accum);
  } else if (warp < TCS_CONV_WARPS) {
    // ---- converters: im2col rows and the hi / lo split, then the epilogue ----------------------
    const int KK = a.KH * a.KW;
    const int grp = warp / TCS_GROUP_WARPS, gtid = tid - grp * (TCS_GROUP_WARPS * 32);
    constexpr int NCT = TCS_GROUP_WARPS * 32;  // threads of one group
    // A: this thread owns tap k = its TMEM lane and half of the step's 32 pixels (two warps of a
    // group share a lane quadrant); taps beyond the real ones are written as zeros
    static_assert(TCS_GROUP_WARPS == 8, "two warps per TMEM lane quadrant in every converter group");
    const int k = 32 * (warp & 3) + lane, phalf = ((warp - grp * TCS_GROUP_WARPS) >> 2) * 16;
    int soff = -1;  // floats into the raw rows (without the step's column offset)
    if (k < a.Kreal) {
      const int c = k / KK, r = k - c * KK, ky = r / a.KW, kx = r - ky * a.KW;
      soff = (c * a.KH + ky) * a.bw + kx + phalf;
    }
    const uint32_t ta_thread = tmem_a + (uint32_t)grp * 64u + ((uint32_t)(warp & 3) << 21) + (uint32_t)phalf;
    constexpr int NB = 128 * 8 / NCT;  // at most 128 out channels x 8 quads per step
    float bacc[NB];                    // bias partials of the (o, quad) items this thread owns
#pragma unroll
    for (int q = 0; q < NB; ++q) bacc[q] = 0.f;
    long long w = 0, t0 = tc_clock(), tq;
    // Every converter warp observes every step's barrier, in order, and takes part in the
    // hand-over, although only the step's group converts: a warp that skipped phases of an
    // mbarrier could no longer tell one phase from the one two later (the wait is by parity).
    for (int s = s_begin; s < s_end; ++s) {
      const uint32_t i = s - s_begin, st = i % a.nst;
      tq = tc_clock();
      if (!mbar_wait_bounded(&tma_full[st], (i / a.nst) & 1)) {
        failed = true;
        break;
      }
      w += tc_clock() - tq;
      if ((int)(i % TCS_GROUPS) != grp) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&op_full[st]);
        continue;
      }
      // this group's A buffer was read by the MMAs of its previous step
      if (i >= 2 && !mbar_wait_bounded(&a_empty[grp], ((i >> 1) - 1) & 1)) {
        failed = true;
        break;
      }
      tc_fence_after();
      uint8_t *p = smem + (size_t)st * STAGE;
      const int x0 = (s % a.nxb) * TCS_PX;
      const int d = (x0 - a.pad_l) - ((x0 - a.pad_l) & ~3);  // offset of the first needed column
      const float *xr = reinterpret_cast<const float *>(p + 2 * BB) + d;
      {
        uint32_t h[16], l[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          float hv, lv;
          split_tf32_rn(soff >= 0 ? xr[soff + q] : 0.f, hv, lv);
          h[q] = __float_as_uint(hv);
          l[q] = __float_as_uint(lv);
        }
        tmem_st16(ta_thread, h);
        tmem_st16(ta_thread + 32, l);
      }
      // B: split the gradient tile in place (hi) and into the lo tile; bias partial sums
#pragma unroll
      for (int slot = 0; slot < NB; ++slot) {
        const int it = gtid + NCT * slot;
        if (it < a.OCp * 8) {
          const int o = it >> 3, quad = it & 7;
          const uint32_t off = (uint32_t)o * 128u + (uint32_t)((quad ^ (o & 7)) << 4);
          float4 v = *reinterpret_cast<float4 *>(p + off);
          float h[4], l[4];
          split_tf32_rn(v.x, h[0], l[0]);
          split_tf32_rn(v.y, h[1], l[1]);
          split_tf32_rn(v.z, h[2], l[2]);
          split_tf32_rn(v.w, h[3], l[3]);
          *reinterpret_cast<float4 *>(p + off) = make_float4(h[0], h[1], h[2], h[3]);
          *reinterpret_cast<float4 *>(p + BB + off) = make_float4(l[0], l[1], l[2], l[3]);
          bacc[slot] += (v.x + v.y) + (v.z + v.w);
        }
      }
      // generic-proxy writes -> visible to the tensor core (async proxy); the TMEM stores have
      // landed; then hand over
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[st]);
    }
    if (a.dbg && tid == 0) {
      a.dbg[blockIdx.x * 8 + 4] = tc_clock() - t0;
      a.dbg[blockIdx.x * 8 + 5] = w;
    }
    // ---- epilogue ------------------------------------------------------------------------------
    float *row = a.part + (size_t)blockIdx.x * a.row;
#pragma unroll
    for (int slot = 0; slot < NB; ++slot) {
      const int it = gtid + NCT * slot;
      if (it < a.OCp * 8) bsum_s[(grp * 8 + (it & 7)) * a.OCp + (it >> 3)] = bacc[slot];
    }
    asm volatile("bar.sync 1, %0;\n" ::"n"(TCS_CONV_WARPS * 32) : "memory");
    for (int o = tid; o < a.OCp; o += TCS_CONV_WARPS * 32) {
      float t = bsum_s[o];
#pragma unroll
      for (int q = 1; q < TCS_GROUPS * 8; ++q) t += bsum_s[q * a.OCp + o];
      row[(size_t)128 * a.OCp + o] = t;
    }
    if (warp < 4 && s_end > s_begin && !failed) {
      if (!mbar_wait_bounded(accum, 0)) failed = true;
      tc_fence_after();
    }
    if (warp < 4 && !failed) {  // one warp per TMEM lane quadrant
      const int k = warp * 32 + lane;
      for (int c0 = 0; c0 < a.OCp; c0 += 16) {
        float v[16];
        if (s_end > s_begin) {
          float w[16];
          tmem_ld16(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
          tmem_ld16(tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(a.OCp + c0), w);
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] += w[q];
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] = 0.f;
        }
        float4 *dst = reinterpret_cast<float4 *>(row + (size_t)k * a.OCp + c0);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
    }
  }
  if (failed && a.err) atomicExch(a.err, 5);
  tc_fence_before();
  __syncthreads();
  if (warp == TCS_CONV_WARPS) tmem_dealloc(tmem_base, (uint32_t)a.tmem_cols);
}

size_t dw_small_stage(const ConvGeom &g, int OCp, int bw) {
  size_t XB = ((size_t)g.C * g.KH * bw * 4 + 1023) & ~(size_t)1023;
  return 2 * (size_t)OCp * 128 + XB;
}

size_t dw_small_fixed(int OCp) {
  return 1024 + (3 * TCS_MAX_STAGES + 3) * 8 + 32 + (size_t)TCS_GROUPS * 8 * OCp * 4 + 64;
}

// pipeline stages that fit (0: the kernel does not fit)
int dw_small_stages(const b200_ctx *ctx, const ConvGeom &g, int OCp, int bw) {
  size_t fixed = dw_small_fixed(OCp), stage = dw_small_stage(g, OCp, bw);
  // at least as many stages as converter groups: a group waiting for the second use of a stage
  // before its first use has happened would see the barrier's parity as already satisfied
  if (ctx->smem_optin < fixed + TCS_GROUPS * stage) return 0;
  size_t n = (ctx->smem_optin - fixed) / stage;
  return (int)(n > TCS_MAX_STAGES ? TCS_MAX_STAGES : n);
}

int dw_small_bw(const ConvGeom &g) { return (TCS_PX + g.KW - 1 + 3 + 3) & ~3; }

}  // namespace

// true when the small-input-channel dW kernel applies
bool conv_dw_small_ok(const b200_ctx *ctx, const ConvGeom &g) {
  if (g.SH != 1 || g.SW != 1 || g.DH != 1 || g.DW != 1) return false;
  if (g.C * g.KH * g.KW > 128 || g.OC > 128) return false;
  if ((g.WI & 3) || (g.OW & 3)) return false;                 // TMA strides are multiples of 16 bytes
  if (((size_t)g.HI * g.WI) & 3 || ((size_t)g.OH * g.OW) & 3) return false;
  if (g.pad_t < 0 || g.pad_l < 0) return false;
  if (g.OH + g.KH - 1 < g.HI + g.pad_t || g.OW + g.KW - 1 < g.WI + g.pad_l) return false;  // windows over all of it
  const int OCp = (g.OC + 15) / 16 * 16;
  return dw_small_stages(ctx, g, OCp, dw_small_bw(g)) >= TCS_GROUPS;
}

int conv_dw_small_splits(const b200_ctx *ctx, const ConvGeom &g, int B) {
  long long nsteps = (long long)B * g.OH * ceil_div(g.OW, TCS_PX);
  return (int)(nsteps < ctx->sm_count ? nsteps : ctx->sm_count);
}

size_t conv_dw_small_floats(const b200_ctx *ctx, const ConvGeom &g, int B) {
  const int OCp = (g.OC + 15) / 16 * 16;
  return ((size_t)conv_dw_small_splits(ctx, g, B) + 1) * ((size_t)129 * OCp);
}

// dW (+ db when the layer has a bias) from the CHW input and gradient; `part` holds conv_dw_small_floats
int conv_dw_small(b200_ctx *ctx, const ConvGeom &g, const float *in, const float *dout, int B, float *part,
                  float *dW, float *db, int accumulate) {
  const int OCp = (g.OC + 15) / 16 * 16, bw = dw_small_bw(g);
  EncodeTiledFn fn = encode_fn();
  B200_REQUIRE(fn != nullptr, "cuTensorMapEncodeTiled is not available from the driver");
  CUtensorMap x_map, dy_map;
  {
    cuuint64_t dims[4] = {(cuuint64_t)g.WI, (cuuint64_t)g.HI, (cuuint64_t)g.C, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)g.WI * 4, (cuuint64_t)g.HI * g.WI * 4, (cuuint64_t)g.C * g.HI * g.WI * 4};
    cuuint32_t box[4] = {(cuuint32_t)bw, (cuuint32_t)g.KH, (cuuint32_t)g.C, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(&x_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(in), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d) for the input rows", (int)r);
  }
  {
    // dimensions ordered (x, o, y, b) so that one box is the K-major tile [o][32 pixels]
    cuuint64_t dims[4] = {(cuuint64_t)g.OW, (cuuint64_t)g.OC, (cuuint64_t)g.OH, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)g.OH * g.OW * 4, (cuuint64_t)g.OW * 4, (cuuint64_t)g.OC * g.OH * g.OW * 4};
    cuuint32_t box[4] = {TCS_PX, (cuuint32_t)OCp, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(&dy_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(dout), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d) for the gradient tiles", (int)r);
  }
  TcDwSmallArgs a;
  a.part = part;
  a.err = ctx->dev_err;
  a.C = g.C;
  a.OC = g.OC;
  a.OCp = OCp;
  a.KH = g.KH;
  a.KW = g.KW;
  a.pad_t = g.pad_t;
  a.pad_l = g.pad_l;
  a.OH = g.OH;
  a.OW = g.OW;
  a.nxb = ceil_div(g.OW, TCS_PX);
  a.Kreal = g.C * g.KH * g.KW;
  a.bw = bw;
  a.nsteps = B * g.OH * a.nxb;
  a.ksplits = conv_dw_small_splits(ctx, g, B);
  a.nst = dw_small_stages(ctx, g, OCp, bw);
  B200_REQUIRE(a.nst >= TCS_GROUPS, "conv_dw_small: the tiles do not fit shared memory");
  a.tmem_cols = pow2_cols(2 * OCp + 128);
  a.row = (long long)129 * OCp;
  const size_t smem = dw_small_fixed(OCp) + (size_t)a.nst * dw_small_stage(g, OCp, bw);
  B200_CUDA(cudaFuncSetAttribute(conv_dw_small_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  a.dbg = nullptr;
#ifdef B200_TC_TIMING
  static const bool timing = getenv("B200_TC_TIMING") != nullptr;
  if (timing) B200_CUDA(cudaMalloc(&a.dbg, (size_t)a.ksplits * 8 * sizeof(long long)));
#endif
  B200_TRY(launch_kernel(ctx, conv_dw_small_tc_kernel, dim3(a.ksplits), dim3(TCS_THREADS), smem, 1, x_map, dy_map, a));
#ifdef B200_TC_TIMING
  if (timing) {  // diagnostic: cycles of the three roles and of their waits, averaged over blocks
    std::vector<long long> h((size_t)a.ksplits * 8);
    B200_CUDA(cudaStreamSynchronize(ctx->stream));
    B200_CUDA(cudaMemcpy(h.data(), a.dbg, h.size() * sizeof(long long), cudaMemcpyDeviceToHost));
    B200_CUDA(cudaFree(a.dbg));
    double s[8] = {0};
    for (int i = 0; i < a.ksplits; ++i)
      for (int k = 0; k < 8; ++k) s[k] += (double)h[(size_t)i * 8 + k] / a.ksplits;
    fprintf(stderr,
            "[tc-timing] dW small: steps/block %.1f stages %d: producer %.0f clk (wait %.0f), mma %.0f (wait %.0f), "
            "converter group 0 %.0f (wait %.0f)\n",
            (double)a.nsteps / a.ksplits, a.nst, s[0], s[1], s[2], s[3], s[4], s[5]);
  }
#endif
  DwFinishArgs f;
  f.part = part;
  f.part_stride = a.row;
  f.splits = a.ksplits;
  f.bsrc = part;            // the bias sums are the last OCp entries of every partial row
  f.bs_stride = a.row;
  f.bs_off = (long long)128 * OCp;
  f.bs_rows = a.ksplits;
  f.dW = dW;
  f.db = g.has_bias ? db : nullptr;
  f.row_w = 128 * OCp;
  f.C = g.C;
  f.OC = g.OC;
  f.OCp = OCp;
  f.KH = g.KH;
  f.KW = g.KW;
  f.tbl = g.tbl;
  f.accumulate = accumulate;
  B200_TRY(launch_dw_finish(ctx, f));
  return 0;
}

}  // namespace b200
