// Weight and bias gradient of a convolution on the 5th-generation tensor cores (tcgen05), fp32-accurate,
// straight from the CHW tensors.  Replaces the loops of kernels::conv2d_grad_op_internal
// (tiny_dnn/core/kernels/conv2d_op_internal.h:130-169 dW, :172-179 db) and the per-sample rows that
// edge::merge_grads adds up (tiny_dnn/node.h:89-103).
//
//   dW[o][c][ky][kx] = sum over output pixels (y, x) of  dY[o][y][x] * X[c][y * SH + ky - pad][x * SW + kx - pad]
//
//   M = 128 TMEM lanes: OB output channels x J window rows.  Lane (j, o) holds dY[o] shifted down by j rows, so
//       the same input row serves the window row ky0 + SH * j of lane j: layers with few output channels
//       still fill the lanes, and the input of a block needs no extra rows
//   N = CB input channels (64, 32 or 16); one MMA and one accumulator for every (window-row group, block of
//       channels, window column) of the CTA, as many as 384 TMEM columns hold: each serves from the same
//       loaded input rows, and it is the loads that would bound the kernel otherwise
//   K = pixels: groups of 8 along an output row, two groups per step of 16
// Every operand is split into three bf16 parts as in conv_gather.cu.  The small products of a step have accumulators of
// their own where the columns are there for both (`lo`); in wide layers all six go to one, six additions a step to a chain,
// whose truncations are the error: 3.7e-5 at 56x56, 64 -> 64, 3x3, 256 samples, 2200 additions, where narrow layers have
// 2e-7 to 8e-7.
// The input lies in shared memory pixel by pixel (a row of CB channels per place) and is the
// MN-major B operand: a window column is a start address that many rows further on, because the swizzle is
// a function of the address.  A strided layer's places are stored one residue after the other, which makes
// a window column's places consecutive again.  The gradient lies channel by channel, eight pixels in 16
// bytes, from where gather warps store it into tensor memory.
// The pixels are cut into slices, one per CTA; conv_gather_dw_finish_kernel adds the partial sums in order.
//
// What bounds it: the tensor pipe (12 MMAs of CB / 2 cycles, 18 at least, per accumulator and 32 pixels) or its issuers
// (about 720 cycles for those 12) where the lanes are full; what an SM gets from L2 (about 18 bytes a cycle) where few
// accumulators share the loads; in calls of a few stages a block the first load, the partial sums' way to memory and the
// pass that adds them up, a third of the time of the CIFAR-10 network's layers.  The loads of the next stage are in flight
// in registers while this one is multiplied.
// Warp roles: 0-15 loaders, 16-19 gather (one per TMEM lane quadrant) and epilogue, 20-24 MMA issuers (an even share of
// the accumulators each, no more of them than that takes).  Every wait is bounded; a timeout sets the context's error word, frees tensor
// memory and returns.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "tc_utils.cuh"

namespace b200 {

namespace {

constexpr int DW_LOAD_WARPS = 16, DW_LOAD_THREADS = DW_LOAD_WARPS * 32;
constexpr int DW_W_GATHER = DW_LOAD_WARPS, DW_W_MMA = DW_W_GATHER + 4;
constexpr int DW_ISSUERS = 5;        // a warp's 12 instructions of an accumulator and unit take longer than their MMAs, and 5 x 5
                                     // windows have five accumulators: with four issuers one of them had two
constexpr int DW_THREADS = (DW_W_MMA + DW_ISSUERS) * 32;
constexpr int DW_A_COLS = 48, DW_D_COLS = 384;  // accumulators, then two 32-pixel units of A
constexpr int DW_YB = 3, DW_XB = 2;  // gradient items and input items a loader thread has in flight
constexpr int DW_MAX_YITEMS = 4096;  // gradient items of a stage
constexpr int DW_MAX_STAGES = 4;
constexpr int DW_MAX_ADDS = 24576;   // additions to an accumulator
constexpr int DW_MAX_KGROUPS = 48;  // window-row groups x window-column groups

// One group of window rows and columns: rows ky0 + SH * (i * J + j) (i < nky, j < J, below KH), columns kx0 ..
struct DwKGroup {
  int ky0, nky, kx0, nkx;
  int splits;         // pixel slices of a (group, channel block) unit
  int first;          // first block; ocb * ccb * splits blocks (ccb: blocks of NB * CB channels)
  long long part0;    // float offset of the partial sums
};

// Layers of few input channels: the window's columns become channels (FOLD).  Channel c * KW + kx of a place is input
// channel c of the place kx to the right, so one accumulator of 16 to 64 columns serves a whole window row, where each
// column of the window would have had one that is mostly padding (32x32, 3 -> 32 channels, 5x5, 256 samples: 70 us,
// folded 41 us; 11x16, 4 -> 250, 5x5, 74 samples: 55 us, folded 20 us).
struct ConvDwArgs {
  const float *in, *dout;
  float *part, *bpart;     // partial sums [unit][split][nky * NB * nkx * CB][128]; bias partials [block of OB][split][OB]
  int *err;
  int C, OC, IH, IW, OH, OW, KH, KW, SH, SW, pad_t, pad_l;
  int OB, J, CB, NB, ocb, ccb;  // output channels and window rows in the lanes; channels per MMA, MMAs side by side; blocks
  int RS, GC, nseg, nyb;   // rows and pixel groups per row of a stage, segments of a row, row blocks of an image
  int pair_rows;           // a step's two groups lie in two rows (GC odd) instead of side by side
  int fold;                // window columns folded into the channels (C and KW are then C * KW and 1); 0: none
  int ftab[64];            // channel c * KW + kx: c << 16 | kx
  int lo;                  // columns from an accumulator to the one of its small products; 0: they share one
  int nstages, nst;        // stages over the batch, stage buffers
  int teams;               // loader teams, each takes every teams-th stage: the memory latency of a small stage is
                           // longer than its MMAs
  int sub, xpos;           // places per residue and row, places of a stage
  int orow;                // bytes of one output channel in a gradient part
  int ny;                  // gradient items of a stage
  int steps;               // steps of 16 pixels per stage
  int nkg;
  DwKGroup kg[DW_MAX_KGROUPS];
  long long *dbg;          // [blocks][16] cycle counters in a build with -DB200_TC_TIMING, else nullptr
};

// where a stage lies: rows y0 .. of the image with the J - 1 extra rows the shifted lanes need
struct DwStage {
  int b, yb, seg;
  __device__ __forceinline__ void at(const ConvDwArgs &a, int s) {
    const int per = a.nyb * a.nseg;
    b = s / per;
    const int r = s - b * per;
    yb = r / a.nseg;
    seg = r - yb * a.nseg;
  }
  __device__ __forceinline__ void next(const ConvDwArgs &a) {
    if (++seg == a.nseg) {
      seg = 0;
      if (++yb == a.nyb) yb = 0, ++b;
    }
  }
};

// eight values of a gradient row, zero past its end (`left` values from here)
template <bool VEC>
__device__ __forceinline__ void load8(const float *p, int left, uint32_t *v) {
  if constexpr (VEC) {
    ldg4_if(p, left > 0, v);
    ldg4_if(p + 4, left > 4, v + 4);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = ldg_if(p + i, i < left);
  }
}

__device__ __forceinline__ void store8(uint8_t *d, size_t part, const uint32_t *v) {
  uint32_t p1[4], p2[4], p3[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split_bf16x3(v[2 * i], v[2 * i + 1], p1[i], p2[i], p3[i]);
  sts_words<4>(d, p1);
  sts_words<4>(d + part, p2);
  sts_words<4>(d + 2 * part, p3);
}

template <bool VEC, bool FOLD>
__global__ void __launch_bounds__(DW_THREADS, 1) conv_gather_dw_kernel(const __grid_constant__ ConvDwArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t RBY = (uint32_t)a.CB * 2u;                                      // bytes of one place
  const uint32_t XB = ((uint32_t)a.xpos * RBY + 1023u) & ~1023u;                 // one part of CB input channels
  const uint32_t XP = XB * a.NB, XS = 3u * XP;                                   // of all; a stage
  const uint32_t YP = (uint32_t)(a.OB * a.orow), YS = 3u * YP;                   // of the gradient
  uint8_t *xsm = smem, *ysm = xsm + (size_t)a.nst * XS;   // OB * orow is a multiple of 16
  int *gtab = reinterpret_cast<int *>(ysm + (size_t)a.nst * YS);  // [64] byte offset of the pixel groups, in step order
  int *xtab = gtab + 64;                                          // [xpos] row << 16 | column of a place
  int *rtab = xtab + ((a.xpos + 1) & ~1);                         // [steps, even] first place of a step, descriptor units
  int *atab = rtab + ((a.steps + 1) & ~1);                        // [24] first place of an accumulator, descriptor units
  int2 *ytab = reinterpret_cast<int2 *>(atab + 24);  // [ny] source offset; group << 25 | row << 17 | place
  float *bsum = reinterpret_cast<float *>(ytab + a.ny);           // [teams][ny] bias partials of the items
  uint64_t *full = reinterpret_cast<uint64_t *>(bsum + ((a.teams * a.ny + 1) & ~1));
  uint64_t *x_empty = full + DW_MAX_STAGES, *y_empty = x_empty + DW_MAX_STAGES, *a_full = y_empty + DW_MAX_STAGES,
           *a_empty = a_full + 2, *accum = a_empty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum + 1);

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  int ki = 0;
  while (ki + 1 < a.nkg && (int)blockIdx.x >= a.kg[ki + 1].first) ++ki;
  const DwKGroup &kg = a.kg[ki];
  const int nkx = kg.nkx, rel = blockIdx.x - kg.first, unit = rel / kg.splits, split = rel - unit * kg.splits;
  const int ob = unit / a.ccb, cb = unit - ob * a.ccb, o0 = ob * a.OB, c0 = cb * a.NB * a.CB;
  const int nacc = kg.nky * a.NB * nkx;       // accumulators
  const int s_begin = (int)((long long)split * a.nstages / kg.splits), s_end = (int)((long long)(split + 1) * a.nstages / kg.splits);
  const int nunits = (a.steps + 1) / 2;       // 32-pixel units of a stage
  const int each = (nacc + DW_ISSUERS - 1) / DW_ISSUERS, issuers = (nacc + each - 1) / each;  // no fewer, and evenly loaded
  const int yrows = a.RS + a.J - 1;           // gradient rows of a stage

  if (tid == 0) {
    for (int i = 0; i < a.nst; ++i) {
      mbar_init(&full[i], DW_LOAD_WARPS / a.teams);
      mbar_init(&x_empty[i], issuers);
      mbar_init(&y_empty[i], 4);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&a_full[i], 4);
      mbar_init(&a_empty[i], issuers);
    }
    mbar_init(accum, issuers);
    mbar_fence_init();
  }
  for (int i = tid; i < a.xpos; i += DW_THREADS) {
    const int row = i / (a.sub * a.SW), r = i - row * a.sub * a.SW, ph = r / a.sub;
    xtab[i] = row << 16 | ((r - ph * a.sub) * a.SW + ph);
  }
  for (int i = tid; i < a.ny; i += DW_THREADS) {
    const int per = yrows * a.GC, o = i / per, q = i - o * per, ry = q / a.GC, cg = q - ry * a.GC;
    ytab[i] = make_int2(o * a.OH * a.OW + ry * a.OW + cg * 8, cg << 25 | ry << 17 | (o * a.orow + q * 16));
    bsum[i] = 0.f;
    if (a.teams > 1) bsum[a.ny + i] = 0.f;
  }
  for (int t = tid; t < nacc; t += DW_THREADS) {
    const int k = t % nkx, nb = t / nkx % a.NB, i = t / (nkx * a.NB), kx = kg.kx0 + k, q = kx / a.SW;
    atab[t] = (int)((nb * XB + (uint32_t)((i * a.J * a.SW + kx - q * a.SW) * a.sub + q) * RBY) >> 4);
  }
  for (int t = tid; t < 64; t += DW_THREADS) {  // groups past the last repeat it: no MMA reads them
    const int step = min(t >> 1, a.steps - 1), e = t & 1;
    int ry, cg;
    if (a.pair_rows) {
      ry = step / a.GC * 2 + e;
      cg = step % a.GC;
    } else {
      ry = step / (a.GC / 2);
      cg = step % (a.GC / 2) * 2 + e;
    }
    gtab[t] = (ry * a.GC + cg) * 16;
    if (e == 0 && (t >> 1) < ((a.steps + 1) & ~1)) rtab[t >> 1] = ((ry * a.sub * a.SW + cg * 8) * (int)RBY) >> 4;
  }
  wait_for_previous_kernel();
  if (warp == DW_W_MMA) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem_base = 0, tmem_a = DW_D_COLS;  // all 512 columns: see conv_gather_kernel
  bool failed = __any_sync(0xffffffffu, *tmem_slot != tmem_base);

  if (warp < DW_W_GATHER) {
    // ---- loaders ----------------------------------------------------------------------------------------
    const size_t in_plane = (size_t)a.IH * a.IW, out_plane = (size_t)a.OH * a.OW;
    const int plane = a.IH * a.IW;
    const int ychunks = yrows * a.GC;
    const int nshift = a.CB == 64 ? 3 : a.CB == 32 ? 2 : 1, cshift = 3 - nshift, cmask = (1 << nshift) - 1;
    const int xper = ((a.xpos + 31) / 32) << nshift, xitems = xper * a.NB;  // 32 places x 8 channels
    const int twarps = DW_LOAD_WARPS / a.teams, tthreads = twarps * 32, team = warp / twarps, tw = warp - team * twarps,
              tt = tw * 32 + lane;
    const int batches = max((a.ny + DW_YB * tthreads - 1) / (DW_YB * tthreads), (xitems + DW_XB * twarps - 1) / (DW_XB * twarps));
    const bool bias = ki == 0 && cb == 0 && a.bpart != nullptr;
    const int ymax = a.OC - o0;
    uint32_t yv[DW_YB][8], xv[DW_XB][8];
    auto load = [&](const DwStage &sg, int k) {
      const int y0 = sg.yb * a.RS, x0 = sg.seg * a.GC * 8, ytop = y0 - (a.J - 1);
      const float *dyb = a.dout + ((size_t)sg.b * a.OC + o0) * out_plane + (ptrdiff_t)ytop * a.OW + x0;
#pragma unroll
      for (int e = 0; e < DW_YB; ++e) {
        const int it = tt + (k * DW_YB + e) * tthreads;
        const int2 t = ytab[min(it, a.ny - 1)];
        const int y = ytop + ((t.y >> 17) & 255), x = (t.y >> 25) * 8 + x0;
        const bool ok = it < a.ny && y >= 0 && y < a.OH && it < ymax * ychunks;
        load8<VEC>(dyb + t.x, ok ? a.OW - x : 0, yv[e]);
      }
      const int iy0 = y0 * a.SH + kg.ky0 - a.pad_t, ix0 = x0 * a.SW - a.pad_l;
      const float *xb = a.in + (FOLD ? (size_t)sg.b * (a.C / a.fold) : (size_t)sg.b * a.C + c0) * in_plane;
#pragma unroll
      for (int e = 0; e < DW_XB; ++e) {
        const int it = tw + (k * DW_XB + e) * twarps, nb = it >= xper ? 1 : 0, ib = it - nb * xper;
        const int cg = ib & cmask, pos = (ib >> nshift) * 32 + lane;
        const int t = xtab[min(pos, a.xpos - 1)], iy = iy0 + (t >> 16) * a.SH, ix = ix0 + (t & 0xffff);
        const int cl = nb * a.CB + cg * 8;
        if constexpr (FOLD) {
          const int nc = it < xitems && iy >= 0 && iy < a.IH ? a.C - cl : 0;
          const float *q = xb + (ptrdiff_t)iy * a.IW + ix;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int f = a.ftab[cl + c], kx = f & 0xffff;
            xv[e][c] = ldg_if(q + (size_t)(f >> 16) * in_plane + kx, c < nc && (unsigned)(ix + kx) < (unsigned)a.IW);
          }
          continue;
        }
        const bool ok = it < xitems && iy >= 0 && iy < a.IH && ix >= 0 && ix < a.IW;
        const int nc = ok ? a.C - c0 - cl : 0;
        const float *q = xb + (size_t)cl * in_plane + (ptrdiff_t)iy * a.IW + ix;
#pragma unroll
        for (int c = 0; c < 8; ++c) xv[e][c] = ldg_if(q + (size_t)(uint32_t)(c * plane), c < nc);
      }
    };
    auto store = [&](uint32_t st, int k) {
      uint8_t *yd = ysm + st * (size_t)YS, *xd = xsm + st * (size_t)XS;
#pragma unroll
      for (int e = 0; e < DW_YB; ++e) {
        const int it = tt + (k * DW_YB + e) * tthreads;
        if (it < a.ny) {
          store8(yd + (ytab[it].y & 0x1ffff), YP, yv[e]);
          if (bias) {
            float t[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = __uint_as_float(yv[e][q]);
            bsum[team * a.ny + it] += ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
          }
        }
      }
#pragma unroll
      for (int e = 0; e < DW_XB; ++e) {
        const int it = tw + (k * DW_XB + e) * twarps, nb = it >= xper ? 1 : 0, ib = it - nb * xper;
        const int cg = ib & cmask, pos = (ib >> nshift) * 32 + lane;
        if (it < xitems && pos < a.xpos) store8(xd + nb * XB + pos * (int)RBY + ((cg ^ ((pos >> cshift) & cmask)) << 4), XP, xv[e]);
      }
    };
    long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
    DwStage sg;
    sg.at(a, s_begin + team);
    if (s_begin + team < s_end) load(sg, 0);
    uint32_t st = team, par = 1;
    for (int s = s_begin + team; s < s_end && !failed; s += a.teams) {
      tq = tc_clock();
      if (s - s_begin >= a.nst && (!mbar_wait_warp(&x_empty[st], par) || !mbar_wait_warp(&y_empty[st], par))) {
        failed = true;
        break;
      }
      w0 += tc_clock() - tq;
      tq = tc_clock();
      store(st, 0);
      w1 += tc_clock() - tq;
      for (int k = 1; k < batches; ++k) {
        load(sg, k);
        store(st, k);
      }
      // generic-proxy writes of the B operand become visible to the tensor core
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[st]);
      for (int k = 0; k < a.teams; ++k) sg.next(a);
      tq = tc_clock();
      if (s + a.teams < s_end) load(sg, 0);
      w2 += tc_clock() - tq;
      st += a.teams;
      if (st >= (uint32_t)a.nst) st -= a.nst, par ^= 1;
    }
    CV_TIMING(0, warp == 0)
    if (bias) {  // rows above the stage's own are counted by the stage before
      asm volatile("bar.sync 1, %0;\n" ::"n"(DW_LOAD_THREADS) : "memory");
      for (int o = tid; o < a.OB; o += DW_LOAD_THREADS) {
        float t = 0.f;
        for (int q = (a.J - 1) * a.GC; q < ychunks; ++q)
          for (int k = 0; k < a.teams; ++k) t += bsum[k * a.ny + o * ychunks + q];
        a.bpart[((size_t)ob * kg.splits + split) * a.OB + o] = t;
      }
    }
  } else if (warp < DW_W_MMA) {
    // ---- gather: lane (j, o) takes the rows j above -----------------------------------------------------------
    const int quad = warp & 3, l = quad * 32 + lane, j = min(l / a.OB, a.J - 1), o = min(l - j * a.OB, a.OB - 1);
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16, loff = (uint32_t)(o * a.orow + (a.J - 1 - j) * a.GC * 16);
    uint32_t v = 0, st = 0, par = 0;
    long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
    for (int s = s_begin; s < s_end && !failed; ++s) {
      tq = tc_clock();
      if (!mbar_wait_warp(&full[st], par)) {
        failed = true;
        break;
      }
      w0 += tc_clock() - tq;
      const uint32_t y1 = smem_u32(ysm + st * (size_t)YS) + loff, y2 = y1 + YP, y3 = y2 + YP, gt = smem_u32(gtab);
      for (int un = 0; un < nunits; ++un, ++v) {
        const uint32_t ab = v & 1;
        tq = tc_clock();
        if (v >= 2 && !mbar_wait_warp(&a_empty[ab], ((v >> 1) - 1) & 1)) {
          failed = true;
          break;
        }
        w1 += tc_clock() - tq;
        tc_fence_after();
        const uint4 go = lds_u4(gt + un * 16);
        const uint32_t gg[4] = {go.x, go.y, go.z, go.w};
        const uint32_t ta = tmem_a + ab * DW_A_COLS + lane_base;
        uint32_t b1[16], b2[16], b3[16];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          lds_words<4>(y1 + gg[e], b1 + 4 * e);
          lds_words<4>(y2 + gg[e], b2 + 4 * e);
          lds_words<4>(y3 + gg[e], b3 + 4 * e);
        }
        tmem_st16(ta, b1);
        tmem_st16(ta + 16, b2);
        tmem_st16(ta + 32, b3);
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_leader<1>(&a_full[ab]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&y_empty[st]);
      if (++st == (uint32_t)a.nst) st = 0, par ^= 1;
    }
    CV_TIMING(1, warp == DW_W_GATHER)
    // ---- epilogue: partial sums, lanes consecutive --------------------------------------------------------------
    if (s_end > s_begin && !failed) failed = !mbar_wait_warp(accum, 0);
    tc_fence_after();
    if (!failed) {
      float *dst = a.part + kg.part0 + ((size_t)unit * kg.splits + split) * (nacc * a.CB) * 128 + l;
      for (int n = 0; n < nacc * a.CB; n += 16) {
        uint32_t x[16];
        if (s_end > s_begin) {
          tmem_ld16_nowait(tmem_base + lane_base + (uint32_t)n, x);
          tmem_ld_wait();
          if (a.lo) {
            uint32_t y[16];
            tmem_ld16_nowait(tmem_base + lane_base + (uint32_t)(a.lo + n), y);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 16; ++q) x[q] = __float_as_uint(__uint_as_float(x[q]) + __uint_as_float(y[q]));
          }
        } else {
#pragma unroll
          for (int q = 0; q < 16; ++q) x[q] = 0u;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q) dst[(size_t)(n + q) * 128] = __uint_as_float(x[q]);
      }
    }
  } else {
    // ---- MMA issuers: every other window column (the whole warp stays converged: see elect_one) ---
    const int me = warp - DW_W_MMA;
    if (me < issuers) {
      const uint32_t idesc = umma_idesc_bf16(128, a.CB) | (1u << 16);  // B is MN-major
      const uint32_t rows = (uint32_t)(a.sub * a.SW), sbo = a.pair_rows ? rows * RBY : 8u * RBY;
      const uint64_t b0 = umma_desc(smem_u32(xsm), 16, sbo, a.CB == 64 ? 2 : a.CB == 32 ? 4 : 6), b0hi = b0 & 0xffffffff00000000ull;
      const uint32_t P = XP >> 4;
      uint32_t v = 0, st = 0, par = 0;
      long long w0 = 0, w1 = 0, w2 = 0, t0 = tc_clock(), tq;
      for (int s = s_begin; s < s_end; ++s) {
        tq = tc_clock();
        if (!failed) failed = !mbar_wait_warp(&full[st], par);
        w0 += tc_clock() - tq;
        for (int un = 0; un < nunits; ++un, ++v) {
          const uint32_t ab = v & 1;
          tq = tc_clock();
          if (!failed) failed = !mbar_wait_warp(&a_full[ab], (v >> 1) & 1);
          w1 += tc_clock() - tq;
          tc_fence_after();
          const uint32_t a1 = uni(tmem_a + ab * DW_A_COLS), more = v != 0;
          const uint32_t base = (uint32_t)b0 + ((st * XS) >> 4);
          const uint32_t r0 = uni(base + (uint32_t)rtab[un * 2]), r1 = uni(base + (uint32_t)rtab[un * 2 + 1]);
          const bool both = un * 2 + 1 < a.steps;
          for (int k = me; k < nacc; k += issuers) {
            const uint32_t shift = uni((uint32_t)atab[k]), d = uni(tmem_base + (uint32_t)(k * a.CB));
            const uint64_t d0 = b0hi | (r0 + shift), d1 = b0hi | (r1 + shift);
            if (!failed && elect_one()) {
              if (a.lo) {
                umma_6<1>(d, d + a.lo, a1, d0, P, idesc, more);
                if (both) umma_6<1>(d, d + a.lo, a1 + 8, d1, P, idesc, 1);
              } else {
                umma_6one<1>(d, a1, d0, P, idesc, more);
                if (both) umma_6one<1>(d, a1 + 8, d1, P, idesc, 1);
              }
            }
            __syncwarp();
          }
          if (!failed && elect_one()) umma_commit(&a_empty[ab]);
          __syncwarp();
        }
        if (!failed && elect_one()) umma_commit(&x_empty[st]);
        __syncwarp();
        if (++st == (uint32_t)a.nst) st = 0, par ^= 1;
      }
      CV_TIMING(2, me == 0)
      if (!failed && elect_one()) umma_commit(accum);
      __syncwarp();
    }
  }
  if (failed && a.err) atomicExch(a.err, 4);
  tc_fence_before();
  __syncthreads();
  if (warp == DW_W_MMA) tmem_dealloc(tmem_base, 512);
}

// ---- partial sums -> gradient -------------------------------------------------------------------------------
//
// A row is 128 lanes (j, o) of one (group, unit, accumulator, input channel), four to a thread.  Few splits: a block
// takes eight rows, a thread adds the splits in order.  Many: a block takes one row, thread row k adds splits k, k + 8,
// ... and the eight sums are added in order.  The last OC blocks add up the bias gradient.  What bounds it is the loads
// in flight: one lane a thread and a quarter of a row a block took 13.5 us for the 12 MB of 16x16, 32 -> 32, 5x5, 256
// samples and 16 us for 8x8, 32 -> 64; now 6.4 and 7.9.
__global__ void __launch_bounds__(256) conv_gather_dw_finish_kernel(const __grid_constant__ ConvDwArgs a, int rows, int spread,
                                                                    float *__restrict__ dW, float *__restrict__ db,
                                                                    const uint8_t *__restrict__ tbl, int accumulate) {
  after_previous_kernel();
  __shared__ float4 lanes[8][32];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nblk = spread ? rows : (rows + 7) / 8;
  if ((int)blockIdx.x >= nblk) {
    const int o = blockIdx.x - nblk, ob = o / a.OB, nsplit = a.kg[0].splits;
    float s = 0.f;
    for (int k = ty * 32 + tx; k < nsplit; k += 256) s += a.bpart[((size_t)ob * nsplit + k) * a.OB + (o - ob * a.OB)];
    s = warp_sum(s);
    if (tx == 0) lanes[ty][0].x = s;
    __syncthreads();
    if (tx == 0 && ty == 0) {
      for (int k = 1; k < 8; ++k) s += lanes[k][0].x;
      db[o] = accumulate ? db[o] + s : s;
    }
    return;
  }
  int row = spread ? blockIdx.x : blockIdx.x * 8 + ty;
  const bool live = row < rows;
  int ki = 0, mine = 0;
  if (live) {
    for (;; ++ki) {
      mine = a.ocb * a.ccb * a.kg[ki].nky * a.NB * a.kg[ki].nkx * a.CB;
      if (row < mine) break;
      row -= mine;
    }
  }
  const DwKGroup &kg = a.kg[ki];
  const int per = kg.nky * a.NB * kg.nkx * a.CB, unit = row / per, n = row - unit * per;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add = [&](const float4 &v) { s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w; };
  if (live) {
    const float4 *p = reinterpret_cast<const float4 *>(a.part + kg.part0 + ((size_t)unit * kg.splits * per + n) * 128) + tx;
    const size_t step = (size_t)per * 32;
#pragma unroll 8
    for (int k = spread ? ty : 0; k < kg.splits; k += spread ? 8 : 1) add(p[(size_t)k * step]);
  }
  if (spread) {
    lanes[ty][tx] = s;
    __syncthreads();
    if (ty != 0) return;
#pragma unroll
    for (int k = 1; k < 8; ++k) add(lanes[k][tx]);
  }
  if (!live) return;
  const int acc = n / a.CB, k = acc % kg.nkx, nb = acc / kg.nkx % a.NB, i = acc / (kg.nkx * a.NB);
  const int ob = unit / a.ccb;
  int c = ((unit - ob * a.ccb) * a.NB + nb) * a.CB + n - acc * a.CB, kx = kg.kx0 + k, C = a.C, KW = a.KW;
  if (c >= C) return;
  if (a.fold) {
    kx = a.ftab[c] & 0xffff;
    c = a.ftab[c] >> 16;
    KW = a.fold;
    C /= KW;
  }
  const float sums[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int l = tx * 4 + e, j = l / a.OB, o = ob * a.OB + l - j * a.OB, ky = kg.ky0 + a.SH * (i * a.J + j);
    if (j >= a.J || o >= a.OC || ky >= a.KH) continue;
    const float v = tbl && !tbl[c * a.OC + o] ? 0.f : sums[e];
    float *d = dW + (((size_t)o * C + c) * a.KH + ky) * KW + kx;
    *d = accumulate ? *d + v : v;
  }
}

// ---- host side ------------------------------------------------------------------------------------------------

// Cycles of a stage of every group; returns the sum over all units.  The tensor pipe and its issuers, against the loads
// (18 bytes a cycle is what an SM draws from the L2 cache with all others doing the same), the loaders' instructions, and
// one load's latency with the conversion behind it, which do not depend on the group.
double dw_group_costs(const ConvDwArgs &a, double *cost) {
  const double bytes = (a.ny * 8.0 + (double)a.xpos * a.CB * a.NB) * 4 / 18;
  const double instr = a.ny / 32.0 * 36 + (a.xpos + 31) / 32 * a.NB * (a.CB / 8) * 40.0;
  double loads = bytes > instr ? bytes : instr, weight = 0;
  if (loads < 3500.0 / a.teams) loads = 3500.0 / a.teams;
  for (int i = 0; i < a.nkg; ++i) {
    // a unit is two steps: the pipe's cycles, and about 720 of an issuer for each of its accumulators
    const int nacc = a.NB * a.kg[i].nky * a.kg[i].nkx;
    const double pipe = nacc * 12. * (a.CB > 32 ? a.CB / 2 : 18), issue = ceil_div(nacc, DW_ISSUERS) * 720.;
    const double mma = a.steps / 2. * (pipe > issue ? pipe : issue);
    cost[i] = (mma > loads ? mma : loads) + 250;
    weight += cost[i] * a.ocb * a.ccb;
  }
  return weight;
}

// blocks of a unit of one group: the SMs dealt out by what a unit costs.  The tensor core truncates when it adds, so a sum loses
// about 2^-25 of itself with every addition, one a step or, where all products share an accumulator, six: no block takes
// more than 24576 of them (0.07 %; 511 x 511 pixels of 8227 images in 148 slices: 4.5 %).
int dw_group_splits(const b200_ctx *ctx, const ConvDwArgs &a, bool lo, long long nstages, double cost, double weight) {
  int n = (int)(ctx->sm_count * cost / weight);
  if (n > nstages) n = (int)nstages;
  if (n < 1) n = 1;
  const long long adds = nstages * a.steps * (lo ? 1 : 6);
  return (int)max((long long)n, (adds + DW_MAX_ADDS - 1) / DW_MAX_ADDS);
}

// splits and partial sums' places of every group; returns the floats that these take
size_t dw_splits(const b200_ctx *ctx, ConvDwArgs *a, int B) {
  a->nstages = B * a->nyb * a->nseg;
  double cost[DW_MAX_KGROUPS];
  const double weight = dw_group_costs(*a, cost);
  size_t floats = 0;
  int first = 0;
  for (int i = 0; i < a->nkg; ++i) {
    DwKGroup &k = a->kg[i];
    k.splits = dw_group_splits(ctx, *a, a->lo != 0, a->nstages, cost[i], weight);
    k.first = first;
    k.part0 = (long long)floats;
    const int units = a->ocb * a->ccb;
    first += units * k.splits;
    floats += (size_t)units * k.splits * k.nky * a->NB * k.nkx * a->CB * 128;
  }
  return floats;
}

// columns from the large products' accumulators to the small ones', where there is room for both; else 0
int dw_low(const ConvDwArgs &a) {
  int cols = 0;
  for (int i = 0; i < a.nkg; ++i) cols = max(cols, a.kg[i].nky * a.kg[i].nkx * a.NB * a.CB);
  return 2 * cols <= DW_D_COLS ? DW_D_COLS / 2 : 0;
}

// Cycles of a call: the longest block -- its stages and its partial sums to memory -- and the pass that adds the partial
// sums up; an SM writes about 30 and reads about 20 bytes a cycle there.  The number of stages of the longest block is a
// whole one, which decides between tilings of small maps (16x16, 32 -> 32, 5x5, 256 samples: one group of 512 stages on
// 148 blocks, 3.5 each but 4 on some, 40.7 us; two groups of five accumulators 36.4 us, with half the partial sums).
// (`best`: what another tiling costs; 0: none yet)
double dw_call_cost(const b200_ctx *ctx, const ConvDwArgs &a, int B, double best) {
  const long long nstages = (long long)B * a.nyb * a.nseg;
  double cost[DW_MAX_KGROUPS], longest = 0, bytes = 0;
  const double weight = dw_group_costs(a, cost), least = nstages * weight / ctx->sm_count;
  if (best > 0 && least > best) return least;  // however it is dealt out
  const bool lo = dw_low(a) != 0;
  int blocks = 0;
  for (int i = 0; i < a.nkg; ++i) {
    const DwKGroup &k = a.kg[i];
    const int splits = dw_group_splits(ctx, a, lo, nstages, cost[i], weight);
    const double part = k.nky * a.NB * k.nkx * a.CB * 512., block = (double)((nstages + splits - 1) / splits) * cost[i] + part / 30.;
    if (block > longest) longest = block;
    blocks += a.ocb * a.ccb * splits;
    bytes += a.ocb * a.ccb * splits * part;
  }
  return longest * ceil_div(blocks, ctx->sm_count) + bytes / (ctx->sm_count * 20.);
}

// tiling of one layer's dW for a batch (returns the cost of the best one, below 0 if there is none)
double search_dw_plan(const b200_ctx *ctx, ConvGeom g, int B, bool fold, ConvDwArgs *out, size_t *smem_out) {
  if (g.pad_t < 0 || g.pad_l < 0 || (long long)g.OH * g.OW > 1 << 23 || (long long)g.HI * g.WI > 1 << 27) return -1;
  ConvDwArgs a = {};
  if (fold) {
    if (g.SW != 1 || g.KW == 1 || g.C * g.KW > 64) return -1;
    a.fold = g.KW;
    for (int c = 0; c < g.C * g.KW; ++c) a.ftab[c] = (c / g.KW) << 16 | (c % g.KW);
    g.C *= g.KW;
    g.KW = 1;
  }
  a.C = g.C;
  a.OC = g.OC;
  a.IH = g.HI;
  a.IW = g.WI;
  a.OH = g.OH;
  a.OW = g.OW;
  a.KH = g.KH;
  a.KW = g.KW;
  a.SH = g.SH;
  a.SW = g.SW;
  a.pad_t = g.pad_t;
  a.pad_l = g.pad_l;
  a.ocb = (g.OC + 127) / 128;
  a.OB = (g.OC + a.ocb - 1) / a.ocb;
  const int gpr = (g.OW + 7) / 8;
  double best = -1;
  for (int CB = 64; CB >= 16; CB /= 2) {
    if (CB > 16 && CB / 2 >= g.C) continue;
    const int accs = DW_D_COLS / CB, jmax = 128 / a.OB, rows1 = (g.KH + g.SH - 1) / g.SH;  // window rows of residue 0
    a.CB = CB;
    for (int NB = 1; NB <= 2; ++NB)
    for (int J = 1; J <= jmax && J <= rows1; ++J)
    for (int nky = 1; nky <= (rows1 + J - 1) / J; ++nky) {
      const int kmax = accs / (NB * nky);
      if (kmax < 1 || (NB == 2 && g.C <= CB) || (fold && NB * CB < g.C)) continue;
      const int kxg = (g.KW + kmax - 1) / kmax, nkx = (g.KW + kxg - 1) / kxg;
      a.NB = NB;
      a.ccb = (g.C + NB * CB - 1) / (NB * CB);
      a.J = J;
      a.nkg = 0;
      bool fits = true;
      for (int res = 0; res < g.SH && res < g.KH; ++res) {
        const int taps = (g.KH - res + g.SH - 1) / g.SH, n = (taps + J - 1) / J;
        for (int i = 0; i < n; i += nky)
          for (int kx = 0; kx < g.KW; kx += nkx) {
            if (a.nkg == DW_MAX_KGROUPS) {
              fits = false;
              break;
            }
            const DwKGroup k = {res + g.SH * J * i, n - i < nky ? n - i : nky, kx, g.KW - kx < nkx ? g.KW - kx : nkx, 0, 0, 0};
            a.kg[a.nkg++] = k;
          }
      }
      if (!fits) continue;
      for (int nseg = 1; nseg <= gpr; ++nseg) {
        a.nseg = nseg;
        for (int up = 0; up < 2; ++up) {
          a.GC = (gpr + nseg - 1) / nseg;
          if (up) {
            if (a.GC % 2 == 0) break;
            ++a.GC;  // an empty group makes the row even
          }
          if ((nseg - 1) * a.GC >= gpr) continue;
          a.pair_rows = a.GC & 1;
          for (int RS = 1 + a.pair_rows; RS * a.GC <= 64; RS += 1 + a.pair_rows) {
            if (RS > g.OH + J - 1 + a.pair_rows) break;
            a.RS = RS;
            a.nyb = (g.OH + J - 1 + RS - 1) / RS;
            a.steps = RS * a.GC / 2;
            a.sub = a.GC * 8 + (g.KW - 1) / g.SW;
            a.xpos = (RS + (nky - 1) * J) * a.sub * g.SW;
            const int yr = RS + J - 1;
            a.orow = yr * a.GC * 16;
            if (a.orow / 16 % 2 == 0) a.orow += 16;  // neighbouring channels in different banks
            a.ny = a.OB * yr * a.GC;
            if (a.ny > DW_MAX_YITEMS || yr > 255 || a.GC > 63 || a.OB * a.orow > 0x1ffff || a.xpos > 16383) break;
            const size_t stage = 3 * NB * align_up((size_t)a.xpos * CB * 2, 1024) + 3 * align_up((size_t)a.OB * a.orow, 16);
            const size_t fixed = 1024 + (64 + 24 + a.xpos + a.steps + 4) * 4 + (size_t)a.ny * 16 + 8 + (3 * DW_MAX_STAGES + 5) * 8 + 16;
            if (fixed + 2 * stage > ctx->smem_optin) break;
            a.nst = (int)((ctx->smem_optin - fixed) / stage);
            if (a.nst > DW_MAX_STAGES) a.nst = DW_MAX_STAGES;
            // two teams of loaders where half of them hold a stage's next loads in registers
            a.teams = a.ny <= DW_YB * DW_LOAD_THREADS / 2 &&
                              (a.xpos + 31) / 32 * NB * (CB / 8) <= DW_XB * DW_LOAD_WARPS / 2 && a.nst > 2
                          ? 2
                          : 1;
            const double cost = dw_call_cost(ctx, a, B, best);
            if (best < 0 || cost < best) {
              best = cost;
              *out = a;
              *smem_out = fixed + a.nst * stage;
            }
          }
        }
      }
    }
  }
  return best;
}

// The search takes 7 to 46 us of host time, and one backward call asks three times: each thread keeps its last plans.
bool dw_plan(const b200_ctx *ctx, const ConvGeom &g, int B, ConvDwArgs *out, size_t *smem_out) {
  struct Entry {
    int key[16] = {0};
    bool ok = false;
    size_t smem = 0;
    ConvDwArgs a;
  };
  constexpr int KEPT = 16;
  static thread_local std::vector<Entry> kept;
  static thread_local int next = 0;
  const int key[16] = {g.C,     g.OC,    g.HI,    g.WI,    g.OH, g.OW, g.KH, g.KW, g.SH, g.SW,
                       g.pad_t, g.pad_l, ctx->sm_count, (int)ctx->smem_optin, 1, B};
  for (Entry &e : kept)
    if (memcmp(e.key, key, sizeof key) == 0) {
      *out = e.a;
      *smem_out = e.smem;
      return e.ok;
    }
  Entry e;
  memcpy(e.key, key, sizeof key);
  e.a = {};
  ConvDwArgs folded = {};
  size_t folded_smem = 0;
  const double cost = search_dw_plan(ctx, g, B, false, &e.a, &e.smem),
               fcost = search_dw_plan(ctx, g, B, true, &folded, &folded_smem);
  if (fcost >= 0 && (cost < 0 || fcost < cost)) {
    e.a = folded;
    e.smem = folded_smem;
  }
  e.ok = cost >= 0 || fcost >= 0;
  e.a.lo = dw_low(e.a);
  *out = e.a;
  *smem_out = e.smem;
  if ((int)kept.size() < KEPT)
    kept.push_back(e);
  else
    kept[next] = e, next = (next + 1) % KEPT;
  return e.ok;
}

}  // namespace

bool conv_gather_dw_ok(const b200_ctx *ctx, const ConvGeom &g) {
  ConvDwArgs a;
  size_t smem;
  return dw_plan(ctx, g, 1, &a, &smem);
}

size_t conv_gather_dw_floats(const b200_ctx *ctx, const ConvGeom &g, int B) {
  ConvDwArgs a;
  size_t smem;
  if (!dw_plan(ctx, g, B, &a, &smem)) return 0;
  const size_t n = dw_splits(ctx, &a, B);
  return n + (size_t)a.kg[0].splits * a.ocb * a.OB + 64;
}

static int dw_blocks(const ConvDwArgs &a) { return a.kg[a.nkg - 1].first + a.ocb * a.ccb * a.kg[a.nkg - 1].splits; }

int conv_gather_dw_blocks(const b200_ctx *ctx, const ConvGeom &g, int B, int plan_batch) {
  ConvDwArgs a;
  size_t smem;
  if (!dw_plan(ctx, g, plan_batch, &a, &smem)) return 0;
  dw_splits(ctx, &a, B);
  return dw_blocks(a);
}

int conv_gather_dw(b200_ctx *ctx, const ConvGeom &g, const float *in, const float *dout, int B, float *part, float *dW,
                   float *db, int accumulate, int plan_batch, bool finish) {
  ConvDwArgs a;
  size_t smem;
  B200_REQUIRE(dw_plan(ctx, g, plan_batch, &a, &smem), "tensor-core dW: the tiles do not fit");
  const size_t n = dw_splits(ctx, &a, B);
  a.in = in;
  a.dout = dout;
  a.part = part;
  a.bpart = db != nullptr && g.has_bias ? part + n : nullptr;
  a.err = ctx->dev_err;
  // gradient rows can be read 16 bytes at a time
  const bool vec = g.OW % 4 == 0 && ((uintptr_t)dout & 15) == 0;
  auto kernel = a.fold ? (vec ? conv_gather_dw_kernel<true, true> : conv_gather_dw_kernel<false, true>)
                       : (vec ? conv_gather_dw_kernel<true, false> : conv_gather_dw_kernel<false, false>);
  const int grid = dw_blocks(a);
  B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
#ifdef B200_TC_TIMING
  static const bool timing = getenv("B200_TC_TIMING") != nullptr;
  if (timing) B200_CUDA(cudaMalloc(&a.dbg, (size_t)grid * 16 * sizeof(long long)));
  if (timing) B200_CUDA(cudaMemset(a.dbg, 0, (size_t)grid * 16 * sizeof(long long)));
#endif
  B200_TRY(launch_kernel(ctx, kernel, dim3(grid), DW_THREADS, smem, 1, a));
#ifdef B200_TC_TIMING
  if (timing) {  // diagnostic: cycles of the roles and of their waits, averaged over blocks
    std::vector<long long> h((size_t)grid * 16);
    B200_CUDA(cudaStreamSynchronize(ctx->stream));
    B200_CUDA(cudaMemcpy(h.data(), a.dbg, h.size() * sizeof(long long), cudaMemcpyDeviceToHost));
    B200_CUDA(cudaFree(a.dbg));
    double s[16] = {0};
    for (int i = 0; i < grid; ++i)
      for (int k = 0; k < 16; ++k) s[k] += (double)h[(size_t)i * 16 + k] / grid;
    fprintf(stderr,
            "[tc-timing] gather dw OB %d J %d CB %d x %d groups %d nky %d nkx %d RS %d GC %d nseg %d teams %d steps %d places %d y items %d stages %d of %d "
            "smem %zu grid %d | loader %.0f (wait %.0f store %.0f load %.0f) | gather %.0f (stage %.0f A %.0f) | mma %.0f (stage %.0f A %.0f)\n",
            a.OB, a.J, a.CB, a.NB, a.nkg, a.kg[0].nky, a.kg[0].nkx, a.RS, a.GC, a.nseg, a.teams, a.steps, a.xpos, a.ny, a.nst, a.nstages, smem, grid, s[0],
            s[1], s[2], s[3], s[4], s[5], s[6], s[8], s[9], s[10]);
  }
#endif
  return finish ? conv_gather_dw_finish(ctx, g, B, part, dW, db, accumulate, plan_batch) : 0;
}

int conv_gather_dw_finish(b200_ctx *ctx, const ConvGeom &g, int B, const float *part, float *dW, float *db, int accumulate,
                          int plan_batch) {
  ConvDwArgs a;
  size_t smem;
  B200_REQUIRE(dw_plan(ctx, g, plan_batch, &a, &smem), "tensor-core dW: the tiles do not fit");
  const size_t n = dw_splits(ctx, &a, B);
  a.part = const_cast<float *>(part);
  a.bpart = db != nullptr && g.has_bias ? a.part + n : nullptr;
  int rows = 0, most = 0;
  for (int i = 0; i < a.nkg; ++i) {
    rows += a.ocb * a.ccb * a.kg[i].nky * a.NB * a.kg[i].nkx * a.CB;
    if (a.kg[i].splits > most) most = a.kg[i].splits;
  }
  const int spread = most > 12;
  const int blocks = (spread ? rows : (rows + 7) / 8) + (a.bpart ? g.OC : 0);
  B200_TRY(launch_kernel(ctx, conv_gather_dw_finish_kernel, dim3(blocks), dim3(32, 8), 0, 1, a, rows, spread, dW, db, g.tbl,
                         accumulate));
  return 0;
}

}  // namespace b200
