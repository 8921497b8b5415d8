// Whole-network kernels for networks that fit one SM: a forward pass, or a forward and a backward pass, of every
// sample in one launch, and the sums over the samples that give the weight gradients in a second one.
//
// What bounds such a network layer by layer is not a kernel's work but the launches: LeNet-5 is 0.4 million
// products a sample, and a training step was 41 kernels of 1 to 15 us with a gap behind each (16 samples: 178 us,
// now 53 us; a prediction of one sample: 67 us, now 19 us).  Here a cluster of up to eight CTAs takes
// one sample: every CTA keeps all activations and gradients of the sample in shared memory, computes a share of each
// layer's values and copies them into the shared memory of the others (DSMEM).  The phases of a step are bound by
// the latency of a few hundred dependent instructions: divisions are multiplications by constants from the host, the
// parameters arrive by bulk copies that are all asked for at the start.
// The values also go to the layers' buffers in global memory, which the rest of the library reads.
// Weight gradients of convolutions and average pooling are left as one row per sample (and slice of the output
// plane); those of fully-connected layers need only the activations and gradients.  small_reduce_kernel adds the rows.
//
// The arithmetic is that of the layer kernels (products added in fp32); only the order of the sums differs.
#include <float.h>

#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "device_utils.cuh"

namespace b200 {

namespace {

constexpr int SN_THREADS = 512, SN_WARPS = SN_THREADS / 32;
constexpr int SN_WHOLE = 8192;  // weights of a fully-connected layer up to which every CTA has all of them

// Exchange between the CTAs of a sample.  A CTA writes its share of a layer, consecutive values, to its own shared
// memory and then copies it to the others in one bulk copy each (up to three values at either end, off the 16-byte
// grid, go by st.async); the copies count their bytes on the receiver's barrier, and a step ends when the barrier has
// seen the rest of the layer.  No fence waits for the stores to global memory on the way, as a cluster barrier per
// step would (LeNet-5 step of 16 samples: 79 us), and a barrier is not updated for every value (91 us).  Every exchange
// has a barrier of its own: a CTA whose share of a layer is empty (10 outputs, 8 CTAs) holds nobody up, so the others may
// be any number of steps ahead of it, and a barrier used again could take their bytes for those of the earlier step.
constexpr int SN_EXCHANGES = 2 * SN_MAX_STEPS;  // at most one a step each way
struct Cluster {
  int n, rank, shift;   // n <= 1 << shift
  SmallDiv by_n;
  uint64_t *bar;   // [SN_EXCHANGES]
  uint32_t step;   // exchanges so far
  bool failed;

  // p[first, first + count) is this CTA's share of a layer of `total` values, written by any of its threads;
  // optionally q[first, first + count) too.  On return all of the layer is there.
  __device__ __forceinline__ void exchange(float *p, int first, int count, int total, float *q = nullptr) {
    if (n == 1) {
      __syncthreads();
      return;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    uint64_t *b = &bar[step];
    if (step == 0) asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");  // every CTA's barriers are there
    if (threadIdx.x < 32) {
      if (threadIdx.x == 0) mbar_expect_tx(b, (uint32_t)(total - count) * (q ? 8u : 4u));
      send(p, first, count, b);
      if (q) send(q, first, count, b);
    }
    if (!failed && !mbar_wait_bounded(b, 0)) failed = true;
    ++step;
  }

  // one warp: a lane for each receiver and piece
  __device__ __forceinline__ void send(float *p, int first, int count, uint64_t *b) const {
    const uint32_t end = smem_u32(p + first + count);
    uint32_t at = smem_u32(p + first), head = min((16u - (at & 15u)) & 15u, end - at);
    const uint32_t bulk = (end - at - head) & ~15u;
    const int to = threadIdx.x & ((1 << shift) - 1);
    for (int piece = threadIdx.x >> shift; piece < 7; piece += 32 >> shift) {
      // piece 0: the bulk, 1 to 3: values before it, 4 to 6 after
      if (to == rank || to >= n) continue;
      uint32_t rb;
      asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(rb) : "r"(smem_u32(b)), "r"(to));
      const uint32_t src = piece == 0 ? at + head : piece < 4 ? at + (piece - 1) * 4 : at + head + bulk + (piece - 4) * 4;
      uint32_t dst;
      asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(dst) : "r"(src), "r"(to));
      if (piece == 0) {
        if (bulk)
          asm volatile(
            "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "r"(src),
            "r"(bulk), "r"(rb)
            : "memory");
      } else if (piece < 4 ? (piece - 1) * 4 < (int)head : src < end) {
        float v;
        asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(src));
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];\n" ::"r"(dst), "f"(v),
                     "r"(rb)
                     : "memory");
      }
    }
  }
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}

// this CTA's share of n values
__device__ __forceinline__ void share(const Cluster &cl, int n, int *first, int *count) {
  const int per = cl.by_n.of(n + cl.n - 1);
  *first = min(n, cl.rank * per);
  *count = min(n, *first + per) - *first;
}

// lanes that share one value's sum, as a power of two: at most `most`
__device__ __forceinline__ int lanes_for(int items, int most) {
  int k = 0;
  while (k < most && items << (k + 1) <= SN_THREADS) ++k;
  return k;
}

__device__ __forceinline__ float lane_sum(float v, int ks) {
  for (int o = ks >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Convolution by tiles of four neighbouring outputs of a row (stride 1): a filter row and KW + 3 inputs in registers
// make 4 KW products, against two loads a product.  The (channel, filter row) pairs are dealt to ks lanes.
constexpr int SN_XT = 4;

template <int KW, bool EDGES>
__device__ __forceinline__ void row_products(const float *row, int x0, int width, const float *w, float *acc) {
  float v[KW + SN_XT - 1];
#pragma unroll
  for (int j = 0; j < KW + SN_XT - 1; ++j) {  // no branch around a load: it would be waited for at the join
    const bool inside = !EDGES || (unsigned)(x0 + j) < (unsigned)width;
    const float t = row[inside ? x0 + j : 0];
    v[j] = inside ? t : 0.f;
  }
#pragma unroll
  for (int kx = 0; kx < KW; ++kx)
#pragma unroll
    for (int t = 0; t < SN_XT; ++t) acc[t] = fmaf(v[t + kx], w[kx], acc[t]);
}

// Without padding a tile reads past its row only for outputs that do not exist.
template <int KW, bool EDGES>
__device__ __forceinline__ void conv_out_tile(const SmallStep &L, const float *in, const float *W, int o, int y, int x, int part,
                                              int ks, float *acc) {
  int c = 0, ky = part;
  for (; ky >= L.KH; ky -= L.KH) ++c;
  while (c < L.C) {
    const int iy = y + ky - L.pad_t;
    if (iy >= 0 && iy < L.HI)
      row_products<KW, EDGES>(in + (c * L.HI + iy) * L.WI, x - L.pad_l, L.WI, W + ((o * L.C + c) * L.KH + ky) * KW, acc);
    for (ky += ks; ky >= L.KH; ky -= L.KH) ++c;
  }
}

// dE/d input: the same with the filter rows read backwards
template <int KW>
__device__ __forceinline__ void conv_din_tile(const SmallStep &L, const float *d, const float *W, int c, int iy, int x, int part,
                                              int ks, float *acc) {
  int o = 0, ky = part;
  for (; ky >= L.KH; ky -= L.KH) ++o;
  while (o < L.OC) {
    const int oy = iy + L.pad_t - ky;
    if (oy >= 0 && oy < L.OH) {
      const float *w = W + ((o * L.C + c) * L.KH + ky) * KW;
      float r[KW];
#pragma unroll
      for (int k = 0; k < KW; ++k) r[k] = w[KW - 1 - k];
      row_products<KW, true>(d + (o * L.OH + oy) * L.OW, x + L.pad_l - (KW - 1), L.OW, r, acc);
    }
    for (ky += ks; ky >= L.KH; ky -= L.KH) ++o;
  }
}

// any window, stride and dilation: one output
__device__ __forceinline__ float conv_out(const SmallStep &L, const float *in, const float *W, int i, int part, int ks) {
  const int plane = L.OH * L.OW, o = i / plane, r = i - o * plane, y = r / L.OW;
  const int x0 = (r - y * L.OW) * L.SW - L.pad_l, y0 = y * L.SH - L.pad_t;
  float acc = 0.f;
  int c = 0, ky = part;
  for (; ky >= L.KH; ky -= L.KH) ++c;
  while (c < L.C) {
    const int iy = y0 + ky * L.DH;
    if (iy >= 0 && iy < L.HI) {
      const float *row = in + (c * L.HI + iy) * L.WI, *w = W + ((o * L.C + c) * L.KH + ky) * L.KW;
      for (int kx = 0; kx < L.KW; ++kx) {
        const int ix = x0 + kx * L.DW;
        if (ix >= 0 && ix < L.WI) acc = fmaf(row[ix], w[kx], acc);
      }
    }
    for (ky += ks; ky >= L.KH; ky -= L.KH) ++c;
  }
  return acc;
}

__device__ __forceinline__ float conv_din(const SmallStep &L, const float *d, const float *W, int i, int part, int ks) {
  const int plane = L.HI * L.WI, c = i / plane, r = i - c * plane, iy = r / L.WI, yp = iy + L.pad_t,
            xp = r - iy * L.WI + L.pad_l;
  float acc = 0.f;
  for (int o = part; o < L.OC; o += ks) {
    const float *w = W + (o * L.C + c) * L.KH * L.KW, *dp = d + o * L.OH * L.OW;
    for (int ky = 0; ky < L.KH; ++ky) {
      const int ty = yp - ky, oy = ty / L.SH;
      if (ty < 0 || oy * L.SH != ty || oy >= L.OH) continue;
      for (int kx = 0; kx < L.KW; ++kx) {
        const int tx = xp - kx, ox = tx / L.SW;
        if (tx < 0 || ox * L.SW != tx || ox >= L.OW) continue;
        acc = fmaf(w[ky * L.KW + kx], dp[oy * L.OW + ox], acc);
      }
    }
  }
  return acc;
}

__device__ __forceinline__ bool tiled_rows(const SmallStep &L) {
  return (L.KW == 5 || L.KW == 3) && L.SH == 1 && L.SW == 1 && L.DH == 1 && L.DW == 1;
}

// value(i, v) for every output (W planes of H x Wd, this CTA's share) of a stride-1 convolution pass
// and [*out_first, + *out_count) the values that the share covers
template <int KW, bool DIN, typename F>
__device__ __forceinline__ void conv_tiles(const SmallStep &L, const float *src, const float *W, const Cluster &cl, F value,
                                           int *out_first, int *out_count) {
  const int H = DIN ? L.HI : L.OH, Wd = DIN ? L.WI : L.OW, P = DIN ? L.C : L.OC, nx = (Wd + SN_XT - 1) / SN_XT;
  int first, count;
  share(cl, P * H * nx, &first, &count);
  const SmallDiv dx = DIN ? L.d_inx : L.d_onx, dh = DIN ? L.d_ih : L.d_oh;
  auto start = [&](int item) {  // first value of a tile
    const int row = dx.of(item);
    return row * Wd + (item - row * nx) * SN_XT;
  };
  *out_first = start(first);
  *out_count = start(first + count) - *out_first;
  const int kl = lanes_for(count, 4), ks = 1 << kl, total = count << kl;
  for (int base = 0; base < total; base += SN_THREADS) {
    const int idx = base + (int)threadIdx.x, item = first + (idx >> kl), part = idx & (ks - 1);
    const int row = dx.of(item), x = (item - row * nx) * SN_XT, p = dh.of(row), y = row - p * H;
    float acc[SN_XT] = {0.f, 0.f, 0.f, 0.f};
    if (idx < total) {
      if (DIN)
        conv_din_tile<KW>(L, src, W, p, y, x, part, ks, acc);
      else if (L.pad_l == 0)
        conv_out_tile<KW, false>(L, src, W, p, y, x, part, ks, acc);
      else
        conv_out_tile<KW, true>(L, src, W, p, y, x, part, ks, acc);
    }
#pragma unroll
    for (int t = 0; t < SN_XT; ++t) acc[t] = lane_sum(acc[t], ks);
    // with four lanes or more each of the first four finishes one value
    for (int t = part; t < SN_XT; t += ks) {
      const float v = t == 0 ? acc[0] : t == 1 ? acc[1] : t == 2 ? acc[2] : acc[3];
      if (idx < total && x + t < Wd) value(row * Wd + x + t, v);
    }
  }
}

__device__ __forceinline__ float avg_window(const SmallStep &L, const float *in, int c, int oy, int ox) {
  float v = 0.f;
  if (oy * L.SH + L.KH <= L.HI && ox * L.SW + L.KW <= L.WI) {
    const float *p = in + (c * L.HI + oy * L.SH) * L.WI + ox * L.SW;
    for (int dy = 0; dy < L.KH; ++dy)
      for (int dx = 0; dx < L.KW; ++dx) v += p[dy * L.WI + dx];
  }
  return v;
}

// Weight gradients of one sample and slice of the output plane for windows of K x K: a warp takes a pair of channels,
// a lane every 32nd pixel and all taps of it; the lanes' sums are added in halves, which leaves tap j in lane j.
template <int K>
__device__ __forceinline__ void conv_dw_pairs(const SmallStep &L, const float *in, const float *d, float *part, const Cluster &cl) {
  constexpr int KK = K * K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, plane = L.OH * L.OW, pairs = L.OC * L.C;
  const int units = pairs * L.slices, span = L.span;
  for (int u = cl.rank * SN_WARPS + warp; u < units; u += cl.n * SN_WARPS) {
    const int sl = L.d_pairs.of(u), oc = u - sl * pairs, o = L.d_c.of(oc), c = oc - o * L.C;
    const bool connected = !L.tbl || L.tbl[c * L.OC + o];
    float *dst = part + (size_t)sl * L.part_len;
    float acc[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = 0.f;
    auto pixels = [&](auto edges) {
      constexpr bool EDGES = decltype(edges)::value;
      for (int p = sl * span + lane; p < min(plane, sl * span + span); p += 32) {
        const int y = L.d_ow.of(p), iy0 = y * L.SH - L.pad_t, ix0 = (p - y * L.OW) * L.SW - L.pad_l;
        const float g = d[o * plane + p], *q = in + c * L.HI * L.WI;
        acc[KK] += g;
#pragma unroll
        for (int ky = 0; ky < K; ++ky)
#pragma unroll
          for (int kx = 0; kx < K; ++kx) {
            const bool inside =
              !EDGES || ((unsigned)(iy0 + ky) < (unsigned)L.HI && (unsigned)(ix0 + kx) < (unsigned)L.WI);
            const float t = q[inside ? (iy0 + ky) * L.WI + ix0 + kx : 0];
            acc[ky * K + kx] = fmaf(g, inside ? t : 0.f, acc[ky * K + kx]);  // padding is 0 whatever was read
          }
      }
    };
    if (connected || c == 0) {
      if (L.pad_t == 0 && L.pad_l == 0 && (L.OH - 1) * L.SH + K <= L.HI && (L.OW - 1) * L.SW + K <= L.WI)
        pixels(std::false_type());
      else
        pixels(std::true_type());
    }
#pragma unroll
    for (int h = 16; h > 0; h >>= 1)
#pragma unroll
      for (int j = 0; j < h; ++j) {
        const bool up = lane & h;
        const float keep = up ? acc[j + h] : acc[j], give = up ? acc[j] : acc[j + h];
        acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, h);
      }
    if (lane < KK)
      dst[oc * KK + lane] = connected ? acc[0] : 0.f;
    else if (lane == KK && c == 0 && L.has_bias)
      dst[L.w_len + o] = acc[0];
  }
}

// any other window: a warp takes a filter row (o, c, ky), five taps at a time
__device__ __forceinline__ void conv_dw(const SmallStep &L, const float *in, const float *d, float *part, const Cluster &cl) {
  constexpr int N = 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, plane = L.OH * L.OW;
  const int rows = L.OC * L.C * L.KH, units = rows * L.slices, span = (plane + L.slices - 1) / L.slices;
  for (int u = cl.rank * SN_WARPS + warp; u < units; u += cl.n * SN_WARPS) {
    const int sl = u / rows, row = u - sl * rows, oc = row / L.KH, ky = row - oc * L.KH, o = oc / L.C, c = oc - o * L.C;
    const bool connected = !L.tbl || L.tbl[c * L.OC + o], bias = L.has_bias && c == 0 && ky == 0;
    float *dst = part + (size_t)sl * L.part_len + row * L.KW;
    float db = 0.f;
    for (int kx0 = 0; kx0 < L.KW; kx0 += N) {
      float acc[N] = {0.f, 0.f, 0.f, 0.f, 0.f};
      if (connected || bias)
        for (int p = sl * span + lane; p < min(plane, sl * span + span); p += 32) {
          const int y = p / L.OW, x = p - y * L.OW, iy = y * L.SH + ky - L.pad_t, x0 = x * L.SW - L.pad_l + kx0;
          const float g = d[o * plane + p];
          if (kx0 == 0) db += g;
          if (iy < 0 || iy >= L.HI) continue;
          const float *q = in + (c * L.HI + iy) * L.WI + x0;
#pragma unroll
          for (int j = 0; j < N; ++j)
            if (kx0 + j < L.KW && x0 + j >= 0 && x0 + j < L.WI) acc[j] = fmaf(g, q[j], acc[j]);
        }
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float s = warp_sum(acc[j]);
        if (lane == 0 && kx0 + j < L.KW) dst[kx0 + j] = connected ? s : 0.f;
      }
    }
    if (bias) {
      db = warp_sum(db);
      if (lane == 0) part[(size_t)sl * L.part_len + L.w_len + o] = db;
    }
  }
}

// n floats to shared memory with one bulk copy: from the 16-byte boundary at or before src to the one behind the last
// value, so that they end up (src mod 4) floats behind dst.  Only for the parameters, whose block has room either side.
__device__ __forceinline__ void copy_in(float *dst, const float *src, int n, uint64_t *bar, bool arrive) {
  const uint32_t off = (uint32_t)(((uintptr_t)src >> 2) & 3), bytes = (off + n + 3) / 4 * 16;
  if (arrive)
    mbar_expect_tx(bar, bytes);
  else
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  bulk_copy_g2s(dst, src - off, bytes, bar);
}

// where such a copy leaves the first value
__device__ __forceinline__ int misplaced(const float *src) { return (int)(((uintptr_t)src >> 2) & 3); }

// floats between the rows of a share of a matrix with `cols` columns
__host__ __device__ __forceinline__ int share_pitch(int cols, int nc) { return ((cols + nc - 1) / nc + 3 + 3) / 4 * 4; }

// unconnected pairs of channels: weights of 0
__device__ __forceinline__ void mask_unconnected(const SmallStep &L, float *wts) {
  if (L.kind != SN_CONV || !L.tbl) return;
  for (int i = threadIdx.x; i < L.OC * L.C; i += SN_THREADS) {
    if (L.tbl[(i % L.C) * L.OC + i / L.C]) continue;
    for (int k = 0; k < L.KH * L.KW; ++k) wts[L.w_off + i * L.KH * L.KW + k] = 0.f;
  }
  __syncthreads();
}

// MODE: 0 forward, 1 forward and backward, 2 backward from the values that an earlier forward pass left in the layers'
// buffers.  A kernel each, because the instructions are fetched once a launch and their number counts (LeNet-5 step of 16
// samples with the third mode in the kernel of the second: 61.6 -> 63.5 us).
template <int MODE>
__global__ void __launch_bounds__(SN_THREADS, 1) small_net_kernel(const __grid_constant__ SmallNet net, const float *__restrict__ x,
                                                                  const float *__restrict__ t, float *in_grad, int loss) {
  constexpr bool backward = MODE != 0;
  extern __shared__ __align__(16) float sm[];
  __shared__ uint64_t bars[SN_EXCHANGES], here, rest;  // exchanges; the first step's parameters, the others'
  // the warps touch the plan's lines in the constant cache side by side, so that the misses overlap
  for (int i = threadIdx.x >> 5; i < (int)(sizeof(SmallNet) / 64); i += SN_WARPS) {
    const int w = reinterpret_cast<const int *>(&net)[i * 16];
    asm volatile("" ::"r"(w));
  }
  Cluster cl;
  cl.bar = bars;
  cl.step = 0;
  cl.failed = false;
  asm("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(cl.n));
  asm("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(cl.rank));
  cl.shift = cl.n > 1 ? 32 - __clz(cl.n - 1) : 0;
  cl.by_n = net.by_ctas;
  const int sample = blockIdx.x / cl.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_act = (net.n_act + 3) & ~3;
  float *act = sm, *grd = sm + n_act, *wts = grd + (backward ? n_act : 0), *scratch = wts + net.n_wts;
  if (tid < SN_EXCHANGES) mbar_init(&bars[tid], 1);
  if (tid == 0) {
    mbar_init(&here, 1);
    mbar_init(&rest, SN_THREADS);
  }
  if (tid < SN_EXCHANGES) mbar_fence_init();
  __syncthreads();
  if (cl.n > 1) asm volatile("barrier.cluster.arrive.aligned;\n" ::: "memory");  // waited for before the first exchange
  if (MODE == 0) after_previous_kernel();  // the others are launched behind the end of the kernel before them
  // Everything that the sample needs from global memory is asked for at once, weights by bulk copies; the first step's
  // share is waited for here, the rest behind the first step.
  if (tid < net.n) {
    const SmallStep &L = net.step[tid];
    if (L.copy_n) copy_in(wts + L.copy_off, L.copy, L.copy_n, tid == 0 ? &here : &rest, tid == 0);
  }
  if (tid == 0 && !net.step[0].copy_n) mbar_arrive(&here);
  for (int i = tid; i < net.in_dim; i += SN_THREADS) act[i] = x[(size_t)sample * net.in_dim + i];
  for (int s = 0; s < net.n; ++s) {
    const SmallStep &L = net.step[s];
    if (L.wf_off < 0) continue;
    // a large fully-connected layer: the weights of this CTA's outputs, then those of its inputs
    for (int back = 0; back <= (backward && (s > 0 || in_grad) ? 1 : 0); ++back) {
      float *dst = wts + (back ? L.wb_off : L.wf_off);
      const int rows = back ? L.out_n : L.in_n, cols = back ? L.in_n : L.out_n;
      int first, count;
      share(cl, cols, &first, &count);
      if ((L.w_rows != 0) != (back != 0)) {
        if (tid == 0 && count) copy_in(dst, L.W + (size_t)first * rows, count * rows, &rest, false);
      } else if (count) {
        for (int k = tid; k < rows; k += SN_THREADS)
          copy_in(dst + k * share_pitch(cols, cl.n), L.W + (size_t)k * cols + first, count, &rest, false);
      }
    }
  }
  mbar_arrive(&rest);
  if (!mbar_wait_bounded(&here, 0)) cl.failed = true;
  if ((net.n == 1 || net.step[0].kind == SN_FC) && !mbar_wait_bounded(&rest, 0)) cl.failed = true;
  __syncthreads();
  mask_unconnected(net.step[0], wts);

  if constexpr (MODE == 2) {
    for (int s = 0; s < net.n; ++s) {
      const SmallStep &L = net.step[s];
      const size_t at = (size_t)sample * L.out_n;
      for (int i = tid; i < L.out_n; i += SN_THREADS) {
        act[L.out_off + i] = L.out[at + i];
        if (L.kind == SN_MAX) act[L.arg_off + i] = __int_as_float(L.argmax[at + i]);
      }
    }
    if (!cl.failed && !mbar_wait_bounded(&rest, 0)) cl.failed = true;
    for (int s = 1; s < net.n; ++s) mask_unconnected(net.step[s], wts);
    __syncthreads();
  }
  // ---- forward ----
  for (int s = 0; MODE != 2 && s < net.n; ++s) {
    const SmallStep &L = net.step[s];
    const float *in = act + L.in_off;
    float *out = act + L.out_off;
    if (s == 1) {
      if (!cl.failed && !mbar_wait_bounded(&rest, 0)) cl.failed = true;
      for (int k = 1; k < net.n; ++k) mask_unconnected(net.step[k], wts);
    }
    int first, count;
    share(cl, L.out_n, &first, &count);
    // value i of the layer: activation, to shared and to global memory
    auto emit = [&](int i, float v) {
      if (L.out_pre) L.out_pre[(size_t)sample * L.out_n + i] = v;
      v = apply_act_p(v, L.act, L.param);
      L.out[(size_t)sample * L.out_n + i] = v;
      out[i] = v;
    };
    auto with_bias = [&](int i, float v) { emit(i, v + (L.has_bias ? wts[L.b_off + L.d_op.of(i)] : 0.f)); };
    if (L.kind == SN_CONV && tiled_rows(L)) {
      if (L.KW == 5)
        conv_tiles<5, false>(L, in, wts + L.w_off, cl, with_bias, &first, &count);
      else
        conv_tiles<3, false>(L, in, wts + L.w_off, cl, with_bias, &first, &count);
    } else if (L.kind == SN_CONV) {
      const int kl = lanes_for(count, 3), ks = 1 << kl, total = count << kl;
      for (int base = 0; base < total; base += SN_THREADS) {
        const int idx = base + tid, i = first + (idx >> kl), part = idx & (ks - 1);
        const float v = lane_sum(idx < total ? conv_out(L, in, wts + L.w_off, i, part, ks) : 0.f, ks);
        if (idx < total && part == 0) with_bias(i, v);
      }
    } else if (L.kind == SN_FC && L.w_rows) {  // a warp for an output, lanes along the row of weights
      for (int i = first + warp; i < first + count; i += SN_WARPS) {
        const float *w = L.wf_off >= 0  ? wts + L.wf_off + misplaced(L.W + (size_t)first * L.in_n) + (i - first) * L.in_n
                         : L.w_off >= 0 ? wts + L.w_off + i * L.in_n
                                        : L.W + (size_t)i * L.in_n;
        float v = 0.f;
#pragma unroll 8
        for (int k = lane; k < L.in_n; k += 32) v = fmaf(in[k], w[k], v);
        v = warp_sum(v);
        if (lane == 0) emit(i, v + (L.has_bias ? wts[L.b_off + i] : 0.f));
      }
    } else if (L.kind == SN_FC) {  // lanes along the outputs, inputs dealt to groups of threads
      // rows of the share start off the 16-byte grid, each in its own place
      const float *w = L.wf_off >= 0 ? wts + L.wf_off : L.w_off >= 0 ? wts + L.w_off + first : L.W + first;
      const int stride = L.wf_off >= 0 ? share_pitch(L.out_n, cl.n) : L.out_n, 
                off1 = L.wf_off >= 0 ? misplaced(L.W + first) : 0, offk = L.wf_off >= 0 ? L.out_n & 3 : 0;
      const int pad = (count + 31) & ~31, parts = pad ? max(1, SN_THREADS / pad) : 1;
      for (int base = 0; base < count; base += SN_THREADS) {  // more than one turn only with one part
        const int j = parts == 1 ? base + tid : tid % pad, part = parts == 1 ? 0 : tid / pad;
        float v = 0.f;
        if (j < count && part < parts) {
#pragma unroll 8
          for (int k = part; k < L.in_n; k += parts) v = fmaf(in[k], w[k * stride + ((off1 + k * offk) & 3) + j], v);
        }
        __syncthreads();
        scratch[tid] = v;
        __syncthreads();
        if (part == 0 && j < count) {
          for (int q = 1; q < parts; ++q) v += scratch[q * pad + j];
          emit(first + j, v + (L.has_bias ? wts[L.b_off + first + j] : 0.f));
        }
      }
    } else if (L.kind == SN_AVG) {
      const float scale = 1.0f / (float)(L.KH * L.KW);
      for (int i = first + tid; i < first + count; i += SN_THREADS) {
        const int plane = L.OH * L.OW, c = L.d_op.of(i), r = i - c * plane, oy = L.d_ow.of(r);
        const float v = avg_window(L, in, c, oy, r - oy * L.OW);
        emit(i, __fadd_rn(__fmul_rn(v, __fmul_rn(wts[L.w_off + c], scale)), wts[L.b_off + c]));
      }
    } else if (L.kind == SN_MAX) {
      for (int i = first + tid; i < first + count; i += SN_THREADS) {
        const int plane = L.OH * L.OW, c = L.d_op.of(i), r = i - c * plane, oy = L.d_ow.of(r), y0 = oy * L.SH,
                  x0 = (r - oy * L.OW) * L.SW, ny = min(L.KH, L.HI - y0), nx = min(L.KW, L.WI - x0);
        float best = -FLT_MAX;
        int at = 0;
        for (int dy = 0; dy < ny; ++dy)
          for (int dx = 0; dx < nx; ++dx) {
            const int k = (L.HI * c + y0 + dy) * L.WI + x0 + dx;
            if (in[k] > best) best = in[k], at = k;
          }
        L.argmax[(size_t)sample * L.out_n + i] = at;
        if (backward) act[L.arg_off + i] = __int_as_float(at);
        emit(i, best);
      }
    } else if (L.kind == SN_SOFTMAX) {  // a few values: every CTA computes all of them
      float top = in[0], sum = 0.f;
      for (int k = 1; k < L.out_n; ++k) top = fmaxf(top, in[k]);
      for (int k = 0; k < L.out_n; ++k) sum += expf(in[k] - top);
      for (int i = tid; i < L.out_n; i += SN_THREADS) {
        const float v = expf(in[i] - top) / sum;
        out[i] = v;
        if (cl.rank == 0) L.out[(size_t)sample * L.out_n + i] = v;
      }
    } else {
      for (int i = first + tid; i < first + count; i += SN_THREADS) emit(i, in[i]);
    }
    if (L.kind == SN_SOFTMAX)
      __syncthreads();
    else
      cl.exchange(out, first, count, L.out_n, L.kind == SN_MAX && backward ? act + L.arg_off : nullptr);
  }
  auto finish = [&]() {
    if (cl.failed) atomicExch(net.err, 8);
    if (cl.n > 1 && cl.step == 0) asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
    if (cl.n > 1) cluster_barrier();  // nobody leaves while others may store into its shared memory
  };
  if (!backward) return finish();

  // ---- backward: grd at a step's out_off holds dE/d of its value before the activation ----
  {
    const SmallStep &L = net.step[net.n - 1];
    const float factor = 2.0f / (float)L.out_n, *y = act + L.out_off;
    float *g = grd + L.out_off;
    for (int i = tid; i < L.out_n; i += SN_THREADS) {
      const float dy = loss_grad_one(loss, y[i], t[(size_t)sample * L.out_n + i], factor);
      const float v = act_grad(L.act, L.param, y[i], dy);
      g[i] = v;
      if (cl.rank == 0) {
        L.grad[(size_t)sample * L.out_n + i] = dy;
        if (L.grad_pre) L.grad_pre[(size_t)sample * L.out_n + i] = v;
      }
    }
    __syncthreads();
  }
  for (int s = net.n - 1; s >= 0; --s) {
    const SmallStep &L = net.step[s];
    const float *in = act + L.in_off, *d = grd + L.out_off;
    float *part = L.part ? L.part + (size_t)sample * L.slices * L.part_len : nullptr;
    // weight gradients of this sample
    if (L.kind == SN_CONV) {
      if (L.KW == 5 && L.KH == 5)
        conv_dw_pairs<5>(L, in, d, part, cl);
      else if (L.KW == 3 && L.KH == 3)
        conv_dw_pairs<3>(L, in, d, part, cl);
      else
        conv_dw(L, in, d, part, cl);
    } else if (L.kind == SN_AVG) {
      const float scale = 1.0f / (float)(L.KH * L.KW);
      const int plane = L.OH * L.OW, span = L.span;
      for (int u = cl.rank * SN_WARPS + warp; u < L.C * L.slices; u += cl.n * SN_WARPS) {
        const int sl = L.d_c.of(u), c = u - sl * L.C;
        float sw = 0.f, sb = 0.f;
        for (int p = sl * span + lane; p < min(plane, sl * span + span); p += 32) {
          const float g = d[c * L.OH * L.OW + p];
          const int oy = L.d_ow.of(p);
          sb += g;
          sw = fmaf(avg_window(L, in, c, oy, p - oy * L.OW), g, sw);
        }
        sw = warp_sum(sw);
        sb = warp_sum(sb);
        if (lane == 0) {
          part[sl * L.part_len + c] = sw * scale;
          part[sl * L.part_len + L.C + c] = sb;
        }
      }
    }
    if (s == 0 && !in_grad) break;
    // dE/d input: the gradient of the step before, and through its activation
    const SmallStep &P = net.step[s > 0 ? s - 1 : 0];
    const bool input = s == 0;
    const int n = L.in_n;
    float *gin = grd + P.out_off;
    auto emit = [&](int i, float v) {
      if (input) {
        in_grad[(size_t)sample * n + i] = v;
        return;
      }
      P.grad[(size_t)sample * n + i] = v;
      v = act_grad(P.act, P.param, act[P.out_off + i], v);
      if (P.grad_pre) P.grad_pre[(size_t)sample * n + i] = v;
      gin[i] = v;
    };
    int first, count;
    share(cl, n, &first, &count);
    const bool exchange = !input && L.kind != SN_SOFTMAX;
    if (L.kind == SN_CONV && tiled_rows(L)) {
      if (L.KW == 5)
        conv_tiles<5, true>(L, d, wts + L.w_off, cl, emit, &first, &count);
      else
        conv_tiles<3, true>(L, d, wts + L.w_off, cl, emit, &first, &count);
    } else if (L.kind == SN_CONV) {
      const int kl = lanes_for(count, 3), ks = 1 << kl, total = count << kl;
      for (int base = 0; base < total; base += SN_THREADS) {
        const int idx = base + tid, i = first + (idx >> kl), p = idx & (ks - 1);
        const float v = lane_sum(idx < total ? conv_din(L, d, wts + L.w_off, i, p, ks) : 0.f, ks);
        if (idx < total && p == 0) emit(i, v);
      }
    } else if (L.kind == SN_FC && !L.w_rows) {  // weights [in][out]: a warp for an input
      for (int i = first + warp; i < first + count; i += SN_WARPS) {
        const float *w = L.wf_off >= 0  ? wts + L.wb_off + misplaced(L.W + (size_t)first * L.out_n) + (i - first) * L.out_n
                         : L.w_off >= 0 ? wts + L.w_off + i * L.out_n
                                        : L.W + (size_t)i * L.out_n;
        float v = 0.f;
#pragma unroll 4
        for (int k = lane; k < L.out_n; k += 32) v = fmaf(d[k], w[k], v);
        v = warp_sum(v);
        if (lane == 0) emit(i, v);
      }
    } else if (L.kind == SN_FC) {
      const float *w = L.wf_off >= 0 ? wts + L.wb_off : L.w_off >= 0 ? wts + L.w_off + first : L.W + first;
      const int stride = L.wf_off >= 0 ? share_pitch(L.in_n, cl.n) : L.in_n,
                off1 = L.wf_off >= 0 ? misplaced(L.W + first) : 0, offk = L.wf_off >= 0 ? L.in_n & 3 : 0;
      const int pad = (count + 31) & ~31, parts = pad ? max(1, SN_THREADS / pad) : 1;
      for (int base = 0; base < count; base += SN_THREADS) {
        const int j = parts == 1 ? base + tid : tid % pad, p = parts == 1 ? 0 : tid / pad;
        float v = 0.f;
        if (j < count && p < parts) {
#pragma unroll 8
          for (int k = p; k < L.out_n; k += parts) v = fmaf(d[k], w[k * stride + ((off1 + k * offk) & 3) + j], v);
        }
        __syncthreads();
        scratch[tid] = v;
        __syncthreads();
        if (p == 0 && j < count) {
          for (int q = 1; q < parts; ++q) v += scratch[q * pad + j];
          emit(first + j, v);
        }
      }
    } else if (L.kind == SN_AVG) {
      const float scale = 1.0f / (float)(L.KH * L.KW);
      const int nwy = (L.HI - L.KH) / L.SH + 1, nwx = (L.WI - L.KW) / L.SW + 1;
      for (int i = first + tid; i < first + count; i += SN_THREADS) {
        const int plane = L.HI * L.WI, c = L.d_ip.of(i), r = i - c * plane, iy = L.d_iw.of(r), ix = r - iy * L.WI;
        const int oy = iy < L.KH ? 0 : (iy - L.KH) / L.SH + 1, ox = ix < L.KW ? 0 : (ix - L.KW) / L.SW + 1;
        const bool covered = oy < nwy && ox < nwx && oy * L.SH <= iy && ox * L.SW <= ix && oy < L.OH && ox < L.OW;
        emit(i, covered ? __fmul_rn(__fmul_rn(wts[L.w_off + c], scale), d[(L.OH * c + oy) * L.OW + ox]) : 0.f);
      }
    } else if (L.kind == SN_MAX) {
      for (int i = first + tid; i < first + count; i += SN_THREADS) {
        const int plane = L.HI * L.WI, c = L.d_ip.of(i), r = i - c * plane, iy = L.d_iw.of(r), ix = r - iy * L.WI;
        const int oy = min(iy / L.SH, L.OH - 1), ox = min(ix / L.SW, L.OW - 1);
        const bool covered = iy < oy * L.SH + L.KH && ix < ox * L.SW + L.KW;
        const int w = covered ? (L.OH * c + oy) * L.OW + ox : 0;
        emit(i, __float_as_int(act[L.arg_off + w]) == i ? d[w] : 0.f);
      }
    } else if (L.kind == SN_SOFTMAX) {  // every CTA computes all of it
      const float *y = act + L.out_off;
      for (int j = tid; j < n; j += SN_THREADS) {
        float v = 0.f;
        for (int k = 0; k < n; ++k)
          v = __fadd_rn(v, __fmul_rn(d[k], k == j ? __fmul_rn(y[j], __fsub_rn(1.f, y[j])) : __fmul_rn(-y[k], y[j])));
        if (input) {
          if (cl.rank == 0) in_grad[(size_t)sample * n + j] = v;
          continue;
        }
        const float pre = act_grad(P.act, P.param, act[P.out_off + j], v);
        gin[j] = pre;
        if (cl.rank == 0) {
          P.grad[(size_t)sample * n + j] = v;
          if (P.grad_pre) P.grad_pre[(size_t)sample * n + j] = pre;
        }
      }
    } else {
      for (int i = first + tid; i < first + count; i += SN_THREADS) emit(i, d[i]);
    }
    if (exchange)
      cl.exchange(gin, first, count, n);
    else
      __syncthreads();
  }
  finish();
}

// Weight gradients, the rows of the samples added in order.  Up to 64 rows a thread owns an entry; of more, thread
// row k of a block adds rows k, k + 8, ... of 32 entries and the eight sums are added in order.
__host__ __device__ __forceinline__ int reduce_entries(const SmallStep &L, int B) { return B * L.slices <= 64 ? 256 : 32; }

__global__ void __launch_bounds__(256) small_reduce_kernel(const __grid_constant__ SmallNet net, const float *__restrict__ x,
                                                           int B) {
  after_previous_kernel();
  __shared__ float lanes[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  int s = 0, blk = blockIdx.x, per_block;
  for (;; ++s) {
    per_block = reduce_entries(net.step[s], B);
    const int nb = (net.step[s].w_len + net.step[s].b_len + per_block - 1) / per_block;
    if (blk < nb) break;
    blk -= nb;
  }
  const SmallStep &L = net.step[s];
  const bool split = per_block == 32;
  const int e = blk * per_block + (split ? tx : (int)threadIdx.x), first = split ? ty : 0, step = split ? 8 : 1;
  const int wlen = L.w_len, blen = L.b_len;
  const bool live = e < wlen + blen;
  float v = 0.f;
  if (live && L.kind == SN_FC) {
    const float *in = s > 0 ? net.step[s - 1].out : x;
    if (e < wlen) {
      const int o = L.w_rows ? e / L.in_n : e % L.out_n, k = L.w_rows ? e - o * L.in_n : e / L.out_n;
#pragma unroll 8
      for (int b = first; b < B; b += step) v = fmaf(in[(size_t)b * L.in_n + k], L.delta[(size_t)b * L.out_n + o], v);
    } else {
#pragma unroll 8
      for (int b = first; b < B; b += step) v += L.delta[(size_t)b * L.out_n + e - wlen];
    }
  } else if (live) {
    // average pooling has K * K weights a channel, of which the first alone is used
    const int i = L.kind == SN_CONV || e < L.C ? e : e >= wlen ? e - wlen + L.C : -1;
    if (i >= 0) {
#pragma unroll 8
      for (int r = first; r < B * L.slices; r += step) v += L.part[(size_t)r * L.part_len + i];
    }
  }
  if (split) {
    lanes[ty][tx] = v;
    __syncthreads();
    if (ty != 0) return;
#pragma unroll
    for (int k = 1; k < 8; ++k) v += lanes[k][tx];
  }
  if (live) (e < wlen ? L.dW[e] : L.db[e - wlen]) = v;
}

size_t small_smem(const SmallNet &n, int backward) {
  return ((size_t)(n.n_act + 3) / 4 * 4 * (backward ? 2 : 1) + n.n_wts + SN_THREADS) * sizeof(float);
}

// what a block may ask for at launch: all but the kernel's own shared variables
constexpr size_t SN_OWN_SMEM = (SN_EXCHANGES + 2) * 8;
size_t small_room(const b200_ctx *ctx) { return ctx->smem_optin - SN_OWN_SMEM; }

// Places for the parameters in shared memory: [weights | biases] of convolutions, pooling and small fully-connected
// layers whole; of large fully-connected layers the biases, and a CTA's shares of the weights as far as they fit.
void place_params(const b200_ctx *ctx, SmallNet *n, int nc, int backward) {
  n->n_wts = 0;
  for (int i = 0; i < n->n; ++i) {
    SmallStep &L = n->step[i];
    L.w_off = L.wf_off = L.wb_off = L.b_off = -1;
    if (L.w_len == 0) continue;
    const bool whole = L.kind != SN_FC || L.w_len <= SN_WHOLE;
    L.copy = whole ? L.W : L.b;
    L.copy_n = (whole ? L.w_len : 0) + L.b_len;
    L.copy_off = n->n_wts;
    const int at = n->n_wts + (int)(((uintptr_t)L.copy >> 2) & 3);
    if (whole) L.w_off = at;
    L.b_off = at + (whole ? L.w_len : 0);
    n->n_wts += (L.copy_n + 3 + 3) / 4 * 4;
  }
  for (int i = n->n - 1; i >= 0; --i) {
    SmallStep &L = n->step[i];
    if (L.kind != SN_FC || L.w_off >= 0) continue;
    const int out = (ceil_div(L.out_n, nc) * L.in_n + 3 + 3) / 4 * 4, in = (ceil_div(L.in_n, nc) * L.out_n + 3 + 3) / 4 * 4;
    const int fwd = L.w_rows ? out : L.in_n * share_pitch(L.out_n, nc);
    const int bwd = !backward ? 0 : L.w_rows ? L.out_n * share_pitch(L.in_n, nc) : in;
    if (small_smem(*n, backward) + ((size_t)fwd + bwd) * sizeof(float) > small_room(ctx)) continue;
    L.wf_off = n->n_wts;
    L.wb_off = n->n_wts + fwd;
    n->n_wts += fwd + bwd;
  }
}

using SmallKernel = void (*)(SmallNet, const float *, const float *, float *, int);

// Whether B clusters of nc CTAs leave one place in fifteen free: clusters that fill the chip wait for each other's SMs
bool leaves_room(const SmallNet &n, int nc, int B) { return nc <= 2 || B * 15 <= n.clusters[nc - 1] * 14; }

// Multiply-adds of a sample's forward pass, for a choice below `nc` CTAs.  Those of a fully-connected layer, which read a weight
// each, take 2.5 times as long; three CTAs, whose shares of the weights lie off the 16-byte grid, are no faster at them than two.
double small_macs(const SmallNet &n, int nc) {
  double macs = 0;
  for (int i = 0; i < n.n; ++i)
    macs += n.step[i].kind == SN_CONV               ? (double)n.step[i].out_n * n.step[i].C * n.step[i].KH * n.step[i].KW
            : n.step[i].kind == SN_FC && nc != 3 ? 2.5 * n.step[i].w_len
                                                    : 0.0;
  return macs;
}

// CTAs for one sample: up to eight (what a cluster may have anywhere), as many as let all samples run at once; how many clusters the
// chip holds depends on how its SMs are grouped (15 of eight, 22 of six, 26 of five, 33 of four, 45 of three, 74 of two).  Any number, not
// powers of two alone: a LeNet-5 step of 16 samples 60 us with four CTAs a sample, 53 with six; of 40 samples 88 with two, 70 with
// three.  More than eight is no faster: one sample 49 us with eight, 51 with sixteen, which have to send to each other.
// A prediction whose clusters fill the chip takes the next fewer CTAs that leave room, which costs a larger share of the products and saves
// 2 us: 3x3 nets of two layers 18.6 us with 22 samples on clusters of six, 15.7 on clusters of five; 784-200-200-10, 26 samples 20.7 on
// five, 16.8 on four.  Not where that share grows by more than 35 thousand (LeNet-5, 45 samples: 24.8 us with three CTAs, 27.1 with
// two, 33 samples 22.8 either way; 784-200-200-10, 32 samples 18.7 with four, 19.1 with three).
int small_cluster(const SmallNet &n, int B, bool predict) {
  int nc = SN_MAX_CTAS;
  while (nc > 1 && B > n.clusters[nc - 1]) --nc;
  if (predict && !leaves_room(n, nc, B)) {
    int less = nc - 1;
    while (!leaves_room(n, less, B)) --less;  // two always do
    if (small_macs(n, nc) * (1.0 / less - 1.0 / nc) < 35e3) nc = less;
  }
  return nc;
}

}  // namespace

bool small_net_fits(const b200_ctx *ctx, const SmallNet &n) {
  if (n.n == 0) return false;
  SmallNet m = n;
  place_params(ctx, &m, 1, 1);
  return small_smem(m, 1) <= small_room(ctx);
}

// Microseconds of a pass either way, fitted (non-negative least squares) to 24 networks of 1 to 7 steps at 17 (predictions) and 29
// (steps) batches from 1 to 2048.
//   A step: on clusters of any size and with the layers' kernels as they are; where neither form is three times the other the fits
// are off by 11 to 13 % (rms), and taking the cheaper one by them costs 1 % on average against always taking the faster
// one.  (With terms of clusters of 1, 2, 4 and 8 and of the layers' older kernels it cost 7 %, and 784-30-10 went to the
// whole-network kernels at 22 samples, 31 us against 21.)
//   A prediction: from those older kernels.  The layers, which have to win by a tenth here, are faster than it knows since a launch
// overlaps the end of the one before it: that costs 11 % on average over the same networks (784-64-64-10, 16 samples: 15.0 us
// in one kernel, 9.8 in four).
//   Whole-network kernels: a phase a step and, for each turn of samples that an SM takes, the products of its CTA; the
// sums over the samples read a sample's values, or its row of partial sums, for every weight.  Windows other than 3 and
// 5 wide have no tiled form.  Layer by layer: launches, then the values that pass through memory; average pooling's
// backward pass is the slow one, and a softmax of more than 16 values, which is one thread's work a sample.
//   (LeNet-5 step: 16 samples 53 us against 104, 592 samples 531 against 785; 3x3 16 -> 16 -> 16 -> 4 on 16x16 maps: 12
// samples 53 us against 66, 60 samples 122 against 83.)
bool small_net_pays(const SmallNet &n, int B, bool train) {
  if (n.n == 0) return false;
  const int nc = small_cluster(n, B, false);
  const double turns = (B + n.clusters[nc - 1] - 1) / n.clusters[nc - 1];
  double weights = 0, tiled = 0, slow = 0, square = 0, fc = 0, fc_all = 0, values = 0, rows = 0;  // of a CTA; of all
  double launches = 0, through = 0, averaged = 0;                                                  // layer by layer
  for (int i = 0; i < n.n; ++i) {
    const SmallStep &L = n.step[i];
    const double v = L.in_n + L.out_n, taps = (double)L.KH * L.KW;
    values += v;
    if (L.kind == SN_CONV) {
      const double macs = L.out_n * L.C * taps;
      const bool fast = (L.KW == 3 || L.KW == 5) && L.SH == 1 && L.SW == 1 && L.DH == 1 && L.DW == 1;
      (fast ? tiled : slow) += macs / nc;
      if (L.KH == L.KW && (L.KW == 3 || L.KW == 5)) square += macs / nc;
      rows += L.w_len;
      weights += L.w_len;
      launches += train ? 21 : 8.6;
    } else if (L.kind == SN_FC) {
      fc += (double)L.w_len / nc;
      fc_all += L.w_len;
      weights += L.w_len <= SN_WHOLE ? L.w_len : (double)L.w_len / nc * (train ? 2 : 1);
      launches += train ? 6.6 : 5.1;
    } else if (L.kind == SN_MAX) {
      launches += train ? 0.7 : 4.1;
    } else if (L.kind == SN_AVG) {
      launches += train ? 4.2 : 2.8;
    } else if (L.kind == SN_SOFTMAX && L.out_n > 16 && train) {
      launches += 0.023 * L.out_n * L.out_n;
    }
    if (L.own_act) launches += train ? 5.8 : 5.1;
    (L.kind == SN_AVG ? averaged : through) += v;
  }
  if (!train)
    return 6.5 + turns * (1.8 * n.n + 0.6e-4 * weights + 0.4e-4 * tiled + 1e-4 * slow + 0.18e-4 * fc + 0.075e-3 * values) <
           1.1 * (2.8 + launches + B * (0.083e-6 * fc_all + 4.1e-6 * through + 4.8e-6 * averaged));
  const double chain = B <= 64 ? B : B / 8.0;  // rows that a thread of the sums adds
  return 7.3 + turns * (4.7 * n.n + 2.2e-4 * weights + 37e-4 * slow + 1.3e-4 * square + 0.06e-4 * fc + 0.47e-3 * values) +
           0.073 * chain + B * (1.1e-6 * fc_all + 110e-6 * rows) <
         5.7 + launches + B * (0.77e-6 * fc_all + 19e-6 * through + 140e-6 * averaged);
}

// The counts depend on the device alone (a CTA's registers leave no room for a second one on its SM, whatever its shared memory), and the
// driver takes a tenth of a millisecond and more to work one out: they are asked for once.
int small_net_plan(b200_ctx *ctx, SmallNet *n) {
  static std::mutex lock;
  static std::map<int, std::array<int, SN_MAX_CTAS>> known;
  std::lock_guard<std::mutex> guard(lock);
  auto it = known.find(ctx->device);
  if (it == known.end()) {
    std::array<int, SN_MAX_CTAS> most;
    const size_t smem = small_room(ctx);
    B200_CUDA(cudaFuncSetAttribute(small_net_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int nc = 1; nc <= SN_MAX_CTAS; ++nc) {
      cudaLaunchAttribute at;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = (unsigned)nc;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cudaLaunchConfig_t c = {};
      c.gridDim = dim3((unsigned)nc);
      c.blockDim = dim3(SN_THREADS);
      c.dynamicSmemBytes = smem;
      c.stream = ctx->stream;
      c.attrs = &at;
      c.numAttrs = 1;
      B200_CUDA(cudaOccupancyMaxActiveClusters(&most[nc - 1], small_net_kernel<1>, &c));
    }
    it = known.emplace(ctx->device, most).first;
  }
  std::copy(it->second.begin(), it->second.end(), n->clusters);
  return 0;
}

int small_net_run(b200_ctx *ctx, const SmallNet &n, const float *x, const float *t, float *in_grad, int B,
                  int backward, int loss) {
  B200_REQUIRE(!backward || (loss >= B200_LOSS_MSE && loss <= B200_LOSS_CROSS_ENTROPY_MULTICLASS),
               "loss_grad: unknown loss %d", loss);
  const int nc = small_cluster(n, B, !backward);
  SmallNet m = n;
  m.by_ctas.set(nc);
  place_params(ctx, &m, nc, backward);
  const SmallKernel kernel = backward == 0 ? small_net_kernel<0> : backward == 1 ? small_net_kernel<1> : small_net_kernel<2>;
  const size_t smem = small_smem(m, backward);
  B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // A prediction's launch, plan and barriers overlap the end of the kernel before it in the stream (LeNet-5, one sample: 20.5 us a call
  // behind another prediction, 18.7 so; with an elementwise kernel in front of each 22.6 and 20.6; behind an upload 25.5 to 26.6
  // either way), but not where its clusters only fit if nothing else lies between them: 45 of three CTAs took 28.7 us for
  // 24.6.  The kernels with a backward pass do not wait for the one before them: steps are captured, where a launch costs little.
  const bool overlap = !backward && ctx->overlap && !ctx->waited && leaves_room(n, nc, B);
  B200_TRY(launch_kernel_as(ctx, overlap, kernel, dim3((unsigned)(B * nc)), dim3(SN_THREADS), smem, dim3((unsigned)nc), m, x, t,
                            in_grad, loss));
  if (!backward) return 0;
  int blocks = 0;
  for (int i = 0; i < n.n; ++i) blocks += ceil_div(n.step[i].w_len + n.step[i].b_len, reduce_entries(n.step[i], B));
  if (blocks == 0) return 0;
  B200_TRY(launch_kernel(ctx, small_reduce_kernel, dim3(blocks), dim3(256), 0, 1, n, x, B));
  return 0;
}

}  // namespace b200
