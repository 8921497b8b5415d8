// Layers that commonly sit between the hot operators of a tiny-dnn network: batch normalization
// (forward in both phases, backward), dropout with a mask supplied by the host, and the forward pass
// of local response normalization across channels (its backward pass does not exist in the
// reference).  All are HBM-bound: a per-channel reduction over batch x spatial positions, or one
// pass over the tensor.
#include "common.cuh"
#include "device_utils.cuh"

namespace b200 {

namespace {

constexpr int BN_THREADS = 256;

// Slices of the batch a channel's reduction is cut into: enough blocks to fill the GPU, few enough
// that every later block can add the slices up again by itself.
__host__ __device__ inline int bn_slices(int B, int channels, int sm_count) {
  int want = (4 * sm_count + channels - 1) / channels;
  if (want > 64) want = 64;
  if (want > B) want = B;
  return want < 1 ? 1 : want;
}

// sum of `vals` over the block, returned to every thread
__device__ __forceinline__ float block_sum_all(float v) {
  __shared__ float total;
  v = block_sum(v);
  if (threadIdx.x == 0) total = v;
  __syncthreads();
  v = total;
  __syncthreads();
  return v;
}

__device__ __forceinline__ void warp_sum2(double &a, double &b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
}

// the slices' results of channel c, fetched side by side (one after the other they cost a block 6 us)
struct Slices {
  float a[64], b[64];
  __device__ __forceinline__ void fetch(const float *pa, const float *pb, int c, int C, int slices) {
    if ((int)threadIdx.x < slices) {
      a[threadIdx.x] = pa[(size_t)threadIdx.x * C + c];
      b[threadIdx.x] = pb[(size_t)threadIdx.x * C + c];
    }
    __syncthreads();
  }
};
// added in slice order (every block gets the same bits)
__device__ __forceinline__ float add_slices(const float *part, int slices) {
  float s = 0.f;
  for (int z = 0; z < slices; ++z) s += part[z];
  return s;
}

// Every value, or 16-byte piece (S4 of them a map), of channel c in the samples n0 .. n1 - 1: f(its index).  One loop over all of them, so
// that a thread has several loads on the way; a loop per sample had one (256 samples of 64 maps of 32x32: 29 us for
// the 67 MB of a forward sum).
template <typename F>
__device__ __forceinline__ void pieces_of(int c, int C, int S4, int n0, int n1, F f) {
  const unsigned total = (unsigned)(n1 - n0) * (unsigned)S4;
  const size_t base = ((size_t)n0 * C + c) * S4, skip = (size_t)(C - 1) * S4;
#pragma unroll 8
  for (unsigned i = threadIdx.x; i < total; i += BN_THREADS) f(base + i + (i / (unsigned)S4) * skip);
}

// The same for a pass that also stores: `load` fetches the operands of four pieces before `store` writes the first,
// because the compiler may not move a load past a store on its own.
template <typename V, typename Load, typename Store>
__device__ __forceinline__ void pieces_map(int c, int C, int S4, int n0, int n1, Load load, Store store) {
  const unsigned total = (unsigned)(n1 - n0) * (unsigned)S4;
  const size_t base = ((size_t)n0 * C + c) * S4, skip = (size_t)(C - 1) * S4;
  for (unsigned i = threadIdx.x; i < total; i += 4 * BN_THREADS) {
    V v[4];
    size_t at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned k = min(i + u * BN_THREADS, total - 1);
      at[u] = base + k + (k / (unsigned)S4) * skip;
      v[u] = load(at[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * BN_THREADS < total) store(at[u], v[u]);
  }
}

// moments() (tiny_dnn/util/math_functions.h:25-61) in one pass: per (channel, batch slice) the sums of x and of x^2 in
// double precision, where their difference keeps 32-bit accuracy for a mean of up to thousands of deviations.  Of eight
// values at a time only the mean takes part in that, five operations on the double-precision pipe in place of 24 (256
// samples of 64 maps of 32x32: 6 us less); the squares about it are summed in 32 bits.  (In 32 bits relative to a rough mean of four values of a slice, one value a million deviations off among them
// left the variance with five digits.)
__global__ void __launch_bounds__(BN_THREADS) bn_moments_kernel(const float *__restrict__ x, int S, int B,
                                                                double2 *__restrict__ part, int vec4) {
  after_previous_kernel();
  const int c = blockIdx.x, C = gridDim.x, z = blockIdx.y, Z = gridDim.y;
  const int n0 = (int)((long long)B * z / Z), n1 = (int)((long long)B * (z + 1) / Z);
  double s1 = 0., s2 = 0.;
  if (vec4) {
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    float about = 0.f;
    const unsigned S4 = (unsigned)S / 4, total = (unsigned)(n1 - n0) * S4;
    const size_t base = ((size_t)n0 * C + c) * S4, skip = (size_t)(C - 1) * S4;
    auto piece = [&](unsigned i) { return x4[base + i + (i / S4) * skip]; };
    unsigned i = threadIdx.x;
#pragma unroll 4
    for (; i + BN_THREADS < total; i += 2 * BN_THREADS) {
      const float4 v = piece(i), w = piece(i + BN_THREADS);
      const float a = v.y - v.x, b = v.z - v.x, e = v.w - v.x, f = w.x - v.x, g = w.y - v.x, h = w.z - v.x, k = w.w - v.x;
      const float d = ((a + b) + (e + f)) + ((g + h) + k), m = 0.125f * d;
      auto sq = [&](float t, float u) { return fmaf(t - m, t - m, (u - m) * (u - m)); };
      about += (sq(0.f, a) + sq(b, e)) + (sq(f, g) + sq(h, k));
      const double mean = fma(0.125, (double)d, (double)v.x);
      s1 += mean;
      s2 = fma(mean, mean, s2);
    }
    s1 *= 8.;
    s2 = fma(8., s2, (double)about);
    if (i < total) {
      const float4 v = piece(i);
      const double a = v.x, b = v.y, e = v.z, f = v.w;
      s1 += (a + b) + (e + f);
      s2 += fma(a, a, b * b) + fma(e, e, f * f);
    }
  } else {
    pieces_of(c, C, S, n0, n1, [&](size_t i) {
      const double a = x[i];
      s1 += a;
      s2 = fma(a, a, s2);
    });
  }
  __shared__ double2 warps[BN_THREADS / 32];
  warp_sum2(s1, s2);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = make_double2(s1, s2);
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < BN_THREADS / 32; ++w) s1 += warps[w].x, s2 += warps[w].y;
    part[(size_t)z * C + c] = make_double2(s1, s2);
  }
}

// by a warp: mean and sum of (x - mean)^2 of channel c over all slices, added by a fixed tree (every block gets the same bits)
__device__ __forceinline__ void merge_slices(const double2 *part, int c, int C, int slices, double count, float *mean_out,
                                             float *sq_out) {
  double s1 = 0., s2 = 0.;
  for (int z = threadIdx.x; z < slices; z += 32) {
    const double2 p = part[(size_t)z * C + c];
    s1 += p.x;
    s2 += p.y;
  }
  warp_sum2(s1, s2);
  const double mean = s1 / count, sq = s2 - s1 * mean;
  *mean_out = (float)mean;
  *sq_out = (float)(sq < 0. ? 0. : sq);
}

// backward: per (channel, batch slice) the sums of dy and of dy * y
__global__ void __launch_bounds__(BN_THREADS) bn_sum_kernel(const float *__restrict__ x, const float *__restrict__ y,
                                                            int S, int B, float *__restrict__ part_x,
                                                            float *__restrict__ part_xy, int vec4) {
  after_previous_kernel();
  const int c = blockIdx.x, C = gridDim.x, z = blockIdx.y, Z = gridDim.y;
  const int n0 = (int)((long long)B * z / Z), n1 = (int)((long long)B * (z + 1) / Z);
  float sx = 0.f, sxy = 0.f;
  if (vec4) {  // 16-byte loads: S a multiple of 4 and the tensors 16-byte aligned (checked by the launcher)
    const float4 *x4 = reinterpret_cast<const float4 *>(x), *y4 = reinterpret_cast<const float4 *>(y);
    pieces_of(c, C, S / 4, n0, n1, [&](size_t i) {
      const float4 v = x4[i], w = y4[i];
      sx += (v.x + v.y) + (v.z + v.w);
      sxy += (v.x * w.x + v.y * w.y) + (v.z * w.z + v.w * w.w);
    });
  } else {
    pieces_of(c, C, S, n0, n1, [&](size_t i) {
      const float v = x[i];
      sx += v;
      sxy += v * y[i];
    });
  }
  sx = block_sum_all(sx);
  sxy = block_sum_all(sxy);
  if (threadIdx.x == 0) {
    part_x[(size_t)z * C + c] = sx;
    part_xy[(size_t)z * C + c] = sxy;
  }
}

// y = (x - mean) / sqrt(variance + eps) (batch_normalization_layer.h:136-168).  Train phase
// (part != nullptr): mean and variance come from the slices (variance over max(1, B*S - 1)) and are
// stored by the channel's first block; test phase: they are read.
__global__ void __launch_bounds__(BN_THREADS) bn_apply_kernel(const float *__restrict__ x, float *__restrict__ y, int S,
                                                              int B, float eps, int slices,
                                                              const double2 *__restrict__ part, float *mean_io, float *var_io,
                                                              float *__restrict__ stddev, int vec4) {
  after_previous_kernel();
  const int c = blockIdx.x, C = gridDim.x, z = blockIdx.y, Z = gridDim.y;
  float mean, var;
  if (part != nullptr) {
    __shared__ float both[2];
    if (threadIdx.x < 32) {
      float m, sq;
      merge_slices(part, c, C, slices, (double)B * S, &m, &sq);
      if (threadIdx.x == 0) both[0] = m, both[1] = sq;
    }
    __syncthreads();
    mean = both[0];
    const float sq = both[1];
    var = __fdiv_rn(sq, fmaxf(1.0f, __fsub_rn((float)((long long)B * S), 1.0f)));
  } else {
    mean = mean_io[c];
    var = var_io[c];
  }
  const float sd = __fsqrt_rn(__fadd_rn(var, eps));
  if (z == 0 && threadIdx.x == 0) {
    if (part != nullptr) {
      mean_io[c] = mean;
      var_io[c] = var;
    }
    stddev[c] = sd;
  }
  const int n0 = (int)((long long)B * z / Z), n1 = (int)((long long)B * (z + 1) / Z);
  if (vec4) {
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    float4 *y4 = reinterpret_cast<float4 *>(y);
    pieces_map<float4>(c, C, S / 4, n0, n1, [&](size_t i) { return x4[i]; }, [&](size_t i, float4 v) {
      v.x = __fdiv_rn(__fsub_rn(v.x, mean), sd);
      v.y = __fdiv_rn(__fsub_rn(v.y, mean), sd);
      v.z = __fdiv_rn(__fsub_rn(v.z, mean), sd);
      v.w = __fdiv_rn(__fsub_rn(v.w, mean), sd);
      y4[i] = v;
    });
    return;
  }
  pieces_map<float>(c, C, S, n0, n1, [&](size_t i) { return x[i]; },
                    [&](size_t i, float v) { y[i] = __fdiv_rn(__fsub_rn(v, mean), sd); });
}

// dx = (dy - mean(dy) - mean(dy*y) * y) / stddev (batch_normalization_layer.h:94-134).  Five blocks an SM, so that the grid of about
// four is there at once: with four a few blocks made a second turn (256 samples of 64 maps of 32x32: 35.8 us, now 31).
__global__ void __launch_bounds__(BN_THREADS, 5) bn_bwd_kernel(const float *__restrict__ y, const float *__restrict__ dy,
                                                            float *__restrict__ dx, int S, int B, int slices,
                                                            const float *__restrict__ part_d,
                                                            const float *__restrict__ part_dy,
                                                            const float *__restrict__ stddev, int vec4) {
  after_previous_kernel();
  const int c = blockIdx.x, C = gridDim.x, z = blockIdx.y, Z = gridDim.y;
  const float count = (float)B * (float)S;
  __shared__ Slices p;
  p.fetch(part_d, part_dy, c, C, slices);
  const float mean_d = __fdiv_rn(add_slices(p.a, slices), count);
  const float mean_dy = __fdiv_rn(add_slices(p.b, slices), count);
  const float sd = stddev[c];
  const int n0 = (int)((long long)B * z / Z), n1 = (int)((long long)B * (z + 1) / Z);
  if (vec4) {
    const float4 *y4 = reinterpret_cast<const float4 *>(y), *g4 = reinterpret_cast<const float4 *>(dy);
    float4 *d4 = reinterpret_cast<float4 *>(dx);
    struct Pair {
      float4 a, g;
    };
    pieces_map<Pair>(c, C, S / 4, n0, n1, [&](size_t i) { return Pair{y4[i], g4[i]}; }, [&](size_t i, const Pair &p) {
      const float4 a = p.a, g = p.g;
      float4 o;
      o.x = __fdiv_rn(__fsub_rn(__fsub_rn(g.x, mean_d), __fmul_rn(mean_dy, a.x)), sd);
      o.y = __fdiv_rn(__fsub_rn(__fsub_rn(g.y, mean_d), __fmul_rn(mean_dy, a.y)), sd);
      o.z = __fdiv_rn(__fsub_rn(__fsub_rn(g.z, mean_d), __fmul_rn(mean_dy, a.z)), sd);
      o.w = __fdiv_rn(__fsub_rn(__fsub_rn(g.w, mean_d), __fmul_rn(mean_dy, a.w)), sd);
      d4[i] = o;
    });
    return;
  }
  pieces_map<float2>(c, C, S, n0, n1, [&](size_t i) { return make_float2(y[i], dy[i]); }, [&](size_t i, float2 v) {
    dx[i] = __fdiv_rn(__fsub_rn(__fsub_rn(v.y, mean_d), __fmul_rn(mean_dy, v.x)), sd);
  });
}

// running = momentum * running + (1 - momentum) * current (batch_normalization_layer.h:174-180)
__global__ void bn_post_update_kernel(int C, float momentum, float *__restrict__ mean, float *__restrict__ var,
                                      const float *__restrict__ mean_cur, const float *__restrict__ var_cur,
                                      const int *__restrict__ skip_if) {
  if (skip_if != nullptr && *skip_if != 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= C) return;
  const float one_m = __fsub_rn(1.0f, momentum);
  mean[i] = __fadd_rn(__fmul_rn(momentum, mean[i]), __fmul_rn(one_m, mean_cur[i]));
  var[i] = __fadd_rn(__fmul_rn(momentum, var[i]), __fmul_rn(one_m, var_cur[i]));
}

// dropout_layer.h:95-115 (train phase): out = mask * scale * in; :66-84: dx = mask * dy (no scale)
__global__ void dropout_kernel(const float *__restrict__ in, const uint8_t *__restrict__ mask, float scale,
                               float *__restrict__ out, size_t n) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t step = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += step) out[i] = __fmul_rn(__fmul_rn((float)mask[i], scale), in[i]);
}

// lrn_layer.h:110-143 (across channels): a window of `size` channels slides over the channel axis,
// the running sum of squares gains channel i + size/2 and loses channel i - size + size/2 in that
// order, out = in * (1 + alpha/size * sum)^-beta.  One thread per pixel walks the channels, so the
// running sum has the reference's additions and subtractions in the reference's order.
__global__ void lrn_across_fwd_kernel(const float *__restrict__ in, float *__restrict__ out, int C, int area, int size,
                                      float alpha_div_size, float beta, long long total) {
  long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (; idx < total; idx += step) {
    const long long n = idx / area;
    const int j = (int)(idx - n * area);
    const float *ip = in + (size_t)n * C * area + j;
    float *op = out + (size_t)n * C * area + j;
    float sq = 0.f;
    for (int i = 0; i < size / 2 && i < C; ++i) {
      const float v = ip[(size_t)i * area];
      sq = __fadd_rn(sq, __fmul_rn(v, v));
    }
    int head = size / 2;
    long long tail = (long long)head - size;
    for (int i = 0; i < C; ++i, ++head, ++tail) {
      if (head < C) {
        const float v = ip[(size_t)head * area];
        sq = __fadd_rn(sq, __fmul_rn(v, v));
      }
      if (tail >= 0) {
        const float v = ip[(size_t)tail * area];
        sq = __fsub_rn(sq, __fmul_rn(v, v));
      }
      op[(size_t)i * area] = __fmul_rn(ip[(size_t)i * area], powf(__fadd_rn(1.0f, __fmul_rn(alpha_div_size, sq)), -beta));
    }
  }
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int elementwise_grid(size_t n, int sm_count) {
  size_t blocks = (n + 255) / 256, cap = (size_t)sm_count * 16;
  if (blocks > cap) blocks = cap;
  return (int)(blocks < 1 ? 1 : blocks);
}

}  // namespace

size_t batchnorm_scratch_floats(const b200_ctx *ctx, int channels, int B) {
  return (size_t)4 * bn_slices(B > 0 ? B : 1, channels, ctx->sm_count) * channels;
}

// `scratch`: batchnorm_scratch_floats floats.  train != 0: mean / variance are outputs (this batch's
// moments); train == 0: inputs.  stddev is always an output.
int batchnorm_fwd(b200_ctx *ctx, int channels, int spatial, float eps, const float *x, float *mean, float *variance,
                  float *stddev, float *y, int B, int train, float *scratch) {
  if (B == 0) return 0;
  const int Z = bn_slices(B, channels, ctx->sm_count);
  const dim3 grid(channels, Z);
  double2 *part = reinterpret_cast<double2 *>(scratch);
  const int vec4 = spatial % 4 == 0 && aligned16(x) && aligned16(y);
  if (train) {
    B200_TRY(launch_kernel(ctx, bn_moments_kernel, dim3(grid), dim3(BN_THREADS), 0, 1, x, spatial, B, part, vec4));
  }
  B200_TRY(launch_kernel(ctx, bn_apply_kernel, dim3(grid), dim3(BN_THREADS), 0, 1, x, y, spatial, B, eps, Z,
                         train ? part : nullptr, mean, variance, stddev, vec4));
  return 0;
}

int batchnorm_bwd(b200_ctx *ctx, int channels, int spatial, const float *y, const float *dy, const float *stddev,
                  float *dx, int B, float *scratch) {
  if (B == 0) return 0;
  const int Z = bn_slices(B, channels, ctx->sm_count);
  const dim3 grid(channels, Z);
  float *part_d = scratch, *part_dy = scratch + (size_t)Z * channels;
  const int vec4 = spatial % 4 == 0 && aligned16(y) && aligned16(dy) && aligned16(dx);
  B200_TRY(launch_kernel(ctx, bn_sum_kernel, dim3(grid), dim3(BN_THREADS), 0, 1, dy, y, spatial, B, part_d, part_dy, vec4));
  B200_TRY(launch_kernel(ctx, bn_bwd_kernel, dim3(grid), dim3(BN_THREADS), 0, 1, y, dy, dx, spatial, B, Z, part_d, part_dy,
                         stddev, vec4));
  return 0;
}

int batchnorm_post_update(b200_ctx *ctx, int channels, float momentum, float *mean, float *variance,
                          const float *mean_cur, const float *var_cur, const int *skip_if) {
  bn_post_update_kernel<<<ceil_div(channels, 128), 128, 0, ctx->stream>>>(channels, momentum, mean, variance, mean_cur,
                                                                         var_cur, skip_if);
  B200_LAUNCHED();
  return 0;
}

int dropout_apply(b200_ctx *ctx, const float *in, const uint8_t *mask, float scale, float *out, size_t n) {
  if (n == 0) return 0;
  dropout_kernel<<<elementwise_grid(n, ctx->sm_count), 256, 0, ctx->stream>>>(in, mask, scale, out, n);
  B200_LAUNCHED();
  return 0;
}

int lrn_across_fwd(b200_ctx *ctx, const float *in, float *out, int channels, int area, int size, float alpha,
                   float beta, int B) {
  const long long total = (long long)B * area;
  if (total == 0) return 0;
  lrn_across_fwd_kernel<<<elementwise_grid((size_t)total, ctx->sm_count), 256, 0, ctx->stream>>>(
    in, out, channels, area, size, alpha / (float)size, beta, total);
  B200_LAUNCHED();
  return 0;
}

}  // namespace b200
