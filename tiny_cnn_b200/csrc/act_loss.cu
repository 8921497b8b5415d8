// Activations (relu, tanh, softmax) forward/backward and the loss gradients
// that sit between the contraction kernels on the training step.
#include <float.h>

#include <algorithm>

#include "common.cuh"
#include "device_utils.cuh"

namespace b200 {

// relu_layer.h:25-29, tanh_layer.h:24-28 -- elementwise, float4 where aligned
__global__ void act_fwd_kernel(int kind, float param, const float *__restrict__ x, float *__restrict__ y,
                               size_t n4, size_t n) {
  after_previous_kernel();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t step = (size_t)gridDim.x * blockDim.x;
  const float4 *x4 = reinterpret_cast<const float4 *>(x);
  float4 *y4 = reinterpret_cast<float4 *>(y);
  for (size_t j = i; j < n4; j += step) {
    float4 v = x4[j];
    v.x = apply_act_p(v.x, kind, param);
    v.y = apply_act_p(v.y, kind, param);
    v.z = apply_act_p(v.z, kind, param);
    v.w = apply_act_p(v.w, kind, param);
    y4[j] = v;
  }
  for (size_t j = n4 * 4 + i; j < n; j += step) y[j] = apply_act_p(x[j], kind, param);
}

__global__ void act_bwd_kernel(int kind, float param, const float *__restrict__ y, const float *__restrict__ dy,
                               float *__restrict__ dx, size_t n4, size_t n) {
  after_previous_kernel();
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t step = (size_t)gridDim.x * blockDim.x;
  const float4 *y4 = reinterpret_cast<const float4 *>(y);
  const float4 *d4 = reinterpret_cast<const float4 *>(dy);
  float4 *o4 = reinterpret_cast<float4 *>(dx);
  for (size_t j = i; j < n4; j += step) {
    float4 a = y4[j], g = d4[j], o;
    o.x = act_grad(kind, param, a.x, g.x);
    o.y = act_grad(kind, param, a.y, g.y);
    o.z = act_grad(kind, param, a.z, g.z);
    o.w = act_grad(kind, param, a.w, g.w);
    o4[j] = o;
  }
  for (size_t j = n4 * 4 + i; j < n; j += step) dx[j] = act_grad(kind, param, y[j], dy[j]);
}

// softmax_layer.h:24-34: subtract the row max, exponentiate, divide by the sum
// accumulated in index order.  One thread per row (rows are 10 wide here); rows of at most
// SM_REG values are kept in registers between the passes.
constexpr int SM_REG = 16;

__global__ void softmax_fwd_kernel(const float *__restrict__ x, float *__restrict__ y, int dim,
                                   int B) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= B) return;
  const float *xr = x + (size_t)n * dim;
  float *yr = y + (size_t)n * dim;
  if (dim <= SM_REG) {
    float v[SM_REG];
#pragma unroll
    for (int j = 0; j < SM_REG; ++j) v[j] = j < dim ? xr[j] : 0.f;
    float alpha = v[0];
#pragma unroll
    for (int j = 1; j < SM_REG; ++j)
      if (j < dim) alpha = fmaxf(alpha, v[j]);
    float denom = 0.f;
#pragma unroll
    for (int j = 0; j < SM_REG; ++j)
      if (j < dim) {
        v[j] = expf(v[j] - alpha);
        denom += v[j];
      }
#pragma unroll
    for (int j = 0; j < SM_REG; ++j)
      if (j < dim) yr[j] = v[j] / denom;
    return;
  }
  float alpha = xr[0];
  for (int j = 1; j < dim; ++j) alpha = fmaxf(alpha, xr[j]);
  float denom = 0.f;
  for (int j = 0; j < dim; ++j) {
    float e = expf(xr[j] - alpha);
    yr[j] = e;
    denom += e;
  }
  for (int j = 0; j < dim; ++j) yr[j] = yr[j] / denom;
}

// Rows of at most 16 values, sixteen lanes per row: lane j exponentiates x_j, every lane adds the
// exponentials in index order (fetched from their lanes), so the result has the bits of the
// one-thread form above.
__global__ void __launch_bounds__(256) softmax_fwd16_kernel(const float *__restrict__ x, float *__restrict__ y, int dim,
                                                            int B) {
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, j = threadIdx.x & 15;
  const int base = threadIdx.x & 16;
  const bool live = n < B && j < dim;
  const float xj = live ? x[(size_t)n * dim + j] : 0.f;
  float alpha = __shfl_sync(0xffffffffu, xj, base);
  for (int k = 1; k < dim; ++k) alpha = fmaxf(alpha, __shfl_sync(0xffffffffu, xj, base + k));
  const float ej = expf(xj - alpha);
  float denom = 0.f;
  for (int k = 0; k < dim; ++k) denom += __shfl_sync(0xffffffffu, ej, base + k);
  if (live) y[(size_t)n * dim + j] = ej / denom;
}

// softmax_layer.h:36-55: dx_j = sum_k dy_k * (k == j ? y_j(1-y_j) : -y_k*y_j)
// With `t` != nullptr the incoming gradient is first computed as the loss gradient of (y, t)
// (loss_function.h) and stored to dy: the loss-gradient and softmax-gradient kernels in one.
// The same for rows of at most 16 values with sixteen lanes per row: lane j computes dx_j, fetching y_k
// and the incoming gradient g_k from lane k; the sum over k runs in index order as in the one-thread
// form below, so both give the same bits.
__global__ void __launch_bounds__(256) softmax_bwd16_kernel(const float *__restrict__ y, float *__restrict__ dy,
                                                            float *__restrict__ dx, int dim, int B,
                                                            const float *__restrict__ t, int loss_kind) {
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, j = threadIdx.x & 15;
  const int base = threadIdx.x & 16;  // first lane of this row's group inside the warp
  const bool live = n < B && j < dim;
  const float factor = 2.0f / (float)dim;
  float yj = 0.f, gj = 0.f;
  if (live) {
    yj = y[(size_t)n * dim + j];
    if (t != nullptr) {
      gj = loss_grad_one(loss_kind, yj, t[(size_t)n * dim + j], factor);
      dy[(size_t)n * dim + j] = gj;
    } else {
      gj = dy[(size_t)n * dim + j];
    }
  }
  float s = 0.f;
  for (int k = 0; k < dim; ++k) {
    const float yk = __shfl_sync(0xffffffffu, yj, base + k);
    const float gk = __shfl_sync(0xffffffffu, gj, base + k);
    const float df = (k == j) ? __fmul_rn(yj, __fsub_rn(1.f, yj)) : __fmul_rn(-yk, yj);
    s = __fadd_rn(s, __fmul_rn(gk, df));
  }
  if (live) dx[(size_t)n * dim + j] = s;
}

__global__ void softmax_bwd_kernel(const float *__restrict__ y, float *__restrict__ dy,
                                   float *__restrict__ dx, int dim, int B, const float *__restrict__ t,
                                   int loss_kind) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= B) return;
  const float *yr = y + (size_t)n * dim;
  float *gr = dy + (size_t)n * dim;
  float *dr = dx + (size_t)n * dim;
  const float factor = 2.0f / (float)dim;
  if (dim <= SM_REG) {
    float yv[SM_REG], gv[SM_REG];
#pragma unroll
    for (int j = 0; j < SM_REG; ++j) {
      yv[j] = j < dim ? yr[j] : 0.f;
      if (t != nullptr) {
        gv[j] = j < dim ? loss_grad_one(loss_kind, yv[j], t[(size_t)n * dim + j], factor) : 0.f;
        if (j < dim) gr[j] = gv[j];
      } else {
        gv[j] = j < dim ? gr[j] : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < SM_REG; ++j) {
      if (j < dim) {
        const float yj = yv[j];
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < SM_REG; ++k)
          if (k < dim) {
            float df = (k == j) ? __fmul_rn(yj, __fsub_rn(1.f, yj)) : __fmul_rn(-yv[k], yj);
            s = __fadd_rn(s, __fmul_rn(gv[k], df));
          }
        dr[j] = s;
      }
    }
    return;
  }
  if (t != nullptr)
    for (int j = 0; j < dim; ++j) gr[j] = loss_grad_one(loss_kind, yr[j], t[(size_t)n * dim + j], factor);
  for (int j = 0; j < dim; ++j) {
    float yj = yr[j];
    float s = 0.f;
    for (int k = 0; k < dim; ++k) {
      float df = (k == j) ? __fmul_rn(yj, __fsub_rn(1.f, yj)) : __fmul_rn(-yr[k], yj);
      s = __fadd_rn(s, __fmul_rn(gr[k], df));
    }
    dr[j] = s;
  }
}

// loss_function.h:28-36 (mse), :120-128 (cross_entropy), :143-150 (multiclass)
__global__ void loss_grad_kernel(int kind, const float *__restrict__ y, const float *__restrict__ t,
                                 float *__restrict__ dy, int dim, size_t n) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t step = (size_t)gridDim.x * blockDim.x;
  const float factor = 2.0f / (float)dim;
  for (; i < n; i += step) {
    dy[i] = loss_grad_one(kind, y[i], t[i], factor);
  }
}

// sum over the batch of E::f (loss_function.h:17-26, :107-118, :132-141)
__global__ void loss_value_kernel(int kind, const float *__restrict__ y, const float *__restrict__ t,
                                  float *__restrict__ out, int dim, int B) {
  float acc = 0.f;
  for (int n = threadIdx.x; n < B; n += blockDim.x) {
    const float *yr = y + (size_t)n * dim;
    const float *tr = t + (size_t)n * dim;
    float d = 0.f;
    for (int j = 0; j < dim; ++j) {
      float yi = yr[j], ti = tr[j];
      if (kind == B200_LOSS_MSE)
        d += (yi - ti) * (yi - ti);
      else if (kind == B200_LOSS_CROSS_ENTROPY)
        d += -ti * logf(yi) - (1.f - ti) * logf(1.f - yi);
      else
        d += -ti * logf(yi);
    }
    if (kind == B200_LOSS_MSE) d /= (float)dim;
    acc += d;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) *out = acc;
}

static int grid_for(size_t total, int block, int sm_count) {
  size_t blocks = (total + block - 1) / block;
  size_t cap = (size_t)sm_count * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int act_fwd(b200_ctx *ctx, int kind, const float *x, float *y, int dim, int B, float param) {
  B200_REQUIRE(kind >= B200_ACT_NONE && kind <= B200_ACT_ELU, "act_fwd: unknown activation %d", kind);
  size_t n = (size_t)dim * B;
  if (n == 0) return 0;
  if (kind == B200_ACT_SOFTMAX) {
    if (dim <= 16)
      softmax_fwd16_kernel<<<ceil_div(B * 16, 256), 256, 0, ctx->stream>>>(x, y, dim, B);
    else
      softmax_fwd_kernel<<<ceil_div(B, 32), 32, 0, ctx->stream>>>(x, y, dim, B);
    B200_LAUNCHED();
    return 0;
  }
  size_t n4 = (aligned16(x) && aligned16(y)) ? n / 4 : 0;
  return launch_kernel(ctx, act_fwd_kernel, dim3(grid_for(n4 ? n4 : n, 256, ctx->sm_count)), dim3(256), 0, 1, kind, param, x, y,
                       n4, n);
}

int act_bwd(b200_ctx *ctx, int kind, const float *y, const float *dy, float *dx, int dim, int B, float param) {
  B200_REQUIRE(kind >= B200_ACT_NONE && kind <= B200_ACT_ELU, "act_bwd: unknown activation %d", kind);
  size_t n = (size_t)dim * B;
  if (n == 0) return 0;
  if (kind == B200_ACT_SOFTMAX) {
    if (dim <= 16)
      softmax_bwd16_kernel<<<ceil_div(B * 16, 256), 256, 0, ctx->stream>>>(y, const_cast<float *>(dy), dx, dim, B,
                                                                           nullptr, 0);
    else
      softmax_bwd_kernel<<<ceil_div(B, 32), 32, 0, ctx->stream>>>(y, const_cast<float *>(dy), dx, dim, B, nullptr, 0);
    B200_LAUNCHED();
    return 0;
  }
  size_t n4 = (aligned16(y) && aligned16(dy) && aligned16(dx)) ? n / 4 : 0;
  return launch_kernel(ctx, act_bwd_kernel, dim3(grid_for(n4 ? n4 : n, 256, ctx->sm_count)), dim3(256), 0, 1, kind, param, y, dy,
                       dx, n4, n);
}

int loss_grad(b200_ctx *ctx, int kind, const float *y, const float *t, float *dy, int dim, int B) {
  B200_REQUIRE(kind >= B200_LOSS_MSE && kind <= B200_LOSS_CROSS_ENTROPY_MULTICLASS,
               "loss_grad: unknown loss %d", kind);
  size_t n = (size_t)dim * B;
  if (n == 0) return 0;
  loss_grad_kernel<<<grid_for(n, 256, ctx->sm_count), 256, 0, ctx->stream>>>(kind, y, t, dy, dim,
                                                                             n);
  B200_LAUNCHED();
  return 0;
}

// loss gradient of (y, t) into dy, then the softmax gradient into dx: one launch
int softmax_loss_bwd(b200_ctx *ctx, int loss_kind, const float *y, const float *t, float *dy, float *dx, int dim,
                     int B) {
  B200_REQUIRE(loss_kind >= B200_LOSS_MSE && loss_kind <= B200_LOSS_CROSS_ENTROPY_MULTICLASS,
               "softmax_loss_bwd: unknown loss %d", loss_kind);
  if ((size_t)dim * B == 0) return 0;
  if (dim <= 16)
    softmax_bwd16_kernel<<<ceil_div(B * 16, 256), 256, 0, ctx->stream>>>(y, dy, dx, dim, B, t, loss_kind);
  else
    softmax_bwd_kernel<<<ceil_div(B, 32), 32, 0, ctx->stream>>>(y, dy, dx, dim, B, t, loss_kind);
  B200_LAUNCHED();
  return 0;
}

// ---- a narrow fully-connected layer followed by a softmax output layer ---------------------
// (the classifier's last two layers: 64 -> 10 in the CIFAR-10 net).  A warp per sample, the inputs dealt to its lanes;
// the weights (K x N floats, N <= 16) sit in shared memory.  With sixteen lanes a sample, each adding all the products
// of an output, the chain of K additions was the kernel's time (500 -> 10, 77 samples: 20 us forward, 16 us backward;
// now 3.4 and 2.8 us with the wide forms below).
constexpr int FCS_N = 16, FCS_THREADS = 256;
constexpr int FCS_NARROW = 256;               // inputs up to which a sample is a warp's work
constexpr int FCS_WIDE = 1024;                // inputs up to which four samples are a block's work (forward)
constexpr int FCW_THREADS = 512, FCW_WARPS = FCW_THREADS / 32, FCW_SAMPLES = 4;
constexpr int FCL_THREADS = 256, FCL_WARPS = FCL_THREADS / 32;
constexpr int FCL_GROUP = 4, FCL_SAMPLES = FCL_WARPS * FCL_GROUP;  // forward: samples of a warp, of a block
constexpr int FCL_CHUNK = 128;                                     // forward: rows of weights in shared memory, twice
constexpr int FCL_BWD = 16;                                        // backward: most samples of a block

// the sum of acc[j] over the lanes, in lane j of each half-warp: sums of halves, which leave half the values a step
__device__ __forceinline__ float lanes_sum16(float *acc) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 8; h > 0; h >>= 1)
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const bool up = lane & h;
      const float keep = up ? acc[j + h] : acc[j], give = up ? acc[j] : acc[j + h];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, h);
    }
  return acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 16);
}

// by a warp: lane j < N holds the products' sum of output j of sample n; z = sum + bias, y = softmax(z)
__device__ __forceinline__ void head_out(float sum, const float *bias, float *z, float *y, int n, int N) {
  const int lane = threadIdx.x & 31, j = lane & 15;
  const float zj = (bias != nullptr && j < N) ? sum + bias[j] : sum;
  if (lane < N) z[(size_t)n * N + j] = zj;
  float alpha = __shfl_sync(0xffffffffu, zj, 0);
  for (int k = 1; k < N; ++k) alpha = fmaxf(alpha, __shfl_sync(0xffffffffu, zj, k));
  const float ej = expf(zj - alpha);
  float denom = 0.f;
  for (int k = 0; k < N; ++k) denom += __shfl_sync(0xffffffffu, ej, k);
  if (lane < N) y[(size_t)n * N + j] = ej / denom;
}

// by a warp: the loss gradient of sample n to dy and the softmax gradient to dz, returned in lane j of each half-warp
__device__ __forceinline__ float head_grad(const float *y, const float *t, int loss_kind, float *dy, float *dz, int n, int N) {
  const int lane = threadIdx.x & 31, j = lane & 15;
  const float factor = 2.0f / (float)N;
  float yj = 0.f, gj = 0.f;
  if (j < N) {
    yj = y[(size_t)n * N + j];
    gj = loss_grad_one(loss_kind, yj, t[(size_t)n * N + j], factor);
    if (dy != nullptr && lane < N) dy[(size_t)n * N + j] = gj;
  }
  float s = 0.f;
  for (int k = 0; k < N; ++k) {
    const float yk = __shfl_sync(0xffffffffu, yj, k);
    const float gk = __shfl_sync(0xffffffffu, gj, k);
    const float df = (k == j) ? __fmul_rn(yj, __fsub_rn(1.f, yj)) : __fmul_rn(-yk, yj);
    s = __fadd_rn(s, __fmul_rn(gk, df));
  }
  if (dz != nullptr && lane < N) dz[(size_t)n * N + j] = s;
  return s;
}

// z = x W + b (fully_connected_op_internal.h:15-36), y = softmax(z) (softmax_layer.h:24-34)
__global__ void __launch_bounds__(FCS_THREADS) fc_softmax_fwd16_kernel(const float *__restrict__ x,
                                                                       const float *__restrict__ W,
                                                                       const float *__restrict__ bias,
                                                                       float *__restrict__ z, float *__restrict__ y,
                                                                       int K, int N, int B) {
  after_previous_kernel();
  extern __shared__ float fcs_w[];  // [K][N]
  for (int i = threadIdx.x; i < K * N; i += FCS_THREADS) cp_async4(fcs_w + i, W + i, true);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int n = (blockIdx.x * FCS_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (n >= B) return;
  const float *xr = x + (size_t)n * K;
  float acc[FCS_N];
#pragma unroll
  for (int i = 0; i < FCS_N; ++i) acc[i] = 0.f;
#pragma unroll 8
  for (int k = lane; k < K; k += 32) {
    const float xk = xr[k];
    const float *w = fcs_w + k * N;
#pragma unroll
    for (int i = 0; i < FCS_N; ++i)
      if (i < N) acc[i] = fmaf(xk, w[i], acc[i]);
  }
  head_out(lanes_sum16(acc), bias, z, y, n, N);
}

// dy = loss gradient of (y, t); dz = softmax gradient (as softmax_bwd16_kernel); dx = dz W^T
// (fully_connected_op_internal.h:45-50), multiplied by the gradient of a relu in front of the layer when
// `relu_x` (that relu's output = this layer's input) is given (relu_layer.h:31-39)
__global__ void __launch_bounds__(FCS_THREADS) fc_softmax_bwd16_kernel(const float *__restrict__ y,
                                                                       const float *__restrict__ t, int loss_kind,
                                                                       const float *__restrict__ W,
                                                                       const float *__restrict__ relu_x,
                                                                       float *__restrict__ dy, float *__restrict__ dz,
                                                                       float *__restrict__ dx, int K, int N, int B) {
  after_previous_kernel();
  extern __shared__ float fcs_w[];  // [K][N]
  for (int i = threadIdx.x; i < K * N; i += FCS_THREADS) cp_async4(fcs_w + i, W + i, true);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int n = (blockIdx.x * FCS_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (n >= B) return;
  const float s = head_grad(y, t, loss_kind, dy, dz, n, N);
  if (dx == nullptr) return;
  float d[FCS_N];
#pragma unroll
  for (int i = 0; i < FCS_N; ++i) d[i] = __shfl_sync(0xffffffffu, s, i);
#pragma unroll 8
  for (int c = lane; c < K; c += 32) {  // dx_c = sum_i dz_i W[c][i]
    const float *w = fcs_w + c * N;
    float a = 0.f;
#pragma unroll
    for (int i = 0; i < FCS_N; ++i)
      if (i < N) a = fmaf(d[i], w[i], a);
    if (relu_x != nullptr && !(relu_x[(size_t)n * K + c] > 0.f)) a = 0.f;
    dx[(size_t)n * K + c] = a;
  }
}

// The same for longer inputs: a block takes four samples, its threads deal the inputs out, and a row of weights is read
// once for the four of them.
__global__ void __launch_bounds__(FCW_THREADS) fc_softmax_fwd_wide_kernel(const float *__restrict__ x,
                                                                          const float *__restrict__ W,
                                                                          const float *__restrict__ bias, float *__restrict__ z,
                                                                          float *__restrict__ y, int K, int N, int B) {
  after_previous_kernel();
  __shared__ float sums[FCW_SAMPLES][FCW_WARPS][FCS_N];
  const int n0 = blockIdx.x * FCW_SAMPLES, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float acc[FCW_SAMPLES][FCS_N];
#pragma unroll
  for (int s = 0; s < FCW_SAMPLES; ++s)
#pragma unroll
    for (int i = 0; i < FCS_N; ++i) acc[s][i] = 0.f;
#pragma unroll 2
  for (int k = threadIdx.x; k < K; k += FCW_THREADS) {
    float xk[FCW_SAMPLES];
#pragma unroll
    for (int s = 0; s < FCW_SAMPLES; ++s) xk[s] = x[(size_t)min(n0 + s, B - 1) * K + k];
#pragma unroll
    for (int i = 0; i < FCS_N; ++i)
      if (i < N) {
        const float w = W[(size_t)k * N + i];
#pragma unroll
        for (int s = 0; s < FCW_SAMPLES; ++s) acc[s][i] = fmaf(xk[s], w, acc[s][i]);
      }
  }
#pragma unroll
  for (int s = 0; s < FCW_SAMPLES; ++s) {
    const float v = lanes_sum16(acc[s]);
    if (lane < FCS_N) sums[s][warp][lane] = v;
  }
  __syncthreads();
  const int n = n0 + warp;
  if (warp >= FCW_SAMPLES || n >= B) return;
  float sum = 0.f;
  for (int w = 0; w < FCW_WARPS; ++w) sum += sums[warp][w][lane & 15];
  head_out(sum, bias, z, y, n, N);
}

// The longest inputs: the blocks of a cluster share the inputs of 32 samples out and add their sums over distributed shared memory.
// A block's rows of weights lie in shared memory, at an odd pitch, for all its samples, and a value read from there serves four
// of them.  NP is N rounded up to a multiple of four: a test of every output would put each product behind the one before.
// (4096 -> 10: with 1024 samples 21.5 us with the kernel above, which the strided reads of the weights hold up, ten lines of the L1
// cache a load, 9.9 with this one; with 8 samples 12.5 and 7.2.  500 -> 10, 77 samples: 3.4 and 4.5, the cluster's barriers.)
template <int NP>
__global__ void __launch_bounds__(FCL_THREADS) fc_softmax_fwd_cluster_kernel(const float *__restrict__ x,
                                                                          const float *__restrict__ W,
                                                                          const float *__restrict__ bias, float *__restrict__ z,
                                                                          float *__restrict__ y, int K, int per, int N, int B) {
  after_previous_kernel();
  __shared__ float rows[2][FCL_CHUNK * (NP + 1)];
  __shared__ float sums[FCL_SAMPLES][FCS_N];
  const int blocks = gridDim.y, rank = blockIdx.y, n0 = blockIdx.x * FCL_SAMPLES, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int pitch = NP + 1;
  const int first = n0 + warp * FCL_GROUP, end = min(K, (rank + 1) * per);
  float acc[FCL_GROUP][FCS_N];
#pragma unroll
  for (int s = 0; s < FCL_GROUP; ++s)
#pragma unroll
    for (int i = 0; i < FCS_N; ++i) acc[s][i] = 0.f;
  constexpr int XK = FCL_CHUNK / 32;
  float next[FCL_GROUP][XK];  // a chunk's values and rows are on their way while the one before is multiplied
  auto fetch = [&](int k0, float *to) {
#pragma unroll
    for (int i = threadIdx.x; i < FCL_CHUNK * NP; i += FCL_THREADS) {
      const int r = i / NP, o = i - r * NP;
      const bool ok = k0 + r < end && o < N;
      cp_async4(to + r * pitch + o, W + (ok ? (size_t)(k0 + r) * N + o : 0), ok);
    }
    cp_async_commit();
#pragma unroll
    for (int s = 0; s < FCL_GROUP; ++s)
#pragma unroll
      for (int j = 0; j < XK; ++j) {
        const int k = k0 + lane + 32 * j;
        next[s][j] = first + s < B && k < end ? x[(size_t)(first + s) * K + k] : 0.f;
      }
  };
  int buf = 0;
  if (rank * per < end) fetch(rank * per, rows[0]);  // the last blocks' shares may be empty: no copy that nobody waits for
  for (int k0 = rank * per; k0 < end; k0 += FCL_CHUNK, buf ^= 1) {
    float xk[FCL_GROUP][XK];
#pragma unroll
    for (int s = 0; s < FCL_GROUP; ++s)
#pragma unroll
      for (int j = 0; j < XK; ++j) xk[s][j] = next[s][j];
    cp_async_wait<0>();
    __syncthreads();
    if (k0 + FCL_CHUNK < end) fetch(k0 + FCL_CHUNK, rows[buf ^ 1]);
    if (first < B) {
#pragma unroll
      for (int j = 0; j < XK; ++j)
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          const float w = rows[buf][(lane + 32 * j) * pitch + i];
#pragma unroll
          for (int s = 0; s < FCL_GROUP; ++s) acc[s][i] = fmaf(xk[s][j], w, acc[s][i]);
        }
    }
  }
#pragma unroll
  for (int s = 0; s < FCL_GROUP; ++s) {
    const float v = lanes_sum16(acc[s]);
    if (lane < FCS_N) sums[warp * FCL_GROUP + s][lane] = v;
  }
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
  for (int s = rank + blocks * warp; s < FCL_SAMPLES && n0 + s < B; s += blocks * FCL_WARPS) {  // a warp a sample
    float sum = 0.f;
    const unsigned at = smem_u32(&sums[s][lane & 15]);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if (b == blocks) break;
      float v;
      unsigned remote;
      asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(at), "r"(b));
      asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(remote) : "memory");
      sum += v;
    }
    head_out(sum, bias, z, y, n0 + s, N);
  }
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}

// Backward a thread keeps the weights of one input in registers for up to 16 samples.  (4096 -> 10, 1024 samples: 19.5 us with a row of
// weights read again for every four, from the L1 cache as above, now 12.5, of which writing dX and reading what the relu gave
// take 5; 8 samples: 9.7 us with all inputs in one block, now 2.9.)
template <int NP>
__global__ void __launch_bounds__(FCL_THREADS) fc_softmax_bwd_wide_kernel(const float *__restrict__ y,
                                                                          const float *__restrict__ t, int loss_kind,
                                                                          const float *__restrict__ W,
                                                                          const float *__restrict__ relu_x,
                                                                          float *__restrict__ dy, float *__restrict__ dz,
                                                                          float *__restrict__ dx, int K, int N, int B, int per) {
  after_previous_kernel();
  __shared__ __align__(16) float ds[FCL_BWD][FCS_N];
  const int n0 = blockIdx.x * per, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, samples = min(per, B - n0);
  int c = blockIdx.y * FCL_THREADS + threadIdx.x;
  const bool writes = blockIdx.y == 0, gated = relu_x != nullptr && dx != nullptr;
  float w[NP], gate[4];
  auto weights = [&]() {
#pragma unroll
    for (int i = 0; i < NP; ++i) w[i] = c < K && i < N ? W[(size_t)c * N + i] : 0.f;
  };
  auto gates = [&](int s0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) gate[e] = !gated ? 1.f : c < K && s0 + e < samples ? relu_x[(size_t)(n0 + s0 + e) * K + c] : 0.f;
  };
  if (dx != nullptr) weights();
  gates(0);
  for (int s = warp; s < samples; s += FCL_WARPS) {
    const float g = head_grad(y, t, loss_kind, writes ? dy : nullptr, writes ? dz : nullptr, n0 + s, N);
    if (lane < FCS_N) ds[s][lane] = lane < N ? g : 0.f;  // behind N an infinite gradient leaves no zero
  }
  __syncthreads();
  if (dx == nullptr) return;
  while (c < K) {
    for (int s0 = 0; s0 < samples; s0 += 4) {  // dx_c = sum_i dz_i W[c][i]
      float a[4], now[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = 0.f, now[e] = gate[e];
      if (s0 + 4 < samples) gates(s0 + 4);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < NP; ++i) a[e] = fmaf(ds[s0 + e][i], w[i], a[e]);  // behind N both are zero
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (s0 + e < samples) dx[(size_t)(n0 + s0 + e) * K + c] = now[e] > 0.f ? a[e] : 0.f;
    }
    c += gridDim.y * FCL_THREADS;
    weights();
    gates(0);
  }
}

bool fc_softmax_fusable(int K, int N) { return N >= 1 && N <= FCS_N && K >= 1; }

int fc_softmax_fwd(b200_ctx *ctx, int K, int N, const float *x, const float *W, const float *bias, float *z, float *y,
                   int B) {
  B200_REQUIRE(fc_softmax_fusable(K, N), "fc_softmax_fwd: shape %d x %d not supported", K, N);
  if (B == 0) return 0;
  if (K <= FCS_NARROW)
    B200_TRY(launch_kernel(ctx, fc_softmax_fwd16_kernel, dim3(ceil_div(B, FCS_THREADS / 32)), dim3(FCS_THREADS),
                           (size_t)K * N * sizeof(float), 1, x, W, bias, z, y, K, N, B));
  else if (K <= FCS_WIDE)
    B200_TRY(launch_kernel(ctx, fc_softmax_fwd_wide_kernel, dim3(ceil_div(B, FCW_SAMPLES)), dim3(FCW_THREADS), 0, 1, x, W,
                           bias, z, y, K, N, B));
  else {
    const int blocks = 8, per = ceil_div(ceil_div(K, blocks), 32) * 32;
    auto kernel = N <= 4   ? fc_softmax_fwd_cluster_kernel<4>
                  : N <= 8 ? fc_softmax_fwd_cluster_kernel<8>
                  : N <= 12 ? fc_softmax_fwd_cluster_kernel<12> : fc_softmax_fwd_cluster_kernel<16>;
    B200_TRY(launch_kernel(ctx, kernel, dim3(ceil_div(B, FCL_SAMPLES), blocks), dim3(FCL_THREADS), 0, dim3(1, blocks), x, W, bias, z, y,
                           K, per, N, B));
  }
  return 0;
}

int fc_softmax_loss_bwd(b200_ctx *ctx, int loss_kind, int K, int N, const float *y, const float *t, const float *W,
                        const float *relu_x, float *dy, float *dz, float *dx, int B) {
  B200_REQUIRE(fc_softmax_fusable(K, N), "fc_softmax_loss_bwd: shape %d x %d not supported", K, N);
  B200_REQUIRE(loss_kind >= B200_LOSS_MSE && loss_kind <= B200_LOSS_CROSS_ENTROPY_MULTICLASS,
               "fc_softmax_loss_bwd: unknown loss %d", loss_kind);
  if (B == 0) return 0;
  if (K <= FCS_NARROW)
    B200_TRY(launch_kernel(ctx, fc_softmax_bwd16_kernel, dim3(ceil_div(B, FCS_THREADS / 32)), dim3(FCS_THREADS),
                           (size_t)K * N * sizeof(float), 1, y, t, loss_kind, W, relu_x, dy, dz, dx, K, N, B));
  else {
    auto kernel = N <= 4   ? fc_softmax_bwd_wide_kernel<4>
                  : N <= 8 ? fc_softmax_bwd_wide_kernel<8>
                  : N <= 12 ? fc_softmax_bwd_wide_kernel<12> : fc_softmax_bwd_wide_kernel<16>;
    const int across = dx ? std::min(ceil_div(K, FCL_THREADS), 65535) : 1;
    // four samples a block, whose loads then are all on their way at once, until they fill the chip
    const int per = (long long)ceil_div(B, 4) * across <= 4LL * ctx->sm_count ? 4 : FCL_BWD;
    B200_TRY(launch_kernel(ctx, kernel, dim3(ceil_div(B, per), across), dim3(FCL_THREADS), 0, 1, y, t, loss_kind, W, relu_x, dy, dz,
                           dx, K, N, B, per));
  }
  return 0;
}

int loss_value(b200_ctx *ctx, int kind, const float *y, const float *t, float *loss_sum, int dim,
               int B) {
  B200_REQUIRE(kind >= B200_LOSS_MSE && kind <= B200_LOSS_CROSS_ENTROPY_MULTICLASS,
               "loss_value: unknown loss %d", kind);
  loss_value_kernel<<<1, 256, 0, ctx->stream>>>(kind, y, t, loss_sum, dim, B);
  B200_LAUNCHED();
  return 0;
}

}  // namespace b200
