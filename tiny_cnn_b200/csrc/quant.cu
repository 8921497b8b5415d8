// uint8 quantized convolution and fully-connected forward, bit-exact with the
// reference's per-sample pipeline
//   tiny_quantized_conv2d_kernel          (core/kernels/tiny_quantized_conv2d_kernel.h:20-148)
//   tiny_quantized_fully_connected_kernel (core/kernels/tiny_quantized_fully_connected_kernel.h:22-128)
// built on the scalar helpers of core/kernels/tiny_quantization_kernel.h.
//
// Every float / double expression below is written with explicit
// round-to-nearest intrinsics in the operand order of the reference so that no
// multiply-add contraction or reassociation can change a bit; this file is also
// compiled with -fmad=false.
//
// Pipeline (all samples of the batch at once):
//   1. per-sample min/max of the input            (conv :27-36, fc :30-35)
//   2. min/max of the filter subset the reference scans, and of the bias
//      (conv :40-71, fc :38-67) -- sample independent, done once
//   3. quantize input, filter, bias to uint8      (float_to_quantized, :59-68)
//   4. per-sample output range, offsets, zero point (conv :73-87, fc :49-81)
//   5. int32 accumulate of (w - off_w)*(x - off_x) + (bias_q - zero)
//   6. per-sample min/max of the accumulators, shrink range, fixed-point
//      requantize to uint8, dequantize to float   (:140-147; kernel.h:145-186,230-254)
#include <limits.h>

#include "common.cuh"
#include "device_utils.cuh"

namespace b200 {

// ---- scalar helpers (tiny_quantization_kernel.h) ---------------------------

// float_to_quantized_unclamped<T> (:32-49); BITS = 8 (uint8, lowest 0) or 32
// (int32, lowest -2^31)
template <int BITS>
__device__ __forceinline__ long long f2q_unclamped(float input, float rmin, float rmax) {
  if (rmin == rmax) return 0;
  const long long steps = 1LL << BITS;
  const double range_adjust = __ddiv_rn((double)steps, __dsub_rn((double)steps, 1.0));
  const double range = __dmul_rn((double)__fsub_rn(rmax, rmin), range_adjust);
  const double range_scale = __ddiv_rn((double)steps, range);
  long long q = (long long)__dsub_rn(round(__dmul_rn((double)input, range_scale)),
                                     round(__dmul_rn((double)rmin, range_scale)));
  const long long lowest = BITS == 8 ? 0LL : -(1LL << 31);
  return q + lowest;
}

// float_to_quantized<T> (:59-68)
template <int BITS>
__device__ __forceinline__ long long f2q(float input, float rmin, float rmax) {
  long long q = f2q_unclamped<BITS>(input, rmin, rmax);
  const long long lowest = BITS == 8 ? 0LL : -(1LL << 31);
  const long long highest = BITS == 8 ? 255LL : (1LL << 31) - 1;
  q = q > lowest ? q : lowest;
  q = q < highest ? q : highest;
  return q;
}

// quantized_to_float<T> (:70-84)
template <int BITS>
__device__ __forceinline__ float q2f(long long input, float rmin, float rmax) {
  if (rmin == rmax) return rmin;
  const long long steps = 1LL << BITS;
  const double range_adjust = __ddiv_rn((double)steps, __dsub_rn((double)steps, 1.0));
  const double range = __dmul_rn((double)__fsub_rn(rmax, rmin), range_adjust);
  const double range_scale = __ddiv_rn(range, (double)steps);
  const long long lowest = BITS == 8 ? 0LL : -(1LL << 31);
  const double offset_input = __dsub_rn((double)input, (double)lowest);
  const double result = __dadd_rn((double)rmin, __dmul_rn(offset_input, range_scale));
  return (float)result;
}

// float_for_one_quantized_level<uint8_t> (:86-93)
__device__ __forceinline__ float one_level_u8(float rmin, float rmax) {
  return __fdiv_rn(__fsub_rn(rmax, rmin), 255.0f);
}

struct QSample {
  float min_in, max_in;    // input range
  float min_out, max_out;  // int32 accumulator range
  int off_in;              // quantized 0.0 of the input
  int zero_total;          // quantized 0.0 of the accumulator space
  int acc_min, acc_max;    // observed accumulator extremes
  int sum_in;              // sum of the quantized input bytes (fully connected)
  // requantize_many_in_new_range<int32,uint8> constants (:159-171)
  long long range_scale_fp, input_offset_fp, output_offset_fp;
  float min_new, max_new;  // shrunk output range
};

struct QGlobal {
  float min_f, max_f;
  float min_b, max_b;
  int off_f;
};

// ---- 1. per-sample input range ----------------------------------------------

// One block per sample.  The scanned region is `nseg` segments of `seg_len`
// elements starting every `seg_stride` elements: the conv kernel scans
// in_padded.height^2 elements per channel plane (:29-35), the fc kernel scans
// the whole row.  Both seed the range with element 0.
__global__ void q_input_range_kernel(const float *__restrict__ in, size_t row_len, int nseg,
                                     size_t seg_stride, size_t seg_len, QSample *qs) {
  const float *r = in + (size_t)blockIdx.x * row_len;
  float mn = r[0], mx = r[0];
  for (int s = 0; s < nseg; ++s) {
    const float *seg = r + s * seg_stride;
    for (size_t e = threadIdx.x; e < seg_len; e += blockDim.x) {
      float v = seg[e];
      mn = fminf(mn, v);
      mx = fmaxf(mx, v);
    }
  }
  __shared__ float smn[32], smx[32];
  mn = warp_min(mn);
  mx = warp_max(mx);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    smn[wid] = mn;
    smx[wid] = mx;
  }
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    mn = lane < nw ? smn[lane] : smn[0];
    mx = lane < nw ? smx[lane] : smx[0];
    mn = warp_min(mn);
    mx = warp_max(mx);
    if (lane == 0) {
      qs[blockIdx.x].min_in = mn;
      qs[blockIdx.x].max_in = mx;
    }
  }
}

// ---- 2. filter / bias ranges ---------------------------------------------------

__device__ __forceinline__ void widen_ranges(float w0, float b0, int nbias, float *mn, float *mx, float *bmn, float *bmx) {
  if (*mn == *mx) {
    *mx = __fadd_rn(w0, 1e-3f);
    *mn = __fsub_rn(w0, 1e-3f);
  }
  if (nbias > 0 && *bmn == *bmx) {
    *bmx = __fadd_rn(b0, 1e-3f);
    *bmn = __fsub_rn(b0, 1e-3f);
  }
}

// By a whole block.  Filter: `nseg` segments of `seg_len` elements every
// `seg_stride`, seeded with W[0]; equal min/max widen to W[0] -+ 1e-3.
// Bias: all `nbias` elements, seeded with 0; equal min/max widen to b[0] -+ 1e-3.
// `qg` lies in shared memory; every thread may read it afterwards.
__device__ __forceinline__ void filter_range(const float *__restrict__ W, int nseg, size_t seg_stride, size_t seg_len,
                                             const float *__restrict__ bias, int nbias, QGlobal &qg) {
  float mn = W[0], mx = W[0];
  size_t total = (size_t)nseg * seg_len;
  for (size_t t = threadIdx.x; t < total; t += blockDim.x) {
    size_t s = nseg == 1 ? 0 : t / seg_len, e = t - s * seg_len;
    float v = W[s * seg_stride + e];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  float bmn = 0.f, bmx = 0.f;
  for (int t = threadIdx.x; t < nbias; t += blockDim.x) {
    bmn = fminf(bmn, bias[t]);
    bmx = fmaxf(bmx, bias[t]);
  }
  __shared__ float s4[4][32];
  mn = warp_min(mn);
  mx = warp_max(mx);
  bmn = warp_min(bmn);
  bmx = warp_max(bmx);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    s4[0][wid] = mn;
    s4[1][wid] = mx;
    s4[2][wid] = bmn;
    s4[3][wid] = bmx;
  }
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    mn = warp_min(lane < nw ? s4[0][lane] : s4[0][0]);
    mx = warp_max(lane < nw ? s4[1][lane] : s4[1][0]);
    bmn = warp_min(lane < nw ? s4[2][lane] : s4[2][0]);
    bmx = warp_max(lane < nw ? s4[3][lane] : s4[3][0]);
    if (lane == 0) {
      widen_ranges(W[0], nbias > 0 ? bias[0] : 0.f, nbias, &mn, &mx, &bmn, &bmx);
      qg.min_f = mn;
      qg.max_f = mx;
      qg.min_b = bmn;
      qg.max_b = bmx;
      qg.off_f = (int)f2q_unclamped<8>(0.0f, mn, mx);
    }
  }
  __syncthreads();
}

__global__ void q_filter_range_kernel(const float *__restrict__ W, int nseg, size_t seg_stride,
                                      size_t seg_len, const float *__restrict__ bias, int nbias,
                                      QGlobal *out) {
  __shared__ QGlobal qg;
  filter_range(W, nseg, seg_stride, seg_len, bias, nbias, qg);
  if (threadIdx.x == 0) *out = qg;
}

// ---- 3. quantize --------------------------------------------------------------

__global__ void q_quantize_filter_kernel(const float *__restrict__ W, size_t lenW,
                                         const float *__restrict__ bias, int nbias,
                                         const QGlobal *__restrict__ qg, uint8_t *__restrict__ Wq,
                                         uint8_t *__restrict__ bq) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  size_t step = (size_t)gridDim.x * blockDim.x;
  const float mn = qg->min_f, mx = qg->max_f;
  for (size_t j = i; j < lenW; j += step) Wq[j] = (uint8_t)f2q<8>(W[j], mn, mx);
  const float bmn = qg->min_b, bmx = qg->max_b;
  for (size_t j = i; j < (size_t)nbias; j += step) bq[j] = (uint8_t)f2q<8>(bias[j], bmn, bmx);
}

__global__ void q_quantize_input_kernel(const float *__restrict__ in, size_t row_len,
                                        const QSample *__restrict__ qs, uint8_t *__restrict__ inq) {
  const int n = blockIdx.y;
  const float mn = qs[n].min_in, mx = qs[n].max_in;
  const float *r = in + (size_t)n * row_len;
  uint8_t *q = inq + (size_t)n * row_len;
  size_t step = (size_t)gridDim.x * blockDim.x;
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < row_len; j += step)
    q[j] = (uint8_t)f2q<8>(r[j], mn, mx);
}

// ---- 4. per-sample output range and offsets -------------------------------------

// quantization_range_for_multiplication<u8,u8,i32> (:95-114); the fc kernel
// then adds the bias range to it (fc :67-68).
__device__ __forceinline__ void sample_params(QSample &s, const QGlobal &qg, int add_bias_range) {
  float a_level = one_level_u8(s.min_in, s.max_in);
  float b_level = one_level_u8(qg.min_f, qg.max_f);
  float c_level = __fmul_rn(a_level, b_level);
  float mn = __fmul_rn(c_level, (float)(-(1LL << 31)));
  float mx = __fmul_rn(c_level, (float)((1LL << 31) - 1));
  if (add_bias_range) {
    mn = __fadd_rn(mn, qg.min_b);
    mx = __fadd_rn(mx, qg.max_b);
  }
  s.min_out = mn;
  s.max_out = mx;
  s.off_in = (int)f2q_unclamped<8>(0.0f, s.min_in, s.max_in);
  s.zero_total = (int)f2q<32>(0.0f, mn, mx);
  s.acc_min = INT_MAX;
  s.acc_max = INT_MIN;
  s.sum_in = 0;
}

__global__ void q_sample_params_kernel(QSample *qs, const QGlobal *__restrict__ qg, int B,
                                       int add_bias_range) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= B) return;
  QSample s = qs[n];
  sample_params(s, *qg, add_bias_range);
  qs[n] = s;
}

// ---- 5. int32 accumulate ----------------------------------------------------------

__device__ __forceinline__ void block_minmax_atomic(int mn, int mx, int *gmin, int *gmax) {
  __shared__ int smn[32], smx[32];
  mn = warp_min_i(mn);
  mx = warp_max_i(mx);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    smn[wid] = mn;
    smx[wid] = mx;
  }
  __syncthreads();
  if (wid == 0) {
    int nw = (blockDim.x + 31) >> 5;
    mn = warp_min_i(lane < nw ? smn[lane] : INT_MAX);
    mx = warp_max_i(lane < nw ? smx[lane] : INT_MIN);
    if (lane == 0) {
      atomicMin(gmin, mn);
      atomicMax(gmax, mx);
    }
  }
}

// conv :89-133.  grid = (blocks per sample, B); one thread per output element.
// `bias_f` != nullptr: the nine-argument kernel's bias term, `bias[o] - zero_in_total_space` formed
// in FLOAT from the float-held bias entry and cast to int32 (tiny_quantized_conv2d_kernel.h:436-441)
__global__ void q_conv_acc_kernel(ConvGeom g, const uint8_t *__restrict__ inq,
                                  const uint8_t *__restrict__ Wq, const uint8_t *__restrict__ bq,
                                  const QGlobal *__restrict__ qg, QSample *qs,
                                  int *__restrict__ acc, const float *__restrict__ bias_f) {
  const int n = blockIdx.y;
  const int out_len = g.OC * g.OH * g.OW;
  const int in_len = g.C * g.HI * g.WI;
  const int off_f = qg->off_f;
  const int off_in = qs[n].off_in;
  const int zero_total = qs[n].zero_total;
  const uint8_t *ib = inq + (size_t)n * in_len;
  int mn = INT_MAX, mx = INT_MIN;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < out_len;
       idx += gridDim.x * blockDim.x) {
    int x = idx % g.OW;
    int r = idx / g.OW;
    int y = r % g.OH;
    int o = r / g.OH;
    int sum = 0;
    for (int inc = 0; inc < g.C; ++inc) {
      if (g.tbl && !g.tbl[inc * g.OC + o]) continue;
      const uint8_t *w = Wq + ((size_t)o * g.C + inc) * g.KH * g.KW;
      const uint8_t *ip = ib + ((size_t)inc * g.HI + y * g.SH) * g.WI + x * g.SW;
      for (int wy = 0; wy < g.KH; ++wy)
        for (int wx = 0; wx < g.KW; ++wx)
          sum += ((int)w[wy * g.KW + wx] - off_f) * ((int)ip[wy * g.WI + wx] - off_in);
    }
    if (g.has_bias)
      sum += bias_f != nullptr ? (int)__fsub_rn(bias_f[o], (float)zero_total) : (int)bq[o] - zero_total;
    acc[(size_t)n * out_len + idx] = sum;
    mn = min(mn, sum);
    mx = max(mx, sum);
  }
  block_minmax_atomic(mn, mx, &qs[n].acc_min, &qs[n].acc_max);
}

// ---- 6. shrink range, requantize, dequantize ---------------------------------------

// quantize_down_and_shrink_range (:230-254) and the constants of
// requantize_many_in_new_range<int32,uint8> (:159-171), once per sample.
__device__ __forceinline__ void requant_params(QSample &s) {
  float min_new = fminf(0.0f, q2f<32>((long long)s.acc_min, s.min_out, s.max_out));
  float max_new = q2f<32>((long long)s.acc_max, s.min_out, s.max_out);
  const float input_range = __fsub_rn(s.max_out, s.min_out);
  const float output_range = __fsub_rn(max_new, min_new);
  const float recip_output_range = __fdiv_rn(255.0f, output_range);
  const long long recip_output_range_fp =
    (long long)__fmul_rn(recip_output_range, (float)(1 << 16));
  s.range_scale_fp = (long long)__fdiv_rn(
    __fmul_rn(__fmul_rn(255.0f, (float)(1 << 16)), input_range), output_range);
  s.input_offset_fp =
    (long long)__fadd_rn(__fmul_rn(s.min_out, __ll2float_rn(recip_output_range_fp)),
                         __ll2float_rn(s.range_scale_fp >> 1));
  s.output_offset_fp = (long long)roundf(__fdiv_rn(__fmul_rn(min_new, 255.0f), output_range));
  s.min_new = min_new;
  s.max_new = max_new;
}

__global__ void q_requant_params_kernel(QSample *qs, int B) {
  int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= B) return;
  QSample s = qs[n];
  requant_params(s);
  qs[n] = s;
}

// inner loop of requantize_many_in_new_range<int32,uint8> (:172-185): the quantized value of one accumulator
__device__ __forceinline__ int requant_one(int acc, const QSample &s) {
  const long long rounding_delta = 1LL << 15;
  const long long fp_value = (((long long)acc * s.range_scale_fp) >> 32) + s.input_offset_fp;
  const long long ri = ((fp_value >= 0) ? (fp_value + rounding_delta) : (fp_value - rounding_delta)) >> 16;
  const long long q = ri - s.output_offset_fp;
  return q > 0 ? (q < 255 ? (int)q : 255) : 0;
}

// inner loop of requantize_many_in_new_range<int32,uint8> (:172-185) followed
// by quantized_to_float<uint8_t> (:70-84)
__global__ void q_requant_dequant_kernel(const int *__restrict__ acc, size_t out_len,
                                         const QSample *__restrict__ qs, float *__restrict__ out) {
  const int n = blockIdx.y;
  const QSample s = qs[n];
  const int *a = acc + (size_t)n * out_len;
  float *o = out + (size_t)n * out_len;
  size_t step = (size_t)gridDim.x * blockDim.x;
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < out_len; j += step)
    o[j] = q2f<8>(requant_one(a[j], s), s.min_new, s.max_new);
}

// ---- 5b. convolution of a whole sample in one kernel ------------------------------------------------
//
// sum (w - off_w)(x - off_x) = sum w*x - off_x * sum w - off_w * sum x + n * off_w * off_x is exact
// in integers, so the products are taken on bytes by the tensor cores (mma.m16n8k32, unsigned bytes, 32-bit
// sums).  All arithmetic is modulo 2^32 and the true value fits an int32, so intermediate wrap-around is harmless.
//
// A cluster of 1 to 8 blocks takes a sample, each block a run of output pixels: it finds the sample's range
// (blocks exchange theirs), quantizes the input rows that it needs into shared memory with the channels fastest,
// takes the products, exchanges the accumulators' extremes and requantizes.  In eight launches each step read and
// wrote memory (28x28x32 -> 64, 5x5, 128 samples: 247 us, of which the dp4a products 174 us and the requantizing
// 20 us; in one 66 us with the sums in shared memory, a filter fragment read for every unit, and values quantized in double
// precision and requantized in 64 bits; this 39 us).  Cycles of a block there: range 7 k (11 k where each warp read planes of its
// own), quantizing 8 k (15 k from global memory, a branch for every value), window sums 4 k, products 24 k (40 k; shared-memory
// reads), extremes 9 k, requantizing 15 k (28 k with a branch for every value, the stores four bytes each).
// A k step is 32 bytes: four groups of 8 channels, wherever in the window they lie (`tab`); channels are
// padded to 8, the filter's rows to 32 bytes with zeros.
__device__ __noinline__ unsigned quantize_in_double(float v, double scale, double low) {
  const long long q = (long long)__dsub_rn(round(__dmul_rn((double)v, scale)), low);
  return (unsigned)(q > 0 ? (q < 255 ? q : 255) : 0);
}

// f2q<8> of one range: the same operations, the ones that do not depend on the value done once.  Almost every value needs no
// double: the 32-bit product is off by 2^-23 of itself at most, so where its distance from the nearest whole number is that
// far from one half, the exact product rounds to the same one.  (In double alone, with a 64-bit conversion, a value took three times
// as many instructions: 9216 -> 256 with 128 samples spent 12 us on them.)
struct QScale {
  double scale, low;
  float scale32;
  int low32;
  bool flat, quick;
  __device__ __forceinline__ void set(float rmin, float rmax) {
    flat = rmin == rmax;
    const double range_adjust = __ddiv_rn(256.0, __dsub_rn(256.0, 1.0));
    const double range = __dmul_rn((double)__fsub_rn(rmax, rmin), range_adjust);
    scale = __ddiv_rn(256.0, range);
    low = round(__dmul_rn((double)rmin, scale));
    scale32 = (float)scale;
    quick = fabs(low) < 2097152.0 && scale > 1e-30 && scale < 1e30;
    low32 = quick ? (int)low : 0;
  }
  // the value by 32 bits alone, and whether they decide it
  __device__ __forceinline__ unsigned in32(float v, bool &ok) const {
    const float f = __fmul_rn(v, scale32), t = __fadd_rn(f, 12582912.f);  // 1.5 * 2^23: the whole number is in the last bits
    ok = fabsf(f) < 2097152.f && fabsf(__fsub_rn(f, __fsub_rn(t, 12582912.f))) < 0.5f - fabsf(f) * 2.4e-7f;
    return (unsigned)min(255, max(0, __float_as_int(t) - 0x4b400000 - low32));
  }
  __device__ __forceinline__ unsigned of(float v) const {
    if (flat) return 0u;
    bool ok;
    const unsigned r = in32(v, ok);
    return quick && ok ? r : quantize_in_double(v, scale, low);
  }
  // four values to the bytes of a word: one branch for all, so that their chains overlap
  __device__ __forceinline__ unsigned of4(const float *v) const {
    if (flat) return 0u;
    unsigned w = 0u;
    bool all = quick;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      bool ok;
      w |= in32(v[k], ok) << (8 * k);
      all = all && ok;
    }
    if (all) return w;
    w = 0u;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) w |= quantize_in_double(k == 0 ? v[0] : k == 1 ? v[1] : k == 2 ? v[2] : v[3], scale, low) << (8 * k);
    return w;
  }
};

// a word whose first `left` bytes are set
__device__ __forceinline__ unsigned first_bytes(int left) { return left >= 4 ? ~0u : left > 0 ? (1u << (8 * left)) - 1u : 0u; }

__device__ __forceinline__ void mma_u8(unsigned *c, const uint2 &a0, const uint2 &a1, const uint2 &b) {
  // lane (g, q) holds bytes 8 q .. 8 q + 7 of rows g and g + 8 and of column g: the order of the k's is free as long
  // as both operands have the same
  asm volatile(
    "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
    : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
    : "r"(a0.x), "r"(a1.x), "r"(a0.y), "r"(a1.y), "r"(b.x), "r"(b.y));
}

struct QConvArgs {
  const float *in;
  float *out;
  const uint8_t *Wq, *bq;
  const unsigned *wsum;
  const QGlobal *qg;
  int C, HI, WI, OC, OH, OW, KH, KW, SH, SW, has_bias;
  int Cp, ksteps, pitch, ntiles;  // channels padded to 8; k steps; bytes of a filter row; 8-channel tiles of the outputs
  int per, rows;                  // output pixels of a block (a multiple of 16), most input rows it needs
  int copies;                     // of the table of results: 32 or 1
  int raw;                        // the input rows wait in shared memory for their range
  int acc_smem;                   // the accumulators wait in shared memory, not in the output's place
};

constexpr int QC_THREADS = 512, QC_WARPS = QC_THREADS / 32;

// bytes of a filter row in shared memory: 32 or 96 more than a multiple of 128, so that rows fall on different banks
__host__ __device__ __forceinline__ int qc_pitch(int ksteps) { return ksteps * 32 + (ksteps % 2 == 0 ? 32 : 0); }

// filter rows quantized as [o][tap][Cp], their byte sums, the quantized biases and the ranges; a block a row
__global__ void __launch_bounds__(256) q_conv_filter_kernel(const float *__restrict__ W, int nseg, size_t seg_stride,
                                                            size_t seg_len, int C, int Cp, int OC, int KK, int pitch,
                                                            const float *__restrict__ bias, int nbias, QGlobal *out_qg,
                                                            uint8_t *__restrict__ Wq, uint8_t *__restrict__ bq,
                                                            unsigned *__restrict__ wsum) {
  after_previous_kernel();
  __shared__ QGlobal qg;
  __shared__ unsigned part[8];
  filter_range(W, nseg, seg_stride, seg_len, bias, nbias, qg);
  const int o = blockIdx.x;
  QScale q;
  q.set(qg.min_f, qg.max_f);
  unsigned sum = 0;
  for (int k = threadIdx.x; k < pitch; k += 256) {
    const int tap = k / Cp, c = k - tap * Cp;
    const unsigned v = tap < KK && c < C && o < OC ? q.of(W[((size_t)o * C + c) * KK + tap]) : 0u;
    Wq[(size_t)o * pitch + k] = (uint8_t)v;
    sum += v;
  }
  for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; ++k) sum += part[k];
    wsum[o] = sum;
    if (o < nbias) bq[o] = (uint8_t)f2q<8>(bias[o], qg.min_b, qg.max_b);
    if (o == 0) *out_qg = qg;
  }
}

__device__ __forceinline__ void q_cluster_sync(int n) {
  if (n == 1)
    __syncthreads();
  else
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned q_remote(const void *p, int rank) {  // a word of another block's shared memory
  unsigned at, v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(at) : "memory");
  return v;
}

// requant_one in 32 bits.  With scale = hi * 2^32 + lo, lo signed, floor(acc * scale / 2^32) = acc * hi + floor(acc * lo / 2^32), and
// modulo 2^32 that is enough where the sum fits an int32, which it does for every accumulator if it does for the least and
// the largest.  Otherwise (`on` not set) in 64 bits.
struct QQuick {
  int hi, lo, offset, out;
  bool on;
  __device__ __forceinline__ void set(const QSample &s) {
    lo = (int)(unsigned)s.range_scale_fp;
    hi = (int)(unsigned)(((unsigned long long)s.range_scale_fp - (unsigned long long)(long long)lo) >> 32);
    offset = (int)(unsigned)s.input_offset_fp;
    out = (int)(unsigned)s.output_offset_fp;
    const double most = fmax(fabs((double)s.acc_min), fabs((double)s.acc_max)) * fabs((double)s.range_scale_fp);
    on = most < 4e18 && fabs((double)s.input_offset_fp) < 4e18 && fits(s.acc_min, s) && fits(s.acc_max, s) &&
         s.output_offset_fp > -(1LL << 30) && s.output_offset_fp < (1LL << 30);
  }
  __device__ __forceinline__ static bool fits(int acc, const QSample &s) {
    const long long v = (((long long)acc * s.range_scale_fp) >> 32) + s.input_offset_fp;
    return v > -(1LL << 31) + 65536 && v < (1LL << 31) - 65536;
  }
  __device__ __forceinline__ int of(int acc) const {
    const int v = (int)((unsigned)acc * (unsigned)hi + (unsigned)__mulhi(acc, lo) + (unsigned)offset), below = v >> 31;
    return min(255, max(0, ((v + ((32768 ^ below) - below)) >> 16) - out));
  }
};
__device__ __forceinline__ uint2 q_lds8(unsigned at) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(at));
  return v;
}

constexpr int QC_UNITS = 5;   // units of 16 pixels x 32 outputs whose sums a warp keeps in registers
constexpr int QC_STAGE = 20;  // words from output to output of a unit in shared memory

// REGS: the sums wait for the sample's extremes in registers, not in shared memory or in the output's place
template <bool REGS>
__global__ void __launch_bounds__(QC_THREADS, 1) q_conv_fused_kernel(const __grid_constant__ QConvArgs a) {
  extern __shared__ __align__(16) uint8_t qsm[];
  __shared__ float rmin[QC_WARPS], rmax[QC_WARPS], range[2];
  __shared__ int amin[QC_WARPS], amax[QC_WARPS], extremes[2];
  __shared__ QSample smp;
  __shared__ QQuick quick;
  __shared__ float lut[256];
  int nc, rank;
  asm("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(nc));
  asm("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  const int n = blockIdx.x / nc, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int npix = a.OH * a.OW, p0 = min(npix, rank * a.per), p1 = min(npix, p0 + a.per), plane = a.HI * a.WI;
  const int iy0 = p1 > p0 ? p0 / a.OW * a.SH : 0, iy1 = p1 > p0 ? (p1 - 1) / a.OW * a.SH + a.KH : 0;
  const int places = (iy1 - iy0) * a.WI, KK = a.KH * a.KW;
  uint8_t *ws = qsm, *xs = ws + (size_t)a.ntiles * 8 * a.pitch;                      // filter, input
  int *tab = reinterpret_cast<int *>(xs + (size_t)a.rows * a.WI * a.Cp);             // [ksteps * 4]
  unsigned *psum = reinterpret_cast<unsigned *>(tab + a.ksteps * 4);                 // [places] byte sums over the channels
  unsigned *xsum = psum + a.rows * a.WI;                                             // [per] over the window
  int *acc = a.acc_smem ? reinterpret_cast<int *>(xsum + a.per) : reinterpret_cast<int *>(a.out) + (size_t)n * a.OC * npix + p0;
  const int acc_step = a.acc_smem ? a.per : npix;                                    // from output channel to output channel
  float *raw = reinterpret_cast<float *>(((uintptr_t)(xsum + a.per) + 15) & ~(uintptr_t)15);  // [C][places], in the accumulators' place
  wait_for_previous_kernel();
  for (int i = tid; i < a.ntiles * 8 * a.pitch / 16; i += QC_THREADS) cp_async16(ws + 16 * i, a.Wq + 16 * i, true);
  cp_async_commit();
  for (int i = tid; i < a.ksteps * 4; i += QC_THREADS) {
    const int k = i * 8, tap = min(k / a.Cp, KK - 1), c = k % a.Cp;  // groups behind the window meet zeros of the filter
    tab[i] = (tap / a.KW * a.WI + tap % a.KW) * a.Cp + c;
  }
  const float *in = a.in + (size_t)n * a.C * plane;
  if (a.raw) {
    const bool vec = ((plane | places | (iy0 * a.WI)) & 3) == 0 && ((uintptr_t)in & 15) == 0;
    const int unit = vec ? 4 : 1, pu = max(1, places / unit), stepc = QC_THREADS / pu, stepp = QC_THREADS - stepc * pu;
    int c = places > 0 ? tid / pu : a.C, p = tid % pu;
    while (c < a.C) {
      const float *src = in + (size_t)c * plane + iy0 * a.WI + p * unit;
      if (vec)
        cp_async16(raw + c * places + p * 4, src, true);
      else
        cp_async4(raw + c * places + p, src, true);
      c += stepc, p += stepp;
      if (p >= pu) p -= pu, ++c;
    }
    cp_async_commit();
  }
  for (int i = tid; i < places; i += QC_THREADS) psum[i] = 0u;
  // the range: the reference scans the first HI * HI values of every plane, starting from the first value
  {
    float mn = in[0], mx = in[0];
    const int scan = a.HI * a.HI, parts = max(1, QC_WARPS * nc / a.C), span = (scan + parts - 1) / parts;
    const bool vec = ((plane | scan) & 3) == 0 && parts == 1 && ((uintptr_t)in & 15) == 0;
    if (a.raw) {
      // the rows behind the last window, then what the blocks hold: together the whole planes
      const int end = ((a.OH - 1) * a.SH + a.KH) * a.WI;
      if (p1 == npix && p1 > p0 && end < scan)
        for (int c = warp; c < a.C; c += QC_WARPS)
          for (int e = end + lane; e < scan; e += 32) {
            const float v = in[(size_t)c * plane + e];
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
          }
      cp_async_wait<0>();
      __syncthreads();
      const int most = min(places, scan - iy0 * a.WI);  // of a plane's values here
      if (most == places) {
        const float4 *r4 = reinterpret_cast<const float4 *>(raw);
        const int len = a.C * places;
#pragma unroll 4
        for (int e = tid; e < len / 4; e += QC_THREADS) {
          const float4 v = r4[e];
          mn = fminf(mn, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
          mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
        }
        if (tid < (len & 3)) {
          mn = fminf(mn, raw[(len & ~3) + tid]);
          mx = fmaxf(mx, raw[(len & ~3) + tid]);
        }
      } else {
        for (int c = warp; c < a.C; c += QC_WARPS)
          for (int e = lane; e < most; e += 32) {
            mn = fminf(mn, raw[c * places + e]);
            mx = fmaxf(mx, raw[c * places + e]);
          }
      }
    }
    for (int u = rank * QC_WARPS + warp; !a.raw && u < a.C * parts; u += nc * QC_WARPS) {
      const int c = u / parts, b = (u - c * parts) * span;
      if (vec) {  // a plane's loads asked for at once
        const float4 *p = reinterpret_cast<const float4 *>(in + (size_t)c * plane);
#pragma unroll 8
        for (int e = lane; e < scan / 4; e += 32) {
          const float4 v = p[e];
          mn = fminf(mn, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
          mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
        }
        continue;
      }
#pragma unroll 8
      for (int e = b + lane; e < min(scan, b + span); e += 32) {
        const float v = in[(size_t)c * plane + e];
        mn = fminf(mn, v);
        mx = fmaxf(mx, v);
      }
    }
    mn = warp_min(mn);
    mx = warp_max(mx);
    if (lane == 0) {
      rmin[warp] = mn;
      rmax[warp] = mx;
    }
    __syncthreads();
    if (warp == 0) {
      mn = warp_min(rmin[lane & (QC_WARPS - 1)]);
      mx = warp_max(rmax[lane & (QC_WARPS - 1)]);
      if (lane == 0) {
        range[0] = mn;
        range[1] = mx;
      }
    }
    q_cluster_sync(nc);
    if (warp == 0 && nc > 1) {  // a lane a block: one after the other they take 250 cycles each
      mn = warp_min(__uint_as_float(q_remote(&range[0], lane & (nc - 1))));
      mx = warp_max(__uint_as_float(q_remote(&range[1], lane & (nc - 1))));
    }
    if (tid == 0) {
      smp.min_in = mn;
      smp.max_in = mx;
      sample_params(smp, *a.qg, 0);
    }
    __syncthreads();
  }
  {
    QScale q;
    q.set(smp.min_in, smp.max_in);
    // Eight channels of a place.  A sample's last blocks may have no pixels, since runs are rounded up to 16, and hence no
    // places: nothing to do, and nothing to divide by.  (A branch around all this costs 0.15 us a call.)
    const int groups = a.Cp / 8, by = max(1, places);
    int cg = tid / by, p = tid - cg * by;
    if (places == 0) cg = groups;
    const int stepg = QC_THREADS / by, stepp = QC_THREADS - stepg * by;
    // with the sums of a place's bytes
    auto write = [&](int c0, int p, const float(&v)[8]) {
      const int left = a.C - c0;  // channels behind the last are zero bytes
      const unsigned w0 = q.of4(v) & first_bytes(left), w1 = q.of4(v + 4) & first_bytes(left - 4);
      *reinterpret_cast<uint2 *>(xs + (size_t)p * a.Cp + c0) = make_uint2(w0, w1);
      atomicAdd(psum + p, __dp4a(w1, 0x01010101u, __dp4a(w0, 0x01010101u, 0u)));
    };
    if (a.raw) {
      while (cg < groups) {
        const float *src = raw + cg * 8 * places + p;
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = cg * 8 + k < a.C ? src[k * places] : 0.f;
        write(cg * 8, p, v);
        cg += stepg, p += stepp;
        if (p >= places) p -= places, ++cg;
      }
    } else {
      float next[8];
      auto fetch = [&]() {
        const float *src = in + (size_t)cg * 8 * plane + iy0 * a.WI + p;
#pragma unroll
        for (int k = 0; k < 8; ++k) next[k] = cg < groups && cg * 8 + k < a.C ? src[(size_t)k * plane] : 0.f;
      };
      fetch();
      while (cg < groups) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = next[k];
        const int c0 = cg * 8, at = p;
        cg += stepg, p += stepp;
        if (p >= places) p -= places, ++cg;
        fetch();  // the next place's values are on their way meanwhile
        write(c0, at, v);
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int p = tid; p < p1 - p0; p += QC_THREADS) {
    const int y = (p0 + p) / a.OW, x = p0 + p - y * a.OW;
    const unsigned *s = psum + (y * a.SH - iy0) * a.WI + x * a.SW;
    unsigned t = 0;
    for (int ky = 0; ky < a.KH; ++ky)
      for (int kx = 0; kx < a.KW; ++kx) t += s[ky * a.WI + kx];
    xsum[p] = t;
  }
  __syncthreads();
  // products: units of 16 pixels x 4 tiles of 8 outputs
  const unsigned off_f = (unsigned)a.qg->off_f, off_in = (unsigned)smp.off_in, both = (unsigned)(KK * a.C) * off_f * off_in;
  const int mtiles = (p1 - p0 + 15) / 16, ngroups = (a.ntiles + 3) / 4, g = lane >> 2, q = lane & 3;
  int mn = INT_MAX, mx = INT_MIN;
  auto products = [&](int u, unsigned(&c)[4][4]) {
    const int ng = u / mtiles, m = u - ng * mtiles, nt = min(4, a.ntiles - ng * 4);
    const uint8_t *x[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int p = min(p0 + m * 16 + g + 8 * e, p1 - 1), y = p / a.OW;
      x[e] = xs + ((size_t)(y * a.SH - iy0) * a.WI + (p - y * a.OW) * a.SW) * a.Cp;
    }
    const uint8_t *w = ws + (size_t)(ng * 32 + g) * a.pitch + q * 8;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k) c[t][k] = 0;
#pragma unroll 2
    for (int ks = 0; ks < a.ksteps; ++ks) {
      const int off = tab[ks * 4 + q];
      const uint2 a0 = *reinterpret_cast<const uint2 *>(x[0] + off), a1 = *reinterpret_cast<const uint2 *>(x[1] + off);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint2 b = *reinterpret_cast<const uint2 *>(w + (size_t)(t < nt ? t : 0) * 8 * a.pitch + ks * 32);
        mma_u8(c[t], a0, a1, b);
      }
    }
  };
  // f(output channel, pixel, sum) for what this lane holds of a unit
  auto each = [&](int u, const unsigned(&c)[4][4], auto f) {
    const int ng = u / mtiles, m = u - ng * mtiles;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int o = (ng * 4 + t) * 8 + q * 2 + (k & 1), p = m * 16 + g + 8 * (k >> 1);
        if (o < a.OC && p < p1 - p0) f(o, p, c[t][k]);
      }
  };
  auto value = [&](int o, int p, unsigned sum) {
    const int v = (int)(sum - off_in * a.wsum[o] - off_f * xsum[p] + both);
    return a.has_bias ? v + (int)a.bq[o] - smp.zero_total : v;
  };
  const int units = mtiles * ngroups;
  // REGS: a warp's units are pixels of one group of outputs, so that a filter fragment serves all of them: 14 reads of
  // shared memory for 20 products (unit by unit 30, and these reads are what the products take their time for)
  const int wper = REGS ? QC_WARPS / ngroups : 1, wgroup = warp / wper, wfirst = wgroup < ngroups ? warp - wgroup * wper : mtiles;
  auto unit_of = [&](int i) { return wgroup * mtiles + wfirst + i * wper; };
  auto has = [&](int i) { return wfirst + i * wper < mtiles; };
  unsigned c[REGS ? QC_UNITS : 1][4][4];
  if (REGS) {
    unsigned x[QC_UNITS][2];
#pragma unroll
    for (int i = 0; i < QC_UNITS; ++i) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int p = min(p0 + (wfirst + i * wper) * 16 + g + 8 * e, p1 - 1), y = p / a.OW;
        x[i][e] = smem_u32(xs) + (unsigned)((y * a.SH - iy0) * a.WI + (p - y * a.OW) * a.SW) * a.Cp;
      }
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) c[i][t][k] = 0;
    }
    if (wfirst < mtiles) {
      const int nt = min(4, a.ntiles - wgroup * 4);
      const unsigned w = smem_u32(ws) + (unsigned)((wgroup * 32 + g) * a.pitch + q * 8);
      const unsigned step[4] = {0u, nt > 1 ? 8u * a.pitch : 0u, nt > 2 ? 16u * a.pitch : 0u, nt > 3 ? 24u * a.pitch : 0u};
      for (int ks = 0; ks < a.ksteps; ++ks) {
        const unsigned off = (unsigned)tab[ks * 4 + q];
        uint2 f[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) f[t] = q_lds8(w + step[t] + ks * 32);
#pragma unroll
        for (int i = 0; i < QC_UNITS; ++i) {
          if (!has(i)) break;
          const uint2 a0 = q_lds8(x[i][0] + off), a1 = q_lds8(x[i][1] + off);
#pragma unroll
          for (int t = 0; t < 4; ++t) mma_u8(c[i][t], a0, a1, f[t]);
        }
      }
    }
    unsigned of_out[4][2];  // what belongs to an output
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int o = (wgroup * 4 + t) * 8 + q * 2 + k;
        of_out[t][k] = wgroup < ngroups && o < a.OC ? both - off_in * a.wsum[o] + (a.has_bias ? (unsigned)((int)a.bq[o] - smp.zero_total) : 0u) : 0u;
      }
#pragma unroll
    for (int i = 0; i < QC_UNITS; ++i) {
      if (!has(i)) break;
      const int m = wfirst + i * wper;
      const int pa = m * 16 + g, pb = pa + 8;
      const unsigned xa = pa < p1 - p0 ? off_f * xsum[pa] : 0u, xb = pb < p1 - p0 ? off_f * xsum[pb] : 0u;
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int o = (wgroup * 4 + t) * 8 + q * 2 + (k & 1);
          c[i][t][k] += of_out[t][k & 1] - (k < 2 ? xa : xb);
          if (o >= a.OC || (k < 2 ? pa : pb) >= p1 - p0) continue;
          mn = min(mn, (int)c[i][t][k]);
          mx = max(mx, (int)c[i][t][k]);
        }
    }
  } else {
    for (int u = warp; u < units; u += QC_WARPS) {
      products(u, c[0]);
      each(u, c[0], [&](int o, int p, unsigned sum) {
        const int v = value(o, p, sum);
        acc[(size_t)o * acc_step + p] = v;
        mn = min(mn, v);
        mx = max(mx, v);
      });
    }
  }
  mn = warp_min_i(mn);
  mx = warp_max_i(mx);
  if (lane == 0) {
    amin[warp] = mn;
    amax[warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    mn = warp_min_i(amin[lane & (QC_WARPS - 1)]);
    mx = warp_max_i(amax[lane & (QC_WARPS - 1)]);
    if (lane == 0) {
      extremes[0] = mn;
      extremes[1] = mx;
    }
  }
  q_cluster_sync(nc);
  if (warp == 0 && nc > 1) {
    mn = warp_min_i((int)q_remote(&extremes[0], lane & (nc - 1)));
    mx = warp_max_i((int)q_remote(&extremes[1], lane & (nc - 1)));
  }
  if (tid == 0) {
    smp.acc_min = mn;
    smp.acc_max = mx;
    requant_params(smp);
    quick.set(smp);
  }
  q_cluster_sync(nc);  // nobody leaves while others may read its extremes
  const QSample s = smp;
  // the 256 results: a copy for every lane where filter and input were, so that no two lanes want the same bank
  if (tid < 256) lut[tid] = q2f<8>(tid, s.min_new, s.max_new);
  __syncthreads();
  const float *table = lut;
  if (a.copies > 1) {
    float *t = reinterpret_cast<float *>(qsm);
    for (int i = warp; i < 256; i += QC_WARPS) t[i * 32 + lane] = lut[i];
    __syncthreads();
    table = t;
  }
  const int tstep = a.copies, tlane = lane & (a.copies - 1);
  float *out = a.out + (size_t)n * a.OC * npix + p0;
  const QQuick qk = quick;
  auto requant = [&](int v) { return qk.on ? qk.of(v) : requant_one(v, s); };
  if (REGS) {
    // A unit at a time through the warp's own shared memory, four neighbouring pixels a lane: only the way there is written out
    // for each of the 80 registers, and rows of 64 bytes are stored.
    int *mine = reinterpret_cast<int *>(qsm + 32 * 256 * sizeof(float)) + warp * (32 * QC_STAGE);
    const bool vec = (npix & 3) == 0 && ((uintptr_t)a.out & 15) == 0;  // p0 is a multiple of 16
#pragma unroll 1
    for (int i = 0; i < QC_UNITS; ++i) {
      if (!has(i)) break;
#pragma unroll
      for (int u = 0; u < QC_UNITS; ++u) {
        if (u != i) continue;
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int k = 0; k < 4; ++k) mine[(t * 8 + q * 2 + (k & 1)) * QC_STAGE + g + 8 * (k >> 1)] = (int)c[u][t][k];
      }
      __syncwarp();
      const int p = (wfirst + i * wper) * 16 + (lane & 3) * 4, left = p1 - p0 - p;
#pragma unroll 1
      for (int t = 0; t < 4; ++t) {
        const int o = (wgroup * 4 + t) * 8 + g;
        if (o >= a.OC || left <= 0) continue;
        const int4 v = *reinterpret_cast<const int4 *>(mine + (t * 8 + g) * QC_STAGE + (lane & 3) * 4);
        const int r4[4] = {v.x, v.y, v.z, v.w};
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) r[e] = table[requant(r4[e]) * tstep + tlane];
        float *dst = out + (size_t)o * npix + p;
        if (vec && left >= 4)
          *reinterpret_cast<float4 *>(dst) = make_float4(r[0], r[1], r[2], r[3]);
        else
          for (int e = 0; e < 4 && e < left; ++e) dst[e] = e == 0 ? r[0] : e == 1 ? r[1] : e == 2 ? r[2] : r[3];
      }
      __syncwarp();
    }
    return;
  }
  const int count = p1 - p0;
  for (int i = tid; i < a.OC * count; i += QC_THREADS) {
    const int o = i / count, p = i - o * count;
    out[(size_t)o * npix + p] = table[requant(acc[(size_t)o * acc_step + p]) * tstep + tlane];
  }
}

// ---- 5c. fully connected ----------------------------------------------------------------------------
//
// Four launches: ranges of the samples and of the filter (B + `wblocks` blocks), quantizing (the filter transposed to
// [out][in]), the byte products (tensor cores as above; tiles of 64 samples x 64 outputs, the inputs dealt to
// enough blocks to fill the chip, whole-number sums added in any order), and a sample's requantizing by one block.
// In nine launches 9216 -> 256 of 128 samples took 64 us, in four 34 us, and 23 us since a launch overlaps the end of the one
// before it and few values are quantized in double precision; what is left is reading the filter twice and four chains of
// load, arithmetic and store.
__global__ void __launch_bounds__(256) q_fc_range_kernel(const float *__restrict__ in, int in_size, int B,
                                                         const float *__restrict__ W, size_t lenW, int out_size, QSample *qs,
                                                         float *__restrict__ part, int *__restrict__ acc,
                                                         unsigned *__restrict__ wsum) {
  after_previous_kernel();
  const bool row = (int)blockIdx.x < B;
  const int w = blockIdx.x - B, nw = gridDim.x - B;
  const float *v = row ? in + (size_t)blockIdx.x * in_size : W;
  const size_t len = row ? (size_t)in_size : lenW;
  const size_t first = row ? threadIdx.x : (size_t)w * 256 + threadIdx.x, step = row ? 256 : (size_t)nw * 256;
  float mn = v[0], mx = v[0];
  if (((uintptr_t)v & 15) == 0) {
    const float4 *v4 = reinterpret_cast<const float4 *>(v);
#pragma unroll 4
    for (size_t i = first; i < len / 4; i += step) {
      const float4 x = v4[i];
      mn = fminf(fminf(fminf(mn, x.x), fminf(x.y, x.z)), x.w);
      mx = fmaxf(fmaxf(fmaxf(mx, x.x), fmaxf(x.y, x.z)), x.w);
    }
    for (size_t i = len / 4 * 4 + first; i < len; i += step) {
      mn = fminf(mn, v[i]);
      mx = fmaxf(mx, v[i]);
    }
  } else {
#pragma unroll 4
    for (size_t i = first; i < len; i += step) {
      mn = fminf(mn, v[i]);
      mx = fmaxf(mx, v[i]);
    }
  }
  __shared__ float smn[8], smx[8];
  mn = warp_min(mn);
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) {
    smn[threadIdx.x >> 5] = mn;
    smx[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    mn = warp_min(smn[threadIdx.x & 7]);
    mx = warp_max(smx[threadIdx.x & 7]);
    if (threadIdx.x == 0) {
      if (row) {
        qs[blockIdx.x].min_in = mn;
        qs[blockIdx.x].max_in = mx;
        qs[blockIdx.x].sum_in = 0;
      } else {
        part[2 * w] = mn;
        part[2 * w + 1] = mx;
      }
    }
  }
  if (row)
    for (int i = threadIdx.x; i < out_size; i += 256) acc[(size_t)blockIdx.x * out_size + i] = 0;
  else if (w == 0)
    for (int i = threadIdx.x; i < out_size; i += 256) wsum[i] = 0u;
}

// The first blocks take 32 outputs x 128 inputs of the filter each, the others 1024 bytes of a sample's row.  Bound by the latency
// of a filter block's chain (range, then loads and conversions), so those start first, are short, and ask for their part of the
// filter before they wait for the ranges (9216 -> 256, 128 samples: 18.3 us with 256 inputs a block behind the rows, 12.07 us
// with every value in double precision and all loads behind the wait).
constexpr int QF_CIN = 128;
__global__ void __launch_bounds__(256) q_fc_quantize_kernel(const float *__restrict__ in, int in_size, int B, int pitch,
                                                            int rblocks, const float *__restrict__ W, int out_size,
                                                            const float *__restrict__ bias, int nbias,
                                                            const float *__restrict__ part, int nparts, QSample *qs,
                                                            QGlobal *out_qg, uint8_t *__restrict__ inq,
                                                            uint8_t *__restrict__ Wt, uint8_t *__restrict__ bq,
                                                            unsigned *__restrict__ wsum) {
  const int b = blockIdx.x, fblocks = gridDim.x - B * rblocks;
  if (b >= fblocks) {
    after_previous_kernel();
    const int n = (b - fblocks) / rblocks, j0 = (b - fblocks - n * rblocks) * 1024 + threadIdx.x * 4;
    const float *r = in + (size_t)n * in_size;
    QScale q;
    q.set(qs[n].min_in, qs[n].max_in);
    int sum = 0;
    if (j0 < pitch) {  // pitch is a multiple of 4
      float x[4];
      if (j0 + 4 <= in_size && ((uintptr_t)(r + j0) & 15) == 0) {
        const float4 y = *reinterpret_cast<const float4 *>(r + j0);
        x[0] = y.x, x[1] = y.y, x[2] = y.z, x[3] = y.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = j0 + k < in_size ? r[j0 + k] : 0.f;
      }
      const unsigned w = q.of4(x) & first_bytes(in_size - j0);
      sum = (int)__dp4a(w, 0x01010101u, 0u);
      *reinterpret_cast<unsigned *>(inq + (size_t)n * pitch + j0) = w;
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&qs[n].sum_in, sum);
    return;
  }
  __shared__ QGlobal qg;
  __shared__ uint8_t tile[QF_CIN][36];
  const int oblocks = (out_size + 31) / 32;
  const int i0 = b % oblocks * 32, c0 = b / oblocks * QF_CIN, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float x[QF_CIN / 8];  // on their way while the range is found
#pragma unroll
  for (int k = 0; k < QF_CIN / 8; ++k) {
    const int c = c0 + warp + 8 * k, i = i0 + lane;
    x[k] = c < in_size && i < out_size ? __ldcg(W + (size_t)c * out_size + i) : 0.f;
  }
  // The filter's values may be asked for ahead of this wait: the ranges' kernel, which let this one begin, only read them and had
  // itself waited for whoever wrote them.  From the L2 cache, where those writes are by then: what the wait also does is
  // to make an SM's L1 cache forget the lines it held from before.
  after_previous_kernel();
  // the partial results stand in for the filter: same extremes, and when all are equal so is W[0]
  filter_range(part, 1, 0, (size_t)2 * nparts, bias, nbias, qg);
  if (b == 0) {
    if (threadIdx.x == 0) *out_qg = qg;
    for (int j = threadIdx.x; j < nbias; j += 256) bq[j] = (uint8_t)f2q<8>(bias[j], qg.min_b, qg.max_b);
  }
  QScale q;
  q.set(qg.min_f, qg.max_f);
  unsigned sum = 0;
#pragma unroll
  for (int k = 0; k < QF_CIN / 8; k += 4) {
    const unsigned v = q.of4(x + k) & first_bytes(i0 + lane < out_size ? (in_size - c0 - warp + 7) / 8 - k : 0);
#pragma unroll
    for (int e = 0; e < 4; ++e) tile[warp + 8 * (k + e)][lane] = (uint8_t)(v >> (8 * e));
    sum = __dp4a(v, 0x01010101u, sum);
  }
  if (i0 + lane < out_size && sum) atomicAdd(&wsum[i0 + lane], sum);
  __syncthreads();
  // a warp writes rows of 128 bytes, a lane 4 bytes of each
  for (int r = warp; r < 32; r += 8) {
    if (i0 + r >= out_size) break;
    unsigned v = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) v |= (unsigned)tile[lane * 4 + k][r] << (8 * k);
    if (c0 + lane * 4 < pitch) *reinterpret_cast<unsigned *>(Wt + (size_t)(i0 + r) * pitch + c0 + lane * 4) = v;
  }
}

constexpr int QF_K = 512;  // bytes of a row in shared memory at a time; pitch 544: rows on different banks
__global__ void __launch_bounds__(256) q_fc_gemm_kernel(int B, int out_size, int pitch, int per,
                                                        const uint8_t *__restrict__ inq, const uint8_t *__restrict__ Wt,
                                                        int *__restrict__ acc) {
  extern __shared__ __align__(16) uint8_t qsm[];
  constexpr int ROW = QF_K + 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64, k0 = blockIdx.z * per, k1 = min(pitch, k0 + per);
  uint8_t *xs = qsm, *ws = xs + 64 * ROW;
  unsigned c[4][4];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int k = 0; k < 4; ++k) c[t][k] = 0;
  const uint8_t *xa = xs + ((warp >> 1) * 16 + g) * ROW + q * 8, *wb = ws + ((warp & 1) * 32 + g) * ROW + q * 8;
  after_previous_kernel();
  for (int kb = k0; kb < k1; kb += QF_K) {
    for (int i = tid; i < 128 * (QF_K / 16); i += 256) {
      const int r = i / (QF_K / 16), at = i % (QF_K / 16) * 16, k = kb + at;
      const bool x = r < 64;
      const int row = x ? m0 + r : n0 + r - 64;
      const bool ok = row < (x ? B : out_size) && k < k1;
      cp_async16((x ? xs : ws) + (size_t)(r & 63) * ROW + at, (x ? inq : Wt) + (ok ? (size_t)row * pitch + k : 0), ok);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int steps = (min(k1 - kb, QF_K) + 31) / 32;
#pragma unroll 4
    for (int ks = 0; ks < steps; ++ks) {
      const uint2 a0 = *reinterpret_cast<const uint2 *>(xa + ks * 32), a1 = *reinterpret_cast<const uint2 *>(xa + 8 * ROW + ks * 32);
#pragma unroll
      for (int t = 0; t < 4; ++t) mma_u8(c[t], a0, a1, *reinterpret_cast<const uint2 *>(wb + t * 8 * ROW + ks * 32));
    }
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int n = m0 + (warp >> 1) * 16 + g + (k >> 1) * 8, o = n0 + (warp & 1) * 32 + t * 8 + q * 2 + (k & 1);
      if (n < B && o < out_size) atomicAdd(&acc[(size_t)n * out_size + o], (int)c[t][k]);
    }
}

__global__ void __launch_bounds__(256) q_fc_requant_kernel(int in_size, int out_size, int has_bias,
                                                           const int *__restrict__ acc, const QSample *__restrict__ qs,
                                                           const QGlobal *__restrict__ qg, const unsigned *__restrict__ wsum,
                                                           const uint8_t *__restrict__ bq, float *__restrict__ out) {
  after_previous_kernel();
  __shared__ QSample s;
  __shared__ int smn[8], smx[8];
  const int n = blockIdx.x, tid = threadIdx.x;
  const unsigned sum_in = (unsigned)qs[n].sum_in;
  if (tid == 0) {
    s = qs[n];
    sample_params(s, *qg, 1);
  }
  __syncthreads();
  const unsigned off_f = (unsigned)qg->off_f, off_in = (unsigned)s.off_in;
  const unsigned both = (unsigned)in_size * off_f * off_in - off_f * sum_in;
  const int zero = s.zero_total;
  auto value = [&](int i) {
    int v = (int)((unsigned)acc[(size_t)n * out_size + i] - off_in * wsum[i] + both);
    return has_bias ? v + (int)bq[i] - zero : v;
  };
  int mn = INT_MAX, mx = INT_MIN;
  for (int i = tid; i < out_size; i += 256) {
    const int v = value(i);
    mn = min(mn, v);
    mx = max(mx, v);
  }
  mn = warp_min_i(mn);
  mx = warp_max_i(mx);
  if ((tid & 31) == 0) {
    smn[tid >> 5] = mn;
    smx[tid >> 5] = mx;
  }
  __syncthreads();
  if (tid == 0) {
    for (int k = 1; k < 8; ++k) mn = min(mn, smn[k]), mx = max(mx, smx[k]);
    s.acc_min = mn;
    s.acc_max = mx;
    requant_params(s);
  }
  __syncthreads();
  const QSample t = s;
  for (int i = tid; i < out_size; i += 256) out[(size_t)n * out_size + i] = q2f<8>(requant_one(value(i), t), t.min_new, t.max_new);
}

// ---- 5d. small fully-connected layers in one launch --------------------------------------------------
//
// What bounds the four launches above on a small layer is the chain: range, quantizing, products, requantizing, with a launch and
// a trip to memory each (232 -> 21, 125 samples: 22.6 us, most of it the host's).  Here one cluster of up to eight blocks goes
// through the phases with two cluster barriers between them.  A block takes a slice of at most 256 inputs, 64
// outputs and 128 samples; it reads its values of the filter and the samples once, into registers, finds their
// ranges, waits for the other blocks', quantizes what it holds into shared memory, and adds its products -- already with the
// zero points' terms, so that no sums over bytes are exchanged -- to the accumulators.  Behind the second barrier
// a warp requantizes a sample.  (That layer 11.7 us, 64 -> 10 of one sample 9.0 for 19.0.  With a grid of up to 144 blocks and
// grid barriers 9216 -> 256 of 128 samples took 43 us, where the launches take 23.)
constexpr int QO_THREADS = 512, QO_WARPS = QO_THREADS / 32, QO_M = 128, QO_N = 64, QO_BLOCKS = 8;
constexpr int QO_ROW = 256 + 32;  // bytes from row to row in shared memory: rows on different banks
constexpr int QO_SMEM = (QO_M + QO_N) * QO_ROW;

struct QFcArgs {
  const float *in, *W, *bias;
  float *out;
  int B, in_size, out_size, nbias;
  int klog, slices, ntiles;   // inputs of a slice as a power of two
  int vec;                    // rows of the input start on 16-byte boundaries
  float2 *wpart, *xpart;      // ranges of the blocks' filter values [blocks] and of the samples' slices [parts][B]
  float2 *xrange;             // [B]
  int *acc;                   // [B][out_size]
};

__global__ void __launch_bounds__(QO_THREADS, 1) q_fc_whole_kernel(const __grid_constant__ QFcArgs a) {
  extern __shared__ __align__(16) uint8_t qsm[];
  __shared__ QScale xq[QO_M], wq, bq;
  __shared__ int xoff[QO_M], xsum[QO_M], wsum[QO_N], off_f;
  __shared__ QGlobal qg;
  __shared__ float wmn[QO_WARPS], wmx[QO_WARPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ks = blockIdx.x % a.slices, nt = blockIdx.x / a.slices % a.ntiles, mt = blockIdx.x / a.slices / a.ntiles;
  const int m0 = mt * QO_M, n0 = nt * QO_N, k0 = ks << a.klog, wlog = a.klog - 2, words = 1 << wlog;  // words of four inputs
  const int nk = min(a.in_size - k0, 1 << a.klog), rows = min(a.B - m0, QO_M);
  after_previous_kernel();
  // ---- values and their ranges ----
  float x[16][4], w[8][4];
#pragma unroll
  for (int j = 0; j < 16; ++j) {  // word kq of row r
    if (j * 4 >= words || (warp * 32 + j * QO_THREADS) >> wlog >= rows) break;
    const int p = tid + j * QO_THREADS, r = p >> wlog, k = (p & (words - 1)) * 4;
    const float *src = a.in + (size_t)(m0 + r) * a.in_size + k0 + k;
    const bool live = r < rows;
    if (a.vec) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live && k < nk) v = *reinterpret_cast<const float4 *>(src);
      x[j][0] = v.x, x[j][1] = v.y, x[j][2] = v.z, x[j][3] = v.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[j][e] = live && k + e < nk ? src[e] : 0.f;
    }
  }
  const int n = tid & (QO_N - 1), q0 = tid >> 6;
#pragma unroll
  for (int j = 0; j < 8; ++j) {  // words q0 + 8 j of output n
    if (j * 8 >= words) break;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = (q0 + 8 * j) * 4 + e;
      w[j][e] = n0 + n < a.out_size && k < nk ? a.W[(size_t)(k0 + k) * a.out_size + n0 + n] : 0.f;
    }
  }
  if (a.slices > 1)
    for (size_t i = blockIdx.x * (size_t)QO_THREADS + tid; i < (size_t)a.B * a.out_size; i += (size_t)gridDim.x * QO_THREADS)
      a.acc[i] = 0;
  {
    float mn = a.W[0], mx = mn;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j * 8 >= words) break;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + n < a.out_size && (q0 + 8 * j) * 4 + e < nk) mn = fminf(mn, w[j][e]), mx = fmaxf(mx, w[j][e]);
    }
    mn = warp_min(mn);
    mx = warp_max(mx);
    if (lane == 0) wmn[warp] = mn, wmx[warp] = mx;
  }
  // the blocks of a slice's output tiles share its rows
  const int halves = words > 32 ? 2 : 1, span = min(words, 32);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j * 4 >= words || (warp * 32 + j * QO_THREADS) >> wlog >= rows) break;
    if (j % a.ntiles != nt) continue;
    const int p = tid + j * QO_THREADS, r = p >> wlog, k = (p & (words - 1)) * 4;
    const bool live = r < rows;
    float mn = live ? a.in[(size_t)(m0 + r) * a.in_size] : 0.f, mx = mn;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (live && k + e < nk) mn = fminf(mn, x[j][e]), mx = fmaxf(mx, x[j][e]);
    for (int o = span >> 1; o > 0; o >>= 1) {
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (live && (lane & (span - 1)) == 0)
      a.xpart[(size_t)(ks * halves + (halves == 2 ? (p >> 5) & 1 : 0)) * a.B + m0 + r] = make_float2(mn, mx);
  }
  __syncthreads();
  if (tid == 0) {
    float mn = wmn[0], mx = wmx[0];
    for (int i = 1; i < QO_WARPS; ++i) mn = fminf(mn, wmn[i]), mx = fmaxf(mx, wmx[i]);
    a.wpart[blockIdx.x] = make_float2(mn, mx);
  }
  q_cluster_sync(2);
  // ---- scales: a thread a sample, a warp the filter and the biases ----
  if (tid < QO_M) {
    if (tid < rows) {
      float mn = a.in[(size_t)(m0 + tid) * a.in_size], mx = mn;
#pragma unroll 8
      for (int i = 0; i < a.slices * halves; ++i) {
        const float2 v = __ldcg(a.xpart + (size_t)i * a.B + m0 + tid);
        mn = fminf(mn, v.x);
        mx = fmaxf(mx, v.y);
      }
      xq[tid].set(mn, mx);
      xoff[tid] = (int)f2q_unclamped<8>(0.0f, mn, mx);
      if (ks == 0 && nt == 0) a.xrange[m0 + tid] = make_float2(mn, mx);
    }
  } else if (warp == QO_M / 32) {
    float mn = a.W[0], mx = mn, bmn = 0.f, bmx = 0.f;
    for (int i = lane; i < (int)gridDim.x; i += 32) {
      const float2 v = __ldcg(a.wpart + i);
      mn = fminf(mn, v.x);
      mx = fmaxf(mx, v.y);
    }
    for (int i = lane; i < a.nbias; i += 32) {
      bmn = fminf(bmn, a.bias[i]);
      bmx = fmaxf(bmx, a.bias[i]);
    }
    mn = warp_min(mn), mx = warp_max(mx), bmn = warp_min(bmn), bmx = warp_max(bmx);
    if (lane == 0) {
      widen_ranges(a.W[0], a.nbias > 0 ? a.bias[0] : 0.f, a.nbias, &mn, &mx, &bmn, &bmx);
      qg.min_f = mn, qg.max_f = mx, qg.min_b = bmn, qg.max_b = bmx;
      off_f = qg.off_f = (int)f2q_unclamped<8>(0.0f, mn, mx);
      wq.set(mn, mx);
      bq.set(bmn, bmx);
    }
  }
  __syncthreads();
  // ---- bytes, the inputs of a row side by side ----
  uint8_t *xs = qsm, *ws = qsm + QO_M * QO_ROW;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (j * 4 >= words || (warp * 32 + j * QO_THREADS) >> wlog >= rows) break;  // rows behind the last are multiplied and not used
    const int p = tid + j * QO_THREADS, r = p >> wlog, k = (p & (words - 1)) * 4;
    *reinterpret_cast<unsigned *>(xs + r * QO_ROW + k) = r < rows ? xq[r].of4(x[j]) & first_bytes(nk - k) : 0u;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (j * 8 >= words) break;
    const int k = (q0 + 8 * j) * 4;
    *reinterpret_cast<unsigned *>(ws + n * QO_ROW + k) = n0 + n < a.out_size ? wq.of4(w[j]) & first_bytes(nk - k) : 0u;
  }
  __syncthreads();
  if (tid < QO_M + QO_N) {  // byte sums of the rows (the filter's lie behind the samples')
    unsigned s = 0;
    for (int i = 0; i < words; i += 4) {
      const uint4 v = *reinterpret_cast<const uint4 *>(qsm + tid * QO_ROW + i * 4);
      s = __dp4a(v.x, 0x01010101u, __dp4a(v.y, 0x01010101u, __dp4a(v.z, 0x01010101u, __dp4a(v.w, 0x01010101u, s))));
    }
    (tid < QO_M ? xsum[tid] : wsum[tid - QO_M]) = (int)s;
  }
  // ---- products: a warp 16 samples x 32 outputs ----
  const int g = lane >> 2, q = lane & 3, mw = warp & 7, nw = warp >> 3;
  unsigned c[4][4];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int k = 0; k < 4; ++k) c[t][k] = 0;
  if (mw * 16 < rows) {
    const uint8_t *xa = xs + (mw * 16 + g) * QO_ROW + q * 8, *wb = ws + (nw * 32 + g) * QO_ROW + q * 8;
    for (int s = 0; s < words / 8; ++s) {
      const uint2 a0 = *reinterpret_cast<const uint2 *>(xa + s * 32), a1 = *reinterpret_cast<const uint2 *>(xa + 8 * QO_ROW + s * 32);
#pragma unroll
      for (int t = 0; t < 4; ++t) mma_u8(c[t], a0, a1, *reinterpret_cast<const uint2 *>(wb + t * 8 * QO_ROW + s * 32));
    }
  }
  __syncthreads();
  // through shared memory, so that a warp adds to 32 neighbours
  int *st = reinterpret_cast<int *>(qsm);
  constexpr int SP = QO_N + 2;
  static_assert(QO_M * SP * 4 <= QO_SMEM, "the sums take the bytes' place");
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int m = mw * 16 + g + (k >> 1) * 8, o = nw * 32 + t * 8 + q * 2 + (k & 1);
      if (m < rows)
        st[m * SP + o] = (int)(c[t][k] - (unsigned)xoff[m] * (unsigned)wsum[o] - (unsigned)off_f * (unsigned)xsum[m] +
                               (unsigned)nk * (unsigned)off_f * (unsigned)xoff[m]);
    }
  __syncthreads();
  for (int i = tid; i < rows * QO_N; i += QO_THREADS) {
    const int m = i / QO_N, o = i % QO_N;
    if (n0 + o >= a.out_size) continue;
    int *dst = a.acc + (size_t)(m0 + m) * a.out_size + n0 + o;
    if (a.slices > 1)
      atomicAdd(dst, st[m * SP + o]);
    else
      *dst = st[m * SP + o];
  }
  q_cluster_sync(2);
  // ---- a warp requantizes a sample ----
  for (int r = blockIdx.x + (int)gridDim.x * warp; r < a.B; r += (int)gridDim.x * QO_WARPS) {
    QSample s = {};
    const float2 range = __ldcg(a.xrange + r);
    s.min_in = range.x;
    s.max_in = range.y;
    sample_params(s, qg, 1);
    const int *acc = a.acc + (size_t)r * a.out_size;
    auto value = [&](int i) {
      const int v = __ldcg(acc + i);
      return a.nbias ? (int)((unsigned)v + bq.of(a.bias[i]) - (unsigned)s.zero_total) : v;
    };
    int mn = INT_MAX, mx = INT_MIN;
    for (int i = lane; i < a.out_size; i += 32) {
      const int v = value(i);
      mn = min(mn, v);
      mx = max(mx, v);
    }
    s.acc_min = warp_min_i(mn);
    s.acc_max = warp_max_i(mx);
    requant_params(s);
    for (int i = lane; i < a.out_size; i += 32)
      a.out[(size_t)r * a.out_size + i] = q2f<8>(requant_one(value(i), s), s.min_new, s.max_new);
  }
}

// ---- 7. the forms for chained quantized layers ("eq") -----------------------------------------
// Operands are uint8 values held in floats, with their ranges; the result leaves the same way
// (tiny_quantized_conv2d_kernel.h:353-466, tiny_quantized_fully_connected_kernel.h:269-370).

// ranges, offsets and the accumulator range of every sample from the supplied ranges
__global__ void q_eq_params_kernel(QSample *qs, QGlobal *qg, const float *__restrict__ in_r,
                                   const float *__restrict__ W_r, const float *__restrict__ b_r, int B, int fc,
                                   int has_bias) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= B) return;
  float min_f = W_r[0], max_f = W_r[1];
  if (min_f == max_f) {
    max_f = __fadd_rn(W_r[1], 1e-3f);
    min_f = __fsub_rn(W_r[0], 1e-3f);
  }
  float min_b = 0.f, max_b = 0.f;
  if (fc) {  // only the fully-connected kernel reads the bias range (:286-293, :313-314)
    min_b = b_r[0];
    max_b = b_r[1];
    if (has_bias && min_b == max_b) {
      max_b = __fadd_rn(b_r[1], 1e-3f);
      min_b = __fsub_rn(b_r[0], 1e-3f);
    }
  }
  QSample s = qs[n];
  s.min_in = in_r[2 * n];
  s.max_in = in_r[2 * n + 1];
  const float c_level = __fmul_rn(one_level_u8(s.min_in, s.max_in), one_level_u8(min_f, max_f));
  float mn = __fmul_rn(c_level, (float)(-(1LL << 31)));
  float mx = __fmul_rn(c_level, (float)((1LL << 31) - 1));
  if (fc) {
    mn = __fadd_rn(mn, min_b);
    mx = __fadd_rn(mx, max_b);
  }
  s.min_out = mn;
  s.max_out = mx;
  s.off_in = (int)f2q_unclamped<8>(0.0f, s.min_in, s.max_in);
  s.zero_total = (int)f2q<32>(0.0f, mn, mx);
  s.acc_min = INT_MAX;
  s.acc_max = INT_MIN;
  s.sum_in = 0;
  qs[n] = s;
  if (n == 0) {
    qg->min_f = min_f;
    qg->max_f = max_f;
    qg->min_b = min_b;
    qg->max_b = max_b;
    qg->off_f = (int)f2q_unclamped<8>(0.0f, min_f, max_f);
  }
}

// static_cast<uint8_t>(float) of values that are uint8 already
__global__ void q_cast_u8_kernel(const float *__restrict__ src, uint8_t *__restrict__ dst, size_t n) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t step = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += step) dst[i] = (uint8_t)__float2int_rz(src[i]);
}

// fully-connected accumulate on the reference's [in][out] byte filter: one thread per (sample, output)
__global__ void q_fc_acc_kernel(int in_size, int out_size, int has_bias, const uint8_t *__restrict__ inq,
                                const uint8_t *__restrict__ Wq, const uint8_t *__restrict__ bq,
                                const QGlobal *__restrict__ qg, QSample *qs, int *__restrict__ acc) {
  const int n = blockIdx.y;
  const int off_f = qg->off_f, off_in = qs[n].off_in, zero_total = qs[n].zero_total;
  const uint8_t *x = inq + (size_t)n * in_size;
  int mn = INT_MAX, mx = INT_MIN;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < out_size; i += gridDim.x * blockDim.x) {
    int sum = 0;
    for (int c = 0; c < in_size; ++c) sum += ((int)Wq[(size_t)c * out_size + i] - off_f) * ((int)x[c] - off_in);
    if (has_bias) sum += (int)bq[i] - zero_total;
    acc[(size_t)n * out_size + i] = sum;
    mn = min(mn, sum);
    mx = max(mx, sum);
  }
  block_minmax_atomic(mn, mx, &qs[n].acc_min, &qs[n].acc_max);
}

// requantize to uint8 held in floats, and hand the shrunk range out (:455-465 / :358-369)
__global__ void q_requant_u8_kernel(const int *__restrict__ acc, size_t out_len, const QSample *__restrict__ qs,
                                    float *__restrict__ out, float *__restrict__ out_r) {
  const int n = blockIdx.y;
  const QSample s = qs[n];
  const int *a = acc + (size_t)n * out_len;
  float *o = out + (size_t)n * out_len;
  size_t step = (size_t)gridDim.x * blockDim.x;
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < out_len; j += step)
    o[j] = (float)requant_one(a[j], s);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    out_r[2 * n] = s.min_new;
    out_r[2 * n + 1] = s.max_new;
  }
}

// ---- host side -------------------------------------------------------------------------

static int blocks_for(size_t n, int block) {
  size_t b = (n + block - 1) / block;
  if (b > 1024) b = 1024;
  if (b < 1) b = 1;
  return (int)b;
}

struct QScratch {
  QSample *qs;
  QGlobal *qg;
  uint8_t *inq, *Wq, *bq;
  float *part;
  int *acc;
};

constexpr int Q_PART_BLOCKS = 592;

static int q_carve(b200_ctx *ctx, int B, size_t in_len, size_t lenW, size_t nbias, size_t out_len,
                   QScratch *s) {
  size_t o_qs = 0;
  size_t o_qg = align_up(o_qs + sizeof(QSample) * (size_t)B, 256);
  size_t o_part = align_up(o_qg + sizeof(QGlobal), 256);
  size_t o_in = align_up(o_part + sizeof(float) * 2 * Q_PART_BLOCKS, 256);
  size_t o_w = align_up(o_in + in_len * B, 256);
  size_t o_b = align_up(o_w + lenW, 256);
  size_t o_acc = align_up(o_b + nbias + 1, 256);
  size_t total = o_acc + sizeof(int) * out_len * B;
  void *base = nullptr;
  B200_TRY(ctx_scratch(ctx, total, &base));
  char *p = static_cast<char *>(base);
  s->qs = reinterpret_cast<QSample *>(p + o_qs);
  s->qg = reinterpret_cast<QGlobal *>(p + o_qg);
  s->part = reinterpret_cast<float *>(p + o_part);
  s->inq = reinterpret_cast<uint8_t *>(p + o_in);
  s->Wq = reinterpret_cast<uint8_t *>(p + o_w);
  s->bq = reinterpret_cast<uint8_t *>(p + o_b);
  s->acc = reinterpret_cast<int *>(p + o_acc);
  return 0;
}

int qconv_fwd(b200_ctx *ctx, const b200_conv_desc *d, const float *in, const float *W,
              const float *bias, float *out, int B) {
  b200_conv_desc dd = *d;
  dd.input_is_padded = 1;  // the quantized layer pads before its backend call
                           // (quantized_convolutional_layer.h:402-437)
  ConvGeom g;
  B200_TRY(conv_geom_from_desc(ctx, &dd, &g));
  B200_REQUIRE(g.DH == 1 && g.DW == 1, "quantized convolution has no dilation");
  if (B == 0) return 0;
  const size_t plane = (size_t)g.HI * g.WI;
  const size_t in_len = plane * g.C, out_len = (size_t)g.OC * g.OH * g.OW;
  const size_t lenW = conv_weight_len(g);
  // The reference scans height*height elements per input plane and
  // k_h*k_h filter elements at input-plane offsets; refuse shapes where those
  // scans would leave the buffers (the reference reads out of bounds there).
  B200_REQUIRE((size_t)(g.C - 1) * plane + (size_t)g.HI * g.HI <= in_len,
               "quantized convolution: in_padded height %d > width %d makes the reference scan "
               "past the input row", g.HI, g.WI);
  B200_REQUIRE((size_t)(g.C - 1) * plane + (size_t)g.KH * g.KH <= lenW,
               "quantized convolution: the reference's filter range scan leaves the filter "
               "tensor for this shape");
  cudaStream_t st = ctx->stream;
  const int nbias = g.has_bias ? g.OC : 0;
  if (!g.tbl) {
    QConvArgs a = {};
    a.in = in, a.out = out;
    a.C = g.C, a.HI = g.HI, a.WI = g.WI, a.OC = g.OC, a.OH = g.OH, a.OW = g.OW;
    a.KH = g.KH, a.KW = g.KW, a.SH = g.SH, a.SW = g.SW, a.has_bias = g.has_bias;
    a.Cp = (g.C + 7) / 8 * 8;
    a.ksteps = (g.KH * g.KW * a.Cp + 31) / 32;
    a.pitch = qc_pitch(a.ksteps);
    a.ntiles = (g.OC + 7) / 8;
    const int npix = g.OH * g.OW;
    // blocks of a sample: as many as leave every sample a place; more where the rows of one do not fit
    int nc = 8;
    while (nc > 1 && ((long long)B * nc > ctx->sm_count || (nc - 1) * 16 >= npix)) nc /= 2;  // 16 pixels each
    size_t smem = 0;
    bool regs = false;
    for (; nc <= 8; nc *= 2) {
      a.per = (ceil_div(npix, nc) + 15) / 16 * 16;
      const int rows = (a.per + g.OW - 2) / g.OW * g.SH + g.KH;  // a run of `per` pixels needs at most that many
      a.rows = rows < g.HI ? rows : g.HI;
      smem = (size_t)a.ntiles * 8 * a.pitch + (size_t)a.rows * g.WI * a.Cp +
             4 * ((size_t)a.ksteps * 4 + (size_t)a.rows * g.WI + a.per);
      const int groups = (a.ntiles + 3) / 4;
      // a warp's only unit needs no more code than that
      regs = groups <= QC_WARPS && a.per / 16 <= QC_WARPS / groups * QC_UNITS && a.per / 16 * groups > QC_WARPS;
      // once the products are done the results' table and the units on their way out take the place of everything else
      const size_t behind = 32 * 256 * sizeof(float) + (size_t)QC_WARPS * 32 * QC_STAGE * sizeof(int);
      a.copies = regs || smem >= 32 * 256 * sizeof(float) ? 32 : 1;
      const size_t with_acc = smem + (regs ? 0 : 4 * (size_t)g.OC * a.per), with_raw = smem + 16 + 4 * (size_t)g.C * a.rows * g.WI;
      a.acc_smem = with_acc + 4096 <= ctx->smem_optin;  // beside the kernel's own shared variables
      if (a.acc_smem) smem = with_acc;
      // read once where the rows of all blocks make up the planes and the range lies inside a plane
      a.raw = with_raw + 4096 <= ctx->smem_optin && g.SH <= g.KH && g.HI <= g.WI;
      if (a.raw && with_raw > smem) smem = with_raw;
      if (regs && behind > smem) smem = behind;
      if (smem + 4096 <= ctx->smem_optin) break;
    }
    if (nc <= 8) {
      QScratch s;
      B200_TRY(q_carve(ctx, 1, 0, (size_t)a.ntiles * 8 * a.pitch, g.OC, (size_t)a.ntiles * 8, &s));
      unsigned *wsum = reinterpret_cast<unsigned *>(s.acc);
      B200_TRY(launch_kernel(ctx, q_conv_filter_kernel, dim3(a.ntiles * 8), dim3(256), 0, 1, W, g.C, plane,
                             (size_t)g.KH * g.KH, g.C, a.Cp, g.OC, g.KH * g.KW, a.pitch, bias, nbias, s.qg, s.Wq, s.bq,
                             wsum));
      a.Wq = s.Wq, a.bq = s.bq, a.wsum = wsum, a.qg = s.qg;
      auto kernel = regs ? q_conv_fused_kernel<true> : q_conv_fused_kernel<false>;
      B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      B200_TRY(launch_kernel(ctx, kernel, dim3((unsigned)(B * nc)), dim3(QC_THREADS), smem, dim3((unsigned)nc), a));
      return 0;
    }
  }
  // with a connection table, or a filter that does not fit shared memory
  QScratch s;
  B200_TRY(q_carve(ctx, B, in_len, lenW, g.OC, out_len, &s));
  q_input_range_kernel<<<B, 1024, 0, st>>>(in, in_len, g.C, plane, (size_t)g.HI * g.HI, s.qs);
  B200_LAUNCHED();
  q_filter_range_kernel<<<1, 256, 0, st>>>(W, g.C, plane, (size_t)g.KH * g.KH, bias, nbias, s.qg);
  B200_LAUNCHED();
  q_quantize_filter_kernel<<<blocks_for(lenW, 256), 256, 0, st>>>(W, lenW, bias, nbias, s.qg, s.Wq, s.bq);
  B200_LAUNCHED();
  q_sample_params_kernel<<<ceil_div(B, 128), 128, 0, st>>>(s.qs, s.qg, B, 0);
  B200_LAUNCHED();
  q_quantize_input_kernel<<<dim3(blocks_for(in_len, 256), B), 256, 0, st>>>(in, in_len, s.qs, s.inq);
  B200_LAUNCHED();
  q_conv_acc_kernel<<<dim3(blocks_for(out_len, 256), B), 256, 0, st>>>(g, s.inq, s.Wq, s.bq, s.qg, s.qs, s.acc, nullptr);
  B200_LAUNCHED();
  q_requant_params_kernel<<<ceil_div(B, 128), 128, 0, st>>>(s.qs, B);
  B200_LAUNCHED();
  q_requant_dequant_kernel<<<dim3(blocks_for(out_len, 256), B), 256, 0, st>>>(s.acc, out_len, s.qs, out);
  B200_LAUNCHED();
  return 0;
}

// Whether one cluster is the faster form, by its microseconds: a start, the words of four inputs and of the filter that a thread
// quantizes, the samples that a warp requantizes, and how sums are added up (non-negative least squares over 1382 layers of 16 to 2048 inputs, 1 to 256
// outputs and 1 to 512 samples, off by 6 %).  The four launches take 14.3 to 18 us on all of these: 16 inputs, 33 outputs, 128 samples 28.1 us in
// one cluster (of one block) and 14.7 in launches; 1626 -> 16, 116 samples 29.6 and 15; 64 -> 10, one sample 7.5 and 14.7.
static bool q_fc_whole_pays(int klog, int slices, int blocks, int out_size, int B) {
  const int words = 1 << (klog - 2), rows = B < QO_M ? B : QO_M, each = ceil_div(B, QO_WARPS * blocks);
  return 4.3 + 0.85 * ceil_div(rows * words, QO_THREADS) + 0.54 * ceil_div(words * QO_N, QO_THREADS) +
           each * (1.25 + 0.62 * ceil_div(out_size, 32)) + (slices > 1 ? 0.13 * ceil_div(rows * QO_N, QO_THREADS) : 0.0) +
           (blocks > 1 ? 1.3 : 0.0) <
         16.0;
}

int qfc_fwd(b200_ctx *ctx, int in_size, int out_size, const float *in, const float *W,
            const float *bias, float *out, int B) {
  B200_REQUIRE(in_size > 0 && out_size > 0, "quantized fc: non-positive size");
  if (B == 0) return 0;
  const size_t lenW = (size_t)in_size * out_size;
  const int nbias = bias ? out_size : 0;
  // one cluster where the slices and tiles of the layer are few enough: the smallest slices for which that is so
  for (int klog = 5; klog <= 8; ++klog) {
    const long long slices = ceil_div(in_size, 1 << klog), tiles = (long long)ceil_div(out_size, QO_N) * ceil_div(B, QO_M);
    if (slices * tiles > QO_BLOCKS) continue;
    if (!q_fc_whole_pays(klog, (int)slices, (int)(slices * tiles), out_size, B)) break;
    const int blocks = (int)(slices * tiles), parts = (int)slices * (klog > 7 ? 2 : 1);
    QFcArgs a = {};
    a.in = in, a.W = W, a.bias = bias, a.out = out;
    a.B = B, a.in_size = in_size, a.out_size = out_size, a.nbias = nbias;
    a.klog = klog, a.slices = (int)slices, a.ntiles = ceil_div(out_size, QO_N);
    a.vec = in_size % 4 == 0 && ((uintptr_t)in & 15) == 0;
    const size_t o_x = align_up(sizeof(float2) * blocks, 256), o_r = align_up(o_x + sizeof(float2) * parts * B, 256),
                 o_acc = align_up(o_r + sizeof(float2) * B, 256);
    void *base = nullptr;
    B200_TRY(ctx_scratch(ctx, o_acc + sizeof(int) * (size_t)B * out_size, &base));
    char *p = static_cast<char *>(base);
    a.wpart = reinterpret_cast<float2 *>(p);
    a.xpart = reinterpret_cast<float2 *>(p + o_x);
    a.xrange = reinterpret_cast<float2 *>(p + o_r);
    a.acc = reinterpret_cast<int *>(p + o_acc);
    B200_CUDA(cudaFuncSetAttribute(q_fc_whole_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, QO_SMEM));
    return launch_kernel(ctx, q_fc_whole_kernel, dim3((unsigned)blocks), dim3(QO_THREADS), QO_SMEM, dim3((unsigned)blocks), a);
  }
  const int pitch = (in_size + 31) / 32 * 32;  // bytes per quantized row, zero padded
  QScratch s;
  B200_TRY(q_carve(ctx, B, pitch, (size_t)pitch * out_size, out_size, (size_t)out_size + ceil_div(out_size, B), &s));
  unsigned *wsum = reinterpret_cast<unsigned *>(s.acc + (size_t)B * out_size);
  int wblocks = blocks_for(lenW, 4096);
  if (wblocks > Q_PART_BLOCKS) wblocks = Q_PART_BLOCKS;
  B200_TRY(launch_kernel(ctx, q_fc_range_kernel, dim3(B + wblocks), dim3(256), 0, 1, in, in_size, B, W, lenW, out_size, s.qs,
                         s.part, s.acc, wsum));
  const int rblocks = ceil_div(pitch, 1024), fblocks = ceil_div(out_size, 32) * ceil_div(pitch, QF_CIN);
  B200_TRY(launch_kernel(ctx, q_fc_quantize_kernel, dim3(B * rblocks + fblocks), dim3(256), 0, 1, in, in_size, B, pitch,
                         rblocks, W, out_size, bias, nbias, s.part, wblocks, s.qs, s.qg, s.inq, s.Wq, s.bq, wsum));
  // the inputs dealt out so that two blocks an SM have work, 128 bytes at least
  const int tiles = ceil_div(out_size, 64) * ceil_div(B, 64);
  int splits = ceil_div(2 * ctx->sm_count, tiles);
  if (splits > ceil_div(pitch, 128)) splits = ceil_div(pitch, 128);
  const int per = (ceil_div(pitch, splits) + 31) / 32 * 32;
  constexpr int gemm_smem = 128 * (QF_K + 32);
  B200_CUDA(cudaFuncSetAttribute(q_fc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem));
  B200_TRY(launch_kernel(ctx, q_fc_gemm_kernel, dim3(ceil_div(out_size, 64), ceil_div(B, 64), ceil_div(pitch, per)),
                         dim3(256), gemm_smem, 1, B, out_size, pitch, per, s.inq, s.Wq, s.acc));
  B200_TRY(launch_kernel(ctx, q_fc_requant_kernel, dim3(B), dim3(256), 0, 1, in_size, out_size, nbias > 0, s.acc, s.qs, s.qg,
                         wsum, s.bq, out));
  return 0;
}

// tiny_backend::conv2d_eq (backend_tiny.h:115-135): padded rows of uint8 values held in floats
int qconv_eq_fwd(b200_ctx *ctx, const b200_conv_desc *d, const float *in, const float *W, const float *bias,
                 const float *in_r, const float *W_r, const float *b_r, float *out, float *out_r, int B) {
  b200_conv_desc dd = *d;
  dd.input_is_padded = 1;
  ConvGeom g;
  B200_TRY(conv_geom_from_desc(ctx, &dd, &g));
  B200_REQUIRE(g.DH == 1 && g.DW == 1, "quantized convolution has no dilation");
  if (B == 0) return 0;
  const size_t in_len = (size_t)g.HI * g.WI * g.C, out_len = (size_t)g.OC * g.OH * g.OW;
  const size_t lenW = conv_weight_len(g);
  QScratch s;
  B200_TRY(q_carve(ctx, B, in_len, lenW, g.OC, out_len, &s));
  cudaStream_t st = ctx->stream;
  q_eq_params_kernel<<<ceil_div(B, 128), 128, 0, st>>>(s.qs, s.qg, in_r, W_r, b_r, B, 0, g.has_bias);
  B200_LAUNCHED();
  q_cast_u8_kernel<<<blocks_for(in_len * B, 256), 256, 0, st>>>(in, s.inq, in_len * B);
  B200_LAUNCHED();
  q_cast_u8_kernel<<<blocks_for(lenW, 256), 256, 0, st>>>(W, s.Wq, lenW);
  B200_LAUNCHED();
  q_conv_acc_kernel<<<dim3(blocks_for(out_len, 256), B), 256, 0, st>>>(g, s.inq, s.Wq, s.bq, s.qg, s.qs, s.acc,
                                                                      g.has_bias ? bias : nullptr);
  B200_LAUNCHED();
  q_requant_params_kernel<<<ceil_div(B, 128), 128, 0, st>>>(s.qs, B);
  B200_LAUNCHED();
  q_requant_u8_kernel<<<dim3(blocks_for(out_len, 256), B), 256, 0, st>>>(s.acc, out_len, s.qs, out, out_r);
  B200_LAUNCHED();
  return 0;
}

// tiny_backend::fully_eq (backend_tiny.h:321-345)
int qfc_eq_fwd(b200_ctx *ctx, int in_size, int out_size, const float *in, const float *W, const float *bias,
               const float *in_r, const float *W_r, const float *b_r, float *out, float *out_r, int B) {
  if (B == 0) return 0;
  const size_t lenW = (size_t)in_size * out_size;
  QScratch s;
  B200_TRY(q_carve(ctx, B, in_size, lenW, out_size, out_size, &s));
  cudaStream_t st = ctx->stream;
  const int has_bias = bias != nullptr;
  q_eq_params_kernel<<<ceil_div(B, 128), 128, 0, st>>>(s.qs, s.qg, in_r, W_r, b_r, B, 1, has_bias);
  B200_LAUNCHED();
  q_cast_u8_kernel<<<blocks_for((size_t)in_size * B, 256), 256, 0, st>>>(in, s.inq, (size_t)in_size * B);
  B200_LAUNCHED();
  q_cast_u8_kernel<<<blocks_for(lenW, 256), 256, 0, st>>>(W, s.Wq, lenW);
  B200_LAUNCHED();
  if (has_bias) {
    q_cast_u8_kernel<<<blocks_for(out_size, 256), 256, 0, st>>>(bias, s.bq, out_size);
    B200_LAUNCHED();
  }
  q_fc_acc_kernel<<<dim3(blocks_for(out_size, 128), B), 128, 0, st>>>(in_size, out_size, has_bias, s.inq, s.Wq, s.bq,
                                                                     s.qg, s.qs, s.acc);
  B200_LAUNCHED();
  q_requant_params_kernel<<<ceil_div(B, 128), 128, 0, st>>>(s.qs, B);
  B200_LAUNCHED();
  q_requant_u8_kernel<<<dim3(blocks_for(out_size, 256), B), 256, 0, st>>>(s.acc, out_size, s.qs, out, out_r);
  B200_LAUNCHED();
  return 0;
}

}  // namespace b200
