// Fully-connected forward / backward as FP32 tiled GEMMs on the reference's
// row-major [in][out] weight layout (no transposes on the hot path).
//
//   forward  out[B][N]  = in[B][K] * W[K][N] + b      (fully_connected_op_internal.h:15-36)
//   dX       din[B][K]  = dout[B][N] * W[K][N]^T      (:45-50)
//   dW       dW[K][N]  += in[B][K]^T * dout[B][N]     (:52-60)
//   db       db[N]     += column sums of dout         (:62-67)
//
// Large problems use 64x64 tiles.  Small ones (the CIFAR net's 1024->64 and
// 64->10 layers give 4..64 such tiles on 148 SMs) use tiles of 1024 results and split
// the reduction dimension over a cluster of up to eight blocks; each block then
// adds up its share of the tile over the cluster's shared memory, slice after slice,
// so the result does not depend on scheduling.  (With the slices in global memory and
// a second kernel to add them, a 784-500-500-10 step of 77 samples took 13 us more.)
#include <type_traits>

#include "common.cuh"
#include "device_utils.cuh"

namespace b200 {

constexpr int GK = 16;  // tile depth

// four neighbouring results, of which `left` exist: (+)= v (+ bias), then an optional activation; in one store where rows allow
// it (vc).  Four stores of four bytes each took as long as everything else together where the sums are short (4096x4096 from
// 8 samples, dW: 76 us, now 46).
__device__ __forceinline__ void store_row(float *c, int left, float *v, const float *bias, int accumulate, int act, int vc) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < left) {
      if (bias) v[j] += bias[j];
      if (accumulate) v[j] += c[j];
      v[j] = apply_act(v[j], act);
      if (!vc) c[j] = v[j];
    }
  if (vc && left > 0) *reinterpret_cast<float4 *>(c) = make_float4(v[0], v[1], v[2], v[3]);
}

// C[m][n] (+)= sum_k A(m,k) * Bm(k,n) (+ bias[n]), then optional activation.
// A(m,k) = A[m*a_m + k*a_k], Bm(k,n) = Bm[k*b_k + n*b_n], C row-major ldc = N.
// A_KFAST / B_NFAST say which index is contiguous so tile loads coalesce.
template <int BT, int TT, bool A_KFAST, bool B_NFAST>
__global__ void __launch_bounds__(256) sgemm_kernel(int M, int N, int K, const float *__restrict__ A,
                                                    long long a_m, long long a_k,
                                                    const float *__restrict__ Bm, long long b_k,
                                                    long long b_n, float *__restrict__ C,
                                                    const float *__restrict__ bias, int accumulate,
                                                    int act, int vc) {
  after_previous_kernel();
  static_assert(BT / TT == 16 && TT == 4, "256 threads as 16 x 16");
  __shared__ __align__(16) float As[GK][BT + 4];
  __shared__ __align__(16) float Bs[GK][BT + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BT, n0 = blockIdx.x * BT;
  const int tm = (tid / 16) * TT, tn = (tid % 16) * TT;
  float acc[TT][TT];
#pragma unroll
  for (int i = 0; i < TT; ++i)
#pragma unroll
    for (int j = 0; j < TT; ++j) acc[i][j] = 0.f;

  constexpr int PER = BT * GK / 256;  // tile elements per thread
  float ar[PER], br[PER];             // the next tile, on its way while this one is multiplied
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int idx = tid + e * 256;
      const int mm = A_KFAST ? idx / GK : idx % BT, kk = A_KFAST ? idx % GK : idx / BT;
      const int nn = B_NFAST ? idx % BT : idx / GK, kb = B_NFAST ? idx / BT : idx % GK;
      const int m = m0 + mm, n = n0 + nn;
      ar[e] = (m < M && k0 + kk < K) ? A[m * a_m + (k0 + kk) * a_k] : 0.f;
      br[e] = (n < N && k0 + kb < K) ? Bm[(k0 + kb) * b_k + n * b_n] : 0.f;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += GK) {
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int idx = tid + e * 256;
      As[A_KFAST ? idx % GK : idx / BT][A_KFAST ? idx / GK : idx % BT] = ar[e];
      Bs[B_NFAST ? idx / BT : idx % GK][B_NFAST ? idx % BT : idx / GK] = br[e];
    }
    __syncthreads();
    if (k0 + GK < K) fetch(k0 + GK);
    auto products = [&](int kk) {
      float av[TT], bv[TT];
#pragma unroll
      for (int i = 0; i < TT; ++i) {
        av[i] = As[kk][tm + i];
        bv[i] = Bs[kk][tn + i];
      }
#pragma unroll
      for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int j = 0; j < TT; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    };
    const int depth = K - k0;
    if (depth >= GK) {
#pragma unroll
      for (int kk = 0; kk < GK; ++kk) products(kk);
    } else {  // the zeros behind the last k left out (4096x4096 from 8 samples, dW: 46 us with them, now 42 beside dX)
#pragma unroll 4
      for (int kk = 0; kk < depth; ++kk) products(kk);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TT; ++i) {
    const int m = m0 + tm + i;
    if (m >= M) break;
    const size_t ci = (size_t)m * N + n0 + tn;
    store_row(C + ci, N - n0 - tn, acc[i], bias ? bias + n0 + tn : nullptr, accumulate, act, vc);
  }
}

// The same product for the sizes whose 64x64 tiles do not fill the chip.  What bounds such a product is latency: a
// block has a few hundred k's.  So its loads are asked for at once, 16 bytes each where the operand allows it (up to
// four stages of 64 k's; a slice of up to 256 k's pays one trip to memory), in the operand's own layout, and four groups
// of 64 threads share a stage's k's, 4 x 4 outputs a thread: eight 16-byte reads of shared memory for 64
// multiplications.  The groups' sums are added first, then those of the cluster's blocks.
// (784-500-500-10 with 77 samples: the first layer 10.9 us with 16 k's a stage and 2 x 2 outputs a thread, which the loads'
// latency and four 4-byte reads for four multiplications held up, now 7.5; with 4096 hidden units the step of 77 samples went
// from 941 to 449 us, of 8 from 411 to 265; with the tiles of fewer rows, 16-byte stores and longer slices they are 422 and 163.)
struct FcTileArgs {
  int M, N, K, k_per;
  const float *A, *Bm;   // rows are contiguous: A [M][K] (A_KFAST) or [K][M], Bm [K][N] (B_NFAST) or [N][K]
  int lda, ldb, va, vb;  // va, vb: 16-byte copies (rows and first value lie on 16-byte boundaries)
  int vc;                // 16-byte stores, the same of C, C2 and y
  float *C;
  const float *bias;
  int accumulate, act;
  float *col_sum;        // optional (B_NFAST): (+)= the sums of Bm over k, the bias gradient beside dW
  const float *y;        // optional: C2 = C through the gradient of an activation whose output is y
  float *C2;
  int y_act;
  float y_param;
};

constexpr int FT_K = 64, FT_GROUPS = 4;
constexpr int FT_KP = FT_K + 4;                // pitch of a row of k's: eight rows' 16 bytes on different banks
// Tiles of 1024 results: 32 x 32, and 16 x 64 or 8 x 128 for a mini-batch of at most 16 or 8 samples, which would leave the rest of 32
// rows empty: the weights then decide, and a block reads four times as many for the same multiplications.
__host__ __device__ constexpr int ft_cols(int FM) { return 1024 / FM; }
__host__ __device__ constexpr int ft_stages(int FM) { return FM == 8 ? 3 : 4; }
__host__ __device__ constexpr int ft_smem(int FM) { return ft_stages(FM) * (FM + ft_cols(FM)) * FT_KP * 4; }

template <int FM, bool A_KFAST, bool B_NFAST>
__global__ void __launch_bounds__(256) fc_tile_kernel(const __grid_constant__ FcTileArgs a) {
  after_previous_kernel();
  extern __shared__ __align__(16) float fsm[];
  constexpr int FN = ft_cols(FM), XM = FM / 4, XN = FN / 4, ST = ft_stages(FM), OP_A = FM * FT_KP, STAGE = (FM + FN) * FT_KP;
  __shared__ __align__(16) float psum[(FM + 1) * FN];  // the block's sums, and those of Bm
  const int tid = threadIdx.x, group = tid >> 6, tm = (tid & 63) / XN, tn = tid % XN;
  const int m0 = blockIdx.y * FM, n0 = blockIdx.x * FN;
  const int kbeg = blockIdx.z * a.k_per, kend = min(a.K, kbeg + a.k_per);
  const int nst = (kend - kbeg + FT_K - 1) / FT_K;
  // T rows of 64 k's, or 64 k rows of T values; outside the matrix and the slice zero
  auto load = [&](auto tile, float *dst, const float *src, int ld, bool kfast, int r0, int rows, int k0, int vec) {
    constexpr int T = decltype(tile)::value;
    if (vec) {
#pragma unroll
      for (int e = 0; e < (T * FT_K / 4 + 255) / 256; ++e) {
        const int p = tid + e * 256, r = kfast ? p / (FT_K / 4) : p % (T / 4) * 4, k = kfast ? p % (FT_K / 4) * 4 : p / (T / 4);
        if (T * FT_K / 4 < 256 && p >= T * FT_K / 4) break;
        const bool ok = r0 + r < rows && k0 + k < kend;
        const size_t at = kfast ? (size_t)(r0 + r) * ld + k0 + k : (size_t)(k0 + k) * ld + r0 + r;
        cp_async16(dst + (kfast ? r * FT_KP + k : k * T + r), src + (ok ? at : 0), ok);
      }
    } else {
#pragma unroll 4
      for (int e = 0; e < T * FT_K / 256; ++e) {
        const int p = tid + e * 256, r = kfast ? p / FT_K : p % T, k = kfast ? p % FT_K : p / T;
        const bool ok = r0 + r < rows && k0 + k < kend;
        const size_t at = kfast ? (size_t)(r0 + r) * ld + k0 + k : (size_t)(k0 + k) * ld + r0 + r;
        cp_async4(dst + (kfast ? r * FT_KP + k : k * T + r), src + (ok ? at : 0), ok);
      }
    }
  };
  auto fetch = [&](int i) {
    if (i < nst) {
      float *d = fsm + (i % ST) * STAGE;
      load(std::integral_constant<int, FM>(), d, a.A, a.lda, A_KFAST, m0, a.M, kbeg + i * FT_K, a.va);
      load(std::integral_constant<int, FN>(), d + OP_A, a.Bm, a.ldb, !B_NFAST, n0, a.N, kbeg + i * FT_K, a.vb);
    }
    cp_async_commit();
  };
  const bool sums = B_NFAST && a.col_sum && blockIdx.y == 0;
  float acc[4][4], cs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int i = 0; i < ST - 1; ++i) fetch(i);
  for (int st = 0; st < nst; ++st) {
    fetch(st + ST - 1);  // into the stage that was read before the last barrier
    cp_async_wait<ST - 1>();
    __syncthreads();
    const float *as = fsm + (st % ST) * STAGE, *bs = as + OP_A;
    // rows of k's: a thread's four are XM or XN apart, so that a warp's rows are neighbours; k rows: four values side by side
#pragma unroll
    for (int kk = 0; kk < FT_K / FT_GROUPS; kk += 4) {
      const int k = group * (FT_K / FT_GROUPS) + kk;
      float av[4][4], bv[4][4];  // [k][row]
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = *reinterpret_cast<const float4 *>(A_KFAST ? as + (i * XM + tm) * FT_KP + k : as + (k + i) * FM + tm * 4);
        const float4 z = *reinterpret_cast<const float4 *>(B_NFAST ? bs + (k + i) * FN + tn * 4 : bs + (i * XN + tn) * FT_KP + k);
        const float xv[4] = {x.x, x.y, x.z, x.w}, zv[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (A_KFAST) av[j][i] = xv[j];
          else av[i][j] = xv[j];
          if (B_NFAST) bv[i][j] = zv[j];
          else bv[j][i] = zv[j];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[q][i], bv[q][j], acc[i][j]);
      if (B_NFAST && sums)
#pragma unroll
        for (int j = 0; j < 4; ++j) cs[j] += (bv[0][j] + bv[1][j]) + (bv[2][j] + bv[3][j]);
    }
    __syncthreads();
  }
  // the groups' sums, in the stages' place: [group][row][FN], row FM the sums of Bm
  cp_async_wait<0>();
  float *part = fsm + group * (FM + 1) * FN;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = A_KFAST ? i * XM + tm : tm * 4 + i;
    if (B_NFAST)
      *reinterpret_cast<float4 *>(part + m * FN + tn * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    else
#pragma unroll
      for (int j = 0; j < 4; ++j) part[m * FN + j * XN + tn] = acc[i][j];
  }
  if (B_NFAST && sums && tm == 0) *reinterpret_cast<float4 *>(part + FM * FN + tn * 4) = make_float4(cs[0], cs[1], cs[2], cs[3]);
  __syncthreads();
  const int quads = (FM * FN + (sums ? FN : 0)) / 4;
  for (int e = tid; e < quads; e += 256) {
    float4 v = reinterpret_cast<const float4 *>(fsm)[e];
#pragma unroll
    for (int g = 1; g < FT_GROUPS; ++g) {
      const float4 w = reinterpret_cast<const float4 *>(fsm + g * (FM + 1) * FN)[e];
      v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
    }
    reinterpret_cast<float4 *>(psum)[e] = v;
  }
  const int Z = gridDim.z;
  if (Z == 1)
    __syncthreads();
  else
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
  const uint32_t at = smem_u32(psum);
  const int share = (quads + Z - 1) / Z, last = min(quads, ((int)blockIdx.z + 1) * share);
  for (int e = blockIdx.z * share + tid; e < last; e += 256) {
    float v[8][4];
#pragma unroll
    for (int z = 0; z < 8; ++z)
      if (z < Z) {
        uint32_t ra = at + 16u * e;
        if (Z > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(at + 16u * e), "r"(z));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                     : "=f"(v[z][0]), "=f"(v[z][1]), "=f"(v[z][2]), "=f"(v[z][3])
                     : "r"(ra)
                     : "memory");
      }
#pragma unroll
    for (int z = 1; z < 8; ++z)
      if (z < Z)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[0][j] += v[z][j];
    const int m = m0 + e / XN, n = n0 + e % XN * 4;
    if (e >= FM * FN / 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < a.N) a.col_sum[n + j] = a.accumulate ? a.col_sum[n + j] + v[0][j] : v[0][j];
      continue;
    }
    if (m >= a.M) continue;
    const size_t ci = (size_t)m * a.N + n;
    store_row(a.C + ci, a.N - n, v[0], a.bias ? a.bias + n : nullptr, a.accumulate, a.act, a.vc);
    if (a.C2) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[0][j] = n + j < a.N ? act_grad(a.y_act, a.y_param, a.y[ci + j], v[0][j]) : 0.f;
      store_row(a.C2 + ci, a.N - n, v[0], nullptr, 0, B200_ACT_NONE, a.vc);
    }
  }
  if (Z > 1) asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}

// db[i] (+)= sum_n dout[n*N + i].  A block sums 128 columns, a warp of it every eighth row, four values of a row a lane; from 128
// rows on the blocks of a cluster share the rows out.  All sums are added in a fixed order.  (4096 columns of 1024 rows: 13.5 us
// with 32 columns a block, whose pieces of 128 bytes and chains of 128 rows held it up, 8.4 now.)
constexpr int CS_COLS = 128;
__global__ void __launch_bounds__(256) col_sum_kernel(const float *__restrict__ d, float *__restrict__ db, int rows, int N,
                                                      int accumulate) {
  after_previous_kernel();
  __shared__ float part[8][CS_COLS];
  const int Z = gridDim.y, rank = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = blockIdx.x * CS_COLS;
  float s[4] = {};
  const float *from[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) from[j] = d + min(c0 + lane + 32 * j, N - 1);
#pragma unroll 8
  for (int r = rank * 8 + warp; r < rows; r += 8 * Z)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] += from[j][(size_t)r * N];
#pragma unroll
  for (int j = 0; j < 4; ++j) part[warp][lane + 32 * j] = s[j];
  __syncthreads();
  const int c = threadIdx.x;
  float t = 0.f;
  if (c < CS_COLS) {
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w][c];
    part[0][c] = t;
  }
  if (Z > 1) {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
    if (c < CS_COLS && c * Z / CS_COLS == rank) {
      const unsigned at = smem_u32(&part[0][c]);
      t = 0.f;
      for (int z = 0; z < Z; ++z) {
        float v;
        unsigned remote;
        asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(at), "r"(z));
        asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(remote) : "memory");
        t += v;
      }
    }
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
  }
  if (c < CS_COLS && c * Z / CS_COLS == rank && c0 + c < N) db[c0 + c] = accumulate ? db[c0 + c] + t : t;
}

// Plan of one GEMM: tile and k slices.
struct GemmPlan {
  int tile;    // rows of a tile: 64 (of 64 x 64), or 32, 16 or 8 of fc_tile_kernel's
  int slices;  // >= 1
  int k_per;
};

static GemmPlan plan_gemm(const b200_ctx *ctx, int M, int N, int K) {
  GemmPlan p;
  long long t64 = (long long)ceil_div(M, 64) * ceil_div(N, 64);
  if (t64 >= ctx->sm_count && M > 16) {
    p.tile = 64;
    p.slices = 1;
    p.k_per = K > 0 ? K : 1;
    return p;
  }
  p.tile = M <= 8 && N >= 128 ? 8 : M <= 16 && N >= 64 ? 16 : 32;
  const long long tiles = (long long)ceil_div(M, p.tile) * ceil_div(N, ft_cols(p.tile));
  int want = (int)((2LL * ctx->sm_count + tiles - 1) / tiles);  // fill the machine twice
  if (want > 8) want = 8;                                       // what a cluster may have anywhere
  // at least 64 of k per slice, 128 where the tiles are one for every SM already (500x500, 77 samples, dW: two slices 9.9 us)
  int max_by_k = ceil_div(K > 0 ? K : 1, tiles >= ctx->sm_count ? 128 : 64);
  int s = want < max_by_k ? want : max_by_k;
  if (s < 1) s = 1;
  int k_per = ceil_div(ceil_div(K > 0 ? K : 1, s), GK) * GK;  // whole 16-byte pieces of a row
  p.k_per = k_per;
  p.slices = ceil_div(K > 0 ? K : 1, k_per);
  return p;
}

static bool tc_can(int M, int N, int K) { return M >= 128 && N >= 64 && K >= 32; }  // one full tile in every direction

// A GEMM goes to the tensor cores when the context allows it and it is big enough
// to pay for splitting its operands.
static bool use_tc(const b200_ctx *ctx, int M, int N, int K) {
  if (ctx->fc_tensor_cores == 0 || !tc_can(M, N, K)) return false;
  if (ctx->fc_tensor_cores >= 2) return true;
  return (long long)M * N * K >= (1LL << 26);
}

// Scratch of a layer's products on the tensor cores: of those that go there now, or (`any`) under any option, for a
// network, whose scratch outlives a change of the option.
size_t fc_scratch_floats(const b200_ctx *ctx, int in_size, int out_size, int B, bool any) {
  const int p[4][3] = {{B, out_size, in_size}, {B, in_size, out_size}, {in_size, out_size, B}, {out_size, in_size, B}};
  size_t need = 0;
  for (const int *e : p)
    if (any ? tc_can(e[0], e[1], e[2]) : use_tc(ctx, e[0], e[1], e[2])) need = max(need, gemm_tc_scratch_floats(e[0], e[1], e[2]));
  return need;
}

// Product with operands in contiguous rows: A [M][K] (A_KFAST) or [K][M], Bm [K][N] (B_NFAST) or [N][K].  `col_sum` and `ag` (see
// FcTileArgs) are taken by the small tiles alone: they are asked for where plan_gemm gives those.
template <bool A_KFAST, bool B_NFAST>
static int run_gemm(b200_ctx *ctx, int M, int N, int K, const float *A, const float *Bm, float *C, const float *bias, int accumulate,
                    int act, float *col_sum = nullptr, const FcActGrad *ag = nullptr) {
  if (M == 0 || N == 0) return 0;
  const GemmPlan p = plan_gemm(ctx, M, N, K);
  const int lda = A_KFAST ? K : M, ldb = B_NFAST ? N : K;
  const auto aligned = [](const void *q) { return ((uintptr_t)q & 15) == 0; };
  if (p.tile == 64) {
    const dim3 grid(ceil_div(N, 64), ceil_div(M, 64));
    return launch_kernel(ctx, sgemm_kernel<64, 4, A_KFAST, B_NFAST>, grid, dim3(256), 0, dim3(1), M, N, K, A, A_KFAST ? lda : 1,
                         A_KFAST ? 1 : lda, Bm, B_NFAST ? ldb : 1, B_NFAST ? 1 : ldb, C, bias, accumulate, act,
                         N % 4 == 0 && aligned(C));
  }
  FcTileArgs a = {};
  a.M = M, a.N = N, a.K = K, a.k_per = p.k_per;
  a.A = A, a.Bm = Bm, a.lda = lda, a.ldb = ldb;
  a.va = lda % 4 == 0 && aligned(A);
  a.vb = ldb % 4 == 0 && aligned(Bm);
  a.vc = N % 4 == 0 && aligned(C) && (!ag || (aligned(ag->dst) && aligned(ag->y)));
  a.C = C, a.bias = bias, a.accumulate = accumulate, a.act = act;
  a.col_sum = col_sum;
  if (ag) a.y = ag->y, a.C2 = ag->dst, a.y_act = ag->act, a.y_param = ag->param;
  auto run = [&](auto rows) -> int {
    constexpr int FM = decltype(rows)::value;
    B200_CUDA(cudaFuncSetAttribute(fc_tile_kernel<FM, A_KFAST, B_NFAST>, cudaFuncAttributeMaxDynamicSharedMemorySize, ft_smem(FM)));
    return launch_kernel(ctx, fc_tile_kernel<FM, A_KFAST, B_NFAST>, dim3(ceil_div(N, ft_cols(FM)), ceil_div(M, FM), p.slices),
                         dim3(256), ft_smem(FM), dim3(1, 1, p.slices), a);
  };
  if (p.tile == 8) return run(std::integral_constant<int, 8>());
  if (p.tile == 16) return run(std::integral_constant<int, 16>());
  return run(std::integral_constant<int, 32>());
}

// whether the product of a pass (0 forward, 1 dX, 2 dW) runs on the tensor cores
bool fc_pass_tc(const b200_ctx *ctx, int in_size, int out_size, int B, int pass, bool w_rows) {
  return pass == 0   ? use_tc(ctx, B, out_size, in_size)
         : pass == 1 ? use_tc(ctx, B, in_size, out_size)
                     : use_tc(ctx, w_rows ? out_size : in_size, w_rows ? in_size : out_size, B);
}

bool fc_any_tc(const b200_ctx *ctx, int in_size, int out_size, int B) {
  return use_tc(ctx, B, out_size, in_size) || use_tc(ctx, B, in_size, out_size) || use_tc(ctx, in_size, out_size, B) ||
         use_tc(ctx, out_size, in_size, B);
}

int fc_split(b200_ctx *ctx, int in_size, int out_size, const float *in, const float *W, const float *dout, int B, FcPlanes *p,
             bool grad) {
  const bool fwd = use_tc(ctx, B, out_size, in_size), dx = use_tc(ctx, B, in_size, out_size), dw = use_tc(ctx, in_size, out_size, B);
  if (!grad) {
    p->x_ready = p->x && (fwd || dw);
    p->w_ready = p->w && (fwd || dx);
    if (p->x_ready) B200_TRY(gemm_tc_split(ctx, in, B, in_size, p->x));
    if (p->w_ready) B200_TRY(gemm_tc_split(ctx, W, in_size, out_size, p->w));
  } else if (p->d && (dx || dw)) {
    B200_TRY(gemm_tc_split(ctx, dout, B, out_size, p->d));
    p->d_ready = true;
  }
  return 0;
}

static GemmOperand operand(const float *src, const void *planes, bool ready) { return {src, ready ? planes : nullptr}; }

// `w_rows`: the weights are stored [out][in] (a convolution whose window is the whole input), not [in][out]; such a
// layer keeps no `planes`
int fc_fwd(b200_ctx *ctx, int in_size, int out_size, const float *in, const float *W,
           const float *bias, float *out, int B, int act, float *scratch, bool w_rows, const FcPlanes *planes) {
  const FcPlanes p = planes ? *planes : FcPlanes();
  if (scratch && use_tc(ctx, B, out_size, in_size))
    // A = in [B][in]; Bt = W^T: W is [in][out], i.e. K x N
    return gemm_tc(ctx, B, out_size, in_size, operand(in, p.x, p.x_ready), false, operand(W, p.w, p.w_ready), !w_rows, out, bias,
                   0, act, scratch);
  // M = B, N = out, K = in; A = in (k fast), Bm(k, n) = W[k][n] (n fast) or W[n][k] (k fast)
  if (w_rows) return run_gemm<true, false>(ctx, B, out_size, in_size, in, W, out, bias, 0, act);
  return run_gemm<true, true>(ctx, B, out_size, in_size, in, W, out, bias, 0, act);
}

// whether the dX pass can also form the gradient through an activation in front of the layer
bool fc_dx_takes_act(const b200_ctx *ctx, int in_size, int out_size, int B, bool scratch) {
  return !(scratch && use_tc(ctx, B, in_size, out_size)) && plan_gemm(ctx, B, in_size, out_size).tile != 64;
}

int fc_bwd(b200_ctx *ctx, int in_size, int out_size, const float *in, const float *W,
           const float *dout, float *din, float *dW, float *db, int accumulate, int B,
           float *scratch, bool w_rows, const FcPlanes *planes, const FcActGrad *ag) {
  const FcPlanes p = planes ? *planes : FcPlanes();
  if (din && scratch && use_tc(ctx, B, in_size, out_size)) {
    // din[B][in] = dout[B][out] * W^T: A = dout; Bt[n = c][k = o] = W[c*out + o] as stored
    B200_TRY(gemm_tc(ctx, B, in_size, out_size, operand(dout, p.d, p.d_ready), false, operand(W, p.w, p.w_ready), w_rows, din,
                     nullptr, 0, 0, scratch));
  } else if (din && w_rows) {
    B200_TRY((run_gemm<true, true>(ctx, B, in_size, out_size, dout, W, din, nullptr, 0, 0, nullptr, ag)));
  } else if (din) {
    // din[B][in] = dout[B][out] * W^T : M = B, N = in, K = out; Bm(k = o, n = c) = W[c*out + o] (k fast)
    B200_TRY((run_gemm<true, false>(ctx, B, in_size, out_size, dout, W, din, nullptr, 0, 0, nullptr, ag)));
  }
  bool db_done = false;
  if (dW) {
    // dW[in][out] (+)= in^T * dout, or dW[out][in] (+)= dout^T * in
    const float *l = w_rows ? dout : in, *r = w_rows ? in : dout;
    const int M = w_rows ? out_size : in_size, N = w_rows ? in_size : out_size;
    if (scratch && use_tc(ctx, M, N, B))
      B200_TRY(gemm_tc(ctx, M, N, B, operand(l, p.x, p.x_ready && !w_rows), true, operand(r, p.d, p.d_ready && !w_rows), true, dW,
                       nullptr, accumulate, 0, scratch));
    else {
      // A(m, k = n) = l[n*M + m] (m fast); the bias gradient is the sum of the right operand over k
      db_done = db && !w_rows && plan_gemm(ctx, M, N, B).tile != 64;
      B200_TRY((run_gemm<false, true>(ctx, M, N, B, l, r, dW, nullptr, accumulate, 0, db_done ? db : nullptr)));
    }
  }
  if (db && !db_done) {
    const int blocks = B >= 512 ? 8 : B >= 256 ? 4 : B >= 128 ? 2 : 1;
    B200_TRY(launch_kernel(ctx, col_sum_kernel, dim3(ceil_div(out_size, CS_COLS), blocks), dim3(256), 0, dim3(1, blocks), dout, db, B,
                           out_size, accumulate));
  }
  return 0;
}

}  // namespace b200
