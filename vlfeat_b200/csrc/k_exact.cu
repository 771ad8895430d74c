// Exact-arithmetic kernels (CUDA cores, float or double).  These evaluate the
// reference's own formulation -- sum_d (x-mu)^2 / sigma^2 per (descriptor,
// component), thresholded statistics, etc. -- and serve VL_TYPE_DOUBLE calls,
// the EXACT precision mode and the M-step / restart machinery of EM.
//
// Determinism: every reduction runs in a fixed order (per-block partials,
// then a fixed-shape final reduction), so results are bitwise reproducible
// run to run, unlike the reference's OpenMP critical-section merge
// (vl/gmm.c:1152-1166).
#include <cmath>
#include <cstring>
#include <type_traits>

#include <cooperative_groups.h>

#include "engine.h"
#include "exact_math.cuh"
#include "ordered_sum.cuh"
#include "seq_sum.cuh"
#include "tc_common.cuh"

namespace vlb {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float dexp(float x) { return expf(x); }
__device__ __forceinline__ double dexp(double x) { return exp(x); }

// Asynchronous global -> shared copies (16, 8 or 4 bytes; bytes past srcBytes
// are zero-filled and nothing is read for them).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t srcBytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(srcBytes) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src, uint32_t srcBytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(srcBytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, uint32_t srcBytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(srcBytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// Elements [0, n) of a row of width w (n <= w) to shared memory, the rest
// zeros, in pieces of VB bytes; w and the addresses suit VB.
template <int VB, typename T>
__device__ __forceinline__ void cp_async_piece(uint32_t dst, const T *src, bool in) {
  if constexpr (VB == 16) cp_async16(dst, src, in ? 16u : 0u);
  else if constexpr (VB == 8) cp_async8(dst, src, in ? 8u : 0u);
  else cp_async4(dst, src, in ? 4u : 0u);
}

// ------------------------------------------------------------ model image
// The E-step streams the means and inverse variances through shared memory
// in chunks of es_dc dimensions.  The image holds them in the order its lanes
// read: components in blocks of 32 NJ (component 32 j + l of a block belongs
// to lane l), per block, dimension, pair of components (j, j + 1) and lane
// [-mu_j, -mu_j+1, 1/s2_j, 1/s2_j+1].  Padding has mean 0 and variance 1: the
// rows' padded dimensions are zeros, so those add nothing to a distance, and a
// padded component's distance stays a number (or infinity, where a row's squares
// overflow), so that with its constant -inf its logit is -inf.  An inverse
// variance of 0 there turned infinity into NaN, which the row's sum of
// exponentials kept.
template <typename T>
__host__ __device__ constexpr int es_dc() { return 64 / (int)sizeof(T); }  // dimensions per chunk
// Pairs of components per lane (NJ / 2) for K components: the smallest block
// that holds them, up to 256; above that the block size that pads least
// (the larger one on a tie).
__host__ __device__ inline int es_half_nj(i64 K) {
  for (int h = 1; h <= 4; ++h)
    if (K <= 64 * h) return h;
  int best = 4;
  i64 pad = (K + 255) / 256 * 256;
  for (int h = 3; h >= 2; --h) {
    const i64 p = (K + 64 * h - 1) / (64 * h) * (64 * h);
    if (p < pad) {
      pad = p;
      best = h;
    }
  }
  return best;
}
__host__ __device__ inline i64 es_blocks(i64 K) {
  const int kb = 64 * es_half_nj(K);
  return (K + kb - 1) / kb;
}
template <typename T>
__host__ __device__ inline i64 es_dpad(i64 D) { return (D + es_dc<T>() - 1) / es_dc<T>() * es_dc<T>(); }

// ------------------------------------------------------------ prepare
// Per-component constants, vl/gmm.c:741-756 and vl/fisher.c:386-390, and the
// E-step's image.  One warp per (padded) component, lanes over dimensions;
// the sum of the logarithms runs over the dimensions in order (a shuffle per
// term, the logarithms themselves formed 32 at a time).  Bound by latency: 10 us
// a launch at K = 256, D = 80, where one thread per component took 39.
template <typename T>
__global__ void k_prepare(const T *__restrict__ priors, const T *__restrict__ means, const T *__restrict__ covs,
                          int K, int D, T halfDimLog2Pi, T *__restrict__ inv, double *__restrict__ cst,
                          T *__restrict__ sis, T *__restrict__ img) {
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
  const int h = es_half_nj(K), kb = 64 * h;
  const int Dp = (int)es_dpad<T>(D);
  if (img) {
    if (k >= (int)es_blocks(K) * kb) return;
    const int j = (k % kb) / 32;
    T *o = img + ((i64)(k / kb) * Dp * h + j / 2) * 128 + (k % 32) * 4 + (j & 1);
    for (int d = lane; d < Dp; d += 32) {
      const bool in = k < K && d < D;
      o[(i64)d * h * 128] = in ? -means[(i64)k * D + d] : (T)0;
      o[(i64)d * h * 128 + 2] = in ? (T)1 / covs[(i64)k * D + d] : (T)1;
    }
  }
  if (k >= K) return;
  T acc = 0;
  for (int d0 = 0; d0 < D; d0 += 32) {
    const int d = d0 + lane;
    T lg = 0;
    if (d < D) {
      const T c = covs[(i64)k * D + d];
      lg = (T)log((double)c);
      if (inv) inv[(i64)k * D + d] = (T)1 / c;
      sis[(i64)k * D + d] = (T)sqrt(1.0 / (double)c);
    }
    const int n = min(32, D - d0);
    for (int l = 0; l < n; ++l) acc += __shfl_sync(0xffffffffu, lg, l);
  }
  if (lane == 0) {
    const T logw = ((double)priors[k] < 1e-6) ? (T)(-INFINITY) : (T)log((double)priors[k]);
    cst[k] = (double)(T)(logw - halfDimLog2Pi) - 0.5 * (double)acc;
  }
}

// ------------------------------------------------------------ E-step
// Log-densities c_k - 1/2 sum_d (x - mu)^2 / sigma^2 and, with NORM, the
// row-wise log-sum-exp normalisation (vl/gmm.c:741-790) and the optional FAST
// one-hot (vl/fisher.c:398-417: first arg-max wins) in one pass over X, the
// posteriors written once.
//
// A warp owns R rows and the block's NJ * 32 components: lane l holds
// components l, l + 32, ..., so a row's reductions stay inside the warp and
// run in the order of a warp striding over the row.  Per (row, component) the
// sum runs over the dimensions in ascending order: (x - mu), its square, and
// the fused square * iv + acc, in packed pairs of components for float.
//
// Bound: the float version issues 3 lane operations per (row, component,
// dimension) and the FMA pipes take 128 a clock and SM, packed or not
// (measured: 123), so R x NJ = 64 accumulators per lane keep the operand loads
// (NJ / 2 16-byte loads per dimension, R broadcast 8-byte loads per two) at
// under half of the shared-memory bandwidth.  Model and row chunks are copied
// asynchronously, two chunks ahead in three stages; two blocks of 64 rows share an SM, so
// that one block's exponentials and divisions run beside the other's sums.
// A packed instruction holds the issue port for two clocks, so the sum of all
// instructions' issue clocks bounds the kernel: 3 x 80 of about 117 a row and
// warp for the sums at D = 80, K = 256, the rest the exponentials, divisions
// and conversions.  1.04 M rows, K = 256, D = 80: 2.86 ms (1.72 at the pipes'
// rate); two kernels with the logits in memory between them took 2.94 + 0.73.
// 100,000 rows, K = 64, D = 64: 0.086 ms against 0.070 + 0.054.
// K above 256 (NORM false): one block per (rows, component block) writes the
// logits and k_normalize finishes the rows.
template <typename T, int NJ, int R>
struct EsLayout {
  static constexpr int DC = es_dc<T>();
  static constexpr int kStages = 3;
  static constexpr int kModel = NJ * 32 * DC * 2;  // elements of a model chunk
  static constexpr size_t bytes(int warps) {
    return sizeof(T) * (size_t)kStages * (kModel + (size_t)warps * R * DC);
  }
};

template <typename T, int NJ, int R, bool NORM, int VB>
__global__ void __launch_bounds__(kThreads, 2) k_estep(const T *__restrict__ X, i64 N, int D, int K,
                                                       const T *__restrict__ img, const double *__restrict__ cst,
                                                       T *__restrict__ q, int fast, double *__restrict__ ll_part) {
  using L = EsLayout<T, NJ, R>;
  constexpr int DC = L::DC, H = NJ / 2, NST = L::kStages;
  constexpr int VE = VB / (int)sizeof(T);  // elements per copied piece of a row
  extern __shared__ __align__(16) unsigned char es_smem[];
  T *sm = (T *)es_smem;                  // [stage][DC][H][32][4]
  T *sx = sm + NST * L::kModel;          // [stage][row][DC]
  const int tid = threadIdx.x, w = tid / 32, lane = tid % 32, nthr = blockDim.x;
  const int rows = nthr / 32 * R;
  const i64 i0 = (i64)blockIdx.x * rows;
  const int nch = (D + DC - 1) / DC;
  img += (i64)blockIdx.y * nch * L::kModel;
  const int kbase = blockIdx.y * NJ * 32;

  auto issue = [&](int c) {
    if (c < nch) {
      const int st = c % NST;
      const T *ms = img + (i64)c * L::kModel;
      T *md = sm + st * L::kModel;
      for (int e = tid; e < L::kModel * (int)sizeof(T) / 16; e += nthr)
        cp_async16(tc::smem_u32((char *)md + 16 * e), (const char *)ms + 16 * e, 16u);
      T *xd = sx + st * rows * DC;
      const int d0 = c * DC;
      for (int e = tid; e < rows * (DC / VE); e += nthr) {
        const int r = e / (DC / VE), v = (e % (DC / VE)) * VE;
        const i64 i = i0 + r;
        const bool in = i < N && d0 + v < D;
        cp_async_piece<VB>(tc::smem_u32(xd + r * DC + v), in ? X + i * D + d0 + v : X, in);
      }
    }
    cp_async_commit();
  };
  issue(0);
  issue(1);

  unsigned long long acc[R][sizeof(T) == 4 ? H : NJ];  // float: packed pairs; double: values
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < (sizeof(T) == 4 ? H : NJ); ++j) acc[r][j] = 0ull;

  for (int c = 0; c < nch; ++c) {
    cp_async_wait<1>();
    __syncthreads();  // chunk c has landed; every warp is done with chunk c - 1's stage
    issue(c + 2);
    const T *mc = sm + (c % NST) * L::kModel + lane * 4;
    const T *xc = sx + (c % NST) * rows * DC + w * R * DC;
    const int dl = min(DC, D - c * DC);
#pragma unroll 1
    for (int dd = 0; dd < dl; dd += 2) {  // an odd last dimension meets a zero one
      if constexpr (sizeof(T) == 4) {
        float2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = *(const float2 *)(xc + r * DC + dd);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int h = 0; h < H; ++h) {
            const ulonglong2 m = *(const ulonglong2 *)(mc + ((dd + e) * H + h) * 128);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const float xv = e ? x[r].y : x[r].x;
              const unsigned long long df = tc::add2(tc::f2u(xv, xv), m.x);
              acc[r][h] = tc::fma2(tc::mul2(df, df), m.y, acc[r][h]);
            }
          }
      } else {
        double2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = *(const double2 *)(xc + r * DC + dd);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int h = 0; h < H; ++h) {
            const double2 mu = *(const double2 *)(mc + ((dd + e) * H + h) * 128);
            const double2 iv = *(const double2 *)(mc + ((dd + e) * H + h) * 128 + 2);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const double xv = e ? x[r].y : x[r].x;
              const double d0 = xv + mu.x, d1 = xv + mu.y;
              acc[r][2 * h] = (unsigned long long)__double_as_longlong(
                  fma(d0 * d0, iv.x, __longlong_as_double((long long)acc[r][2 * h])));
              acc[r][2 * h + 1] = (unsigned long long)__double_as_longlong(
                  fma(d1 * d1, iv.y, __longlong_as_double((long long)acc[r][2 * h + 1])));
            }
          }
      }
    }
  }
  cp_async_wait<0>();

  // ------------------------------------------------------- epilogue
  double ck[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int k = kbase + lane + 32 * j;
    ck[j] = k < K ? cst[k] : -INFINITY;
  }
  const i64 row0 = i0 + w * R;
  constexpr int G = R < 8 ? R : 8;  // rows per log-likelihood partial
  // The logits take the accumulators' place; each reduction step runs over all
  // of the warp's rows, so that their shuffles are in flight together.
  auto get = [&](int r, int j) -> T {
    if constexpr (sizeof(T) == 4) return j & 1 ? tc::hi32(acc[r][j / 2]) : tc::lo32(acc[r][j / 2]);
    else return __longlong_as_double((long long)acc[r][j]);
  };
  auto put = [&](int r, int j, T v) {
    if constexpr (sizeof(T) == 4) acc[r][j / 2] = j & 1 ? tc::f2u(tc::lo32(acc[r][j / 2]), v) : tc::f2u(v, tc::hi32(acc[r][j / 2]));
    else acc[r][j] = (unsigned long long)__double_as_longlong(v);
  };
  T mx[R], sum[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    mx[r] = (T)(-INFINITY);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const T v = (T)(ck[j] - 0.5 * (double)get(r, j));
      put(r, j, v);
      mx[r] = max(mx[r], v);
    }
  }
  if constexpr (!NORM) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      T *row = q + (row0 + r) * K + kbase;
      if (row0 + r < N) {
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          if (kbase + lane + 32 * j < K) row[lane + 32 * j] = get(r, j);
      }
    }
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) mx[r] = max(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], o));
#pragma unroll
    for (int r = 0; r < R; ++r) {
      sum[r] = 0;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const T e = dexp(get(r, j) - mx[r]);
        put(r, j, e);
        sum[r] += e;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
    T rsum = 1, rmax = 0;  // lane r: row r's sum of exponentials and maximum
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (lane == r) {
        rsum = sum[r];
        rmax = mx[r];
      }
      T *row = q + (row0 + r) * K;
#pragma unroll
      for (int j = 0; j < NJ; ++j) put(r, j, get(r, j) / sum[r]);
      if (fast) {
        T bv = (T)(-INFINITY);
        int bi = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          if (get(r, j) > bv && lane + 32 * j < K) {
            bv = get(r, j);
            bi = lane + 32 * j;
          }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const T ov = __shfl_xor_sync(0xffffffffu, bv, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (bi == 0x7fffffff) bi = 0;  // all-NaN row: the reference keeps index 0
#pragma unroll
        for (int j = 0; j < NJ; ++j) put(r, j, (T)(lane + 32 * j == bi));
      }
      if (row0 + r < N) {
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          if (lane + 32 * j < K) row[lane + 32 * j] = get(r, j);
      }
    }
    if (ll_part) {
      // Log-likelihood partials of G rows, added in row order.
      const double lr = (lane < R && row0 + lane < N) ? log((double)rsum) + (double)rmax : 0.0;
#pragma unroll
      for (int g = 0; g < R; g += G) {
        double t = 0;
#pragma unroll
        for (int j = 0; j < G; ++j) t += __shfl_sync(0xffffffffu, lr, g + j);
        if (lane == 0 && row0 + g < N) ll_part[(row0 + g) / G] = t;
      }
    }
  }
}

int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    VLB_CUDA(cudaGetDevice(&dev));
    VLB_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v;
  }();
  return n;
}

template <typename T, int NJ, int R, bool NORM>
void launch_estep_as(const T *X, i64 N, i64 D, i64 K, const T *img, const double *cst, T *q, bool fast,
                     double *ll_part, int warps, bool vec, cudaStream_t s) {
  auto kern = vec ? k_estep<T, NJ, R, NORM, 16> : k_estep<T, NJ, R, NORM, (int)sizeof(T)>;
  const size_t smem = EsLayout<T, NJ, R>::bytes(warps);
  VLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 g((unsigned)((N + warps * R - 1) / (warps * R)), NORM ? 1u : (unsigned)es_blocks(K));
  kern<<<g, warps * 32, smem, s>>>(X, N, (int)D, (int)K, img, cst, q, fast ? 1 : 0, ll_part);
}

// Launches the E-step over N > 0 rows; returns the rows per log-likelihood
// partial (K <= 256), or 0 when the rows still need k_normalize.
template <typename T>
int launch_estep(const T *X, i64 N, i64 D, i64 K, const T *img, const double *cst, T *q, bool fast,
                 double *ll_part, cudaStream_t s) {
  constexpr int VE = 16 / (int)sizeof(T);
  const bool vec = D % VE == 0 && ((uintptr_t)X & 15) == 0;
  const int h = es_half_nj(K);
  const bool f4 = sizeof(T) == 4;
  if (K > 256) {
    if (h == 2) launch_estep_as<T, 4, 8, false>(X, N, D, K, img, cst, q, fast, ll_part, 8, vec, s);
    else if (h == 3) launch_estep_as<T, 6, sizeof(T) == 4 ? 8 : 4, false>(X, N, D, K, img, cst, q, fast, ll_part, 8, vec, s);
    else launch_estep_as<T, 8, sizeof(T) == 4 ? 8 : 4, false>(X, N, D, K, img, cst, q, fast, ll_part, 8, vec, s);
    return 0;
  }
  // Float with up to 128 components takes 16 rows per warp when that still
  // gives every SM its two blocks; otherwise blocks of half the warps spread
  // the rows over more SMs.
  const bool wide = f4 && h <= 2 && N >= (i64)sm_count() * 2 * 128;
  const int warps = N >= (i64)sm_count() * 2 * 64 ? 8 : 4;
  if (h == 1) {
    if constexpr (sizeof(T) == 4)
      if (wide) {
        launch_estep_as<T, 2, 16, true>(X, N, D, K, img, cst, q, fast, ll_part, 8, vec, s);
        return 8;
      }
    launch_estep_as<T, 2, 8, true>(X, N, D, K, img, cst, q, fast, ll_part, warps, vec, s);
    return 8;
  }
  if (h == 2) {
    if constexpr (sizeof(T) == 4)
      if (wide) {
        launch_estep_as<T, 4, 16, true>(X, N, D, K, img, cst, q, fast, ll_part, 8, vec, s);
        return 8;
      }
    launch_estep_as<T, 4, 8, true>(X, N, D, K, img, cst, q, fast, ll_part, warps, vec, s);
    return 8;
  }
  constexpr int R = sizeof(T) == 4 ? 8 : 4;
  if (h == 3) launch_estep_as<T, 6, R, true>(X, N, D, K, img, cst, q, fast, ll_part, warps, vec, s);
  else launch_estep_as<T, 8, R, true>(X, N, D, K, img, cst, q, fast, ll_part, warps, vec, s);
  return R;
}

// Row-wise log-sum-exp normalisation (vl/gmm.c:776-790), one warp per row,
// plus the optional FAST one-hot (vl/fisher.c:398-417: first arg-max wins).
template <typename T>
__global__ void __launch_bounds__(kThreads) k_normalize(T *__restrict__ q, i64 N, int K, int fast,
                                                       double *__restrict__ ll_part) {
  constexpr int W = kThreads / 32;
  __shared__ double sll[W];
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const i64 i = (i64)blockIdx.x * W + w;
  double llrow = 0;
  if (i < N) {
    T *row = q + i * K;
    T mx = (T)(-INFINITY);
    for (int k = lane; k < K; k += 32) mx = max(mx, row[k]);
    mx = warp_max(mx);
    T sum = 0;
    for (int k = lane; k < K; k += 32) {
      T e = dexp(row[k] - mx);
      row[k] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    llrow = log((double)sum) + (double)mx;
    T bv = (T)(-INFINITY);
    int bi = 0x7fffffff;
    for (int k = lane; k < K; k += 32) {
      T v = row[k] / sum;
      row[k] = v;
      if (v > bv) { bv = v; bi = k; }
    }
    if (fast) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        T ov = __shfl_xor_sync(0xffffffffu, bv, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (bi == 0x7fffffff) bi = 0;  // all-NaN row: the reference keeps index 0
      for (int k = lane; k < K; k += 32) row[k] = (T)(k == bi);
    }
  }
  if (lane == 0) sll[w] = llrow;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int j = 0; j < W; ++j) s += sll[j];
    ll_part[blockIdx.x] = s;
  }
}

// One-hot of each row's first arg-max (vl/fisher.c:398-417), one warp per row.
__global__ void __launch_bounds__(kThreads) k_onehot(float *__restrict__ q, i64 N, int K) {
  const i64 i = (i64)blockIdx.x * (kThreads / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x % 32;
  if (i >= N) return;
  float *row = q + i * K;
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  for (int k = lane; k < K; k += 32)
    if (row[k] > bv) { bv = row[k]; bi = k; }
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  if (bi == 0x7fffffff) bi = 0;
  __syncwarp();
  for (int k = lane; k < K; k += 32) row[k] = (float)(k == bi);
}

__global__ void k_sum_doubles(const double *__restrict__ part, i64 n, double *__restrict__ out) {
  __shared__ double sh[kThreads];
  double s = 0;
#pragma unroll 16
  for (i64 j = threadIdx.x; j < n; j += kThreads) s += part[j];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = kThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// ------------------------------------------------------------ M-step
// Thresholded sufficient statistics over one slab of rows for TKC components
// and a block of 8*JMAX dimensions (vl/gmm.c:1093-1149):
//   mass = sum q, S1 = sum q x, S2 = sum q (x - mu_old)^2, with q < 1e-2/K
//   skipped.  Partials are written per slab in double.
template <typename T, int TKC, int RC, int JMAX>
__global__ void __launch_bounds__(kThreads) k_mstep_stats(
    const T *__restrict__ X, const T *__restrict__ q, i64 N, int K, int D, i64 rowsPerSlab,
    const T *__restrict__ oldMeans, double *__restrict__ pmass, double *__restrict__ ps1,
    double *__restrict__ ps2) {
  constexpr int DB = 8 * JMAX;
  __shared__ __align__(16) T sx[RC][DB];
  __shared__ T sq[RC][TKC];
  __shared__ T smo[DB][TKC + 1];
  const int tid = threadIdx.x, c = tid % TKC, dg = tid / TKC;
  const int slab = blockIdx.x, k0 = blockIdx.y * TKC, dbase = blockIdx.z * DB;
  const i64 r0 = (i64)slab * rowsPerSlab;
  const i64 r1 = min(N, r0 + rowsPerSlab);
  const double thr = 1e-2 / (double)K;
  for (int e = tid; e < TKC * DB; e += kThreads) {
    int cc = e / DB, dd = e % DB;
    int k = k0 + cc, d = dbase + dd;
    smo[dd][cc] = (k < K && d < D) ? oldMeans[(i64)k * D + d] : (T)0;
  }
  T s1[JMAX], s2[JMAX], mass = 0;
#pragma unroll
  for (int j = 0; j < JMAX; ++j) s1[j] = s2[j] = 0;
  for (i64 rb = r0; rb < r1; rb += RC) {
    const int rc = (int)min((i64)RC, r1 - rb);
    __syncthreads();
    for (int e = tid; e < RC * DB; e += kThreads) {
      int r = e / DB, dd = e % DB, d = dbase + dd;
      sx[r][dd] = (r < rc && d < D) ? X[(rb + r) * D + d] : (T)0;
    }
    for (int e = tid; e < RC * TKC; e += kThreads) {
      int r = e / TKC, cc = e % TKC, k = k0 + cc;
      T v = (r < rc && k < K) ? q[(rb + r) * K + k] : (T)0;
      sq[r][cc] = ((double)v < thr) ? (T)0 : v;
    }
    __syncthreads();
    if constexpr (sizeof(T) == 4 && JMAX % 2 == 0) {
      // Packed fp32x2 over dimension pairs (j, j + 1): each half is the
      // scalar x - mu_old, its square, p x + s1 and p (x - mu_old)^2 + s2.
      constexpr unsigned long long kNeg = 0x8000000080000000ull;
      unsigned long long mo[JMAX / 2], a1[JMAX / 2], a2[JMAX / 2];
#pragma unroll
      for (int j = 0; j < JMAX; j += 2) {
        mo[j / 2] = tc::f2u(smo[dg + 8 * j][c], smo[dg + 8 * j + 8][c]) ^ kNeg;
        a1[j / 2] = tc::f2u(s1[j], s1[j + 1]);
        a2[j / 2] = tc::f2u(s2[j], s2[j + 1]);
      }
      for (int r = 0; r < rc; ++r) {
        const T p = sq[r][c];
        if (p == (T)0) continue;
        mass += p;
        const unsigned long long pp = tc::f2u(p, p);
#pragma unroll
        for (int j = 0; j < JMAX; j += 2) {
          const unsigned long long xp = tc::f2u(sx[r][dg + 8 * j], sx[r][dg + 8 * j + 8]);
          const unsigned long long df = tc::add2(xp, mo[j / 2]);
          a1[j / 2] = tc::fma2(pp, xp, a1[j / 2]);
          a2[j / 2] = tc::fma2(pp, tc::mul2(df, df), a2[j / 2]);
        }
      }
#pragma unroll
      for (int j = 0; j < JMAX; j += 2) {
        s1[j] = tc::lo32(a1[j / 2]);
        s1[j + 1] = tc::hi32(a1[j / 2]);
        s2[j] = tc::lo32(a2[j / 2]);
        s2[j + 1] = tc::hi32(a2[j / 2]);
      }
    } else {
      for (int r = 0; r < rc; ++r) {
        const T p = sq[r][c];
        if (p == (T)0) continue;
        mass += p;
#pragma unroll
        for (int j = 0; j < JMAX; ++j) {
          const int dd = dg + 8 * j;
          const T x = sx[r][dd];
          const T diff = x - smo[dd][c];
          s1[j] += p * x;
          s2[j] += p * (diff * diff);
        }
      }
    }
  }
  const int k = k0 + c;
  if (k < K) {
    const i64 base = ((i64)slab * K + k) * D;
#pragma unroll
    for (int j = 0; j < JMAX; ++j) {
      const int d = dbase + dg + 8 * j;
      if (d < D) {
        ps1[base + d] = (double)s1[j];
        ps2[base + d] = (double)s2[j];
      }
    }
    if (dg == 0 && blockIdx.z == 0) pmass[(i64)slab * K + k] = (double)mass;
  }
}

// Normalisation, old-to-new mean correction and bounds (vl/gmm.c:1169-1194);
// priors receive the mass, normalised by k_normalize_priors.
// 32 (component, dimension) elements per block, slabs added in order.  296
// slabs of 64 x 64: 12 us a launch (a thread per element: 111).
template <typename T>
__global__ void __launch_bounds__(kOrdThreads) k_mstep_finalize(
    int nslab, int K, int D, const double *__restrict__ pmass, const double *__restrict__ ps1,
    const double *__restrict__ ps2, const double *__restrict__ lb, T *__restrict__ means, T *__restrict__ covs,
    T *__restrict__ priors) {
  __shared__ OrdShared<3> sh;
  const i64 KD = (i64)K * D, idx = (i64)blockIdx.x * 32 + threadIdx.x % 32;
  const i64 at = min(idx, KD - 1);
  const int k = (int)(at / D), d = (int)(at % D);
  double S[3];
  ordered_sums<3>(
      nslab,
      [&](int sl, int q) { return q == 0 ? pmass[(i64)sl * K + k] : q == 1 ? ps1[sl * KD + at] : ps2[sl * KD + at]; },
      sh, S);
  if (threadIdx.x >= 32 || idx >= KD) return;
  const double mass = S[0];
  const double oldmu = (double)means[idx];
  double mu = S[1], v = S[2];
  if (mass >= 1e-6 / (double)K) {
    mu = S[1] / mass;
    v = S[2] / mass;
    const double df = mu - oldmu;
    v -= df * df;
  }
  T vt = (T)v;
  if ((double)vt < lb[d]) vt = (T)lb[d];
  means[idx] = (T)mu;
  covs[idx] = vt;
  if (d == 0) priors[k] = (T)mass;
}

template <typename T>
__global__ void k_normalize_priors(T *__restrict__ priors, int K) {
  __shared__ double sh[kThreads];
  double s = 0;
  for (int k = threadIdx.x; k < K; k += kThreads) s += (double)priors[k];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = kThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  double tot = sh[0];
  if (tot < 1e-12) tot = 1e-12;
  for (int k = threadIdx.x; k < K; k += kThreads) priors[k] = (T)((double)priors[k] / tot);
}

template <typename T>
__global__ void k_apply_bounds(T *__restrict__ covs, i64 n, int D, const double *__restrict__ lb) {
  i64 idx = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int d = (int)(idx % D);
  if ((double)covs[idx] < lb[d]) covs[idx] = (T)lb[d];
}

// Column sums of the posteriors per slab (vl/gmm.c:835-844).
template <typename T>
__global__ void k_colmass(const T *__restrict__ q, i64 N, int K, i64 rowsPerSlab,
                          double *__restrict__ part) {
  const i64 r0 = (i64)blockIdx.x * rowsPerSlab, r1 = min(N, r0 + rowsPerSlab);
  for (int k = threadIdx.x; k < K; k += kThreads) {
    double s = 0;
    for (i64 i = r0; i < r1; ++i) s += (double)q[i * K + k];
    part[(i64)blockIdx.x * K + k] = s;
  }
}

// The same sums for fp32 posteriors with K a multiple of 4 (K <= 1024):
// each thread reads four columns as a float4, the block covers
// 1024 / K rows per pass (coalesced 16-byte loads), four rows per thread are
// in flight, and the row groups are summed in index order at the end.
__global__ void __launch_bounds__(kThreads) k_colmass4(const float *__restrict__ q, i64 N, int K,
                                                       i64 rowsPerSlab, double *__restrict__ part) {
  __shared__ double sh[4 * kThreads];  // [row group][column]
  const int tpr = K / 4, rpb = kThreads / tpr;
  const int rg = threadIdx.x / tpr, c4 = threadIdx.x % tpr;
  const i64 r0 = (i64)blockIdx.x * rowsPerSlab, r1 = min(N, r0 + rowsPerSlab);
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  if (rg < rpb) {
    i64 i = r0 + rg;
    for (; i + 3 * rpb < r1; i += 4 * rpb) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg((const float4 *)(q + (i + u * rpb) * K) + c4);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s0 += (double)v[u].x;
        s1 += (double)v[u].y;
        s2 += (double)v[u].z;
        s3 += (double)v[u].w;
      }
    }
    for (; i < r1; i += rpb) {
      const float4 v = __ldg((const float4 *)(q + i * K) + c4);
      s0 += (double)v.x;
      s1 += (double)v.y;
      s2 += (double)v.z;
      s3 += (double)v.w;
    }
    double *row = sh + rg * K + 4 * c4;
    row[0] = s0;
    row[1] = s1;
    row[2] = s2;
    row[3] = s3;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += kThreads) {
    double t = 0;
    for (int g = 0; g < rpb; ++g) t += sh[g * K + k];
    part[(i64)blockIdx.x * K + k] = t;
  }
}

__global__ void __launch_bounds__(kOrdThreads) k_sum_slabs(const double *__restrict__ part, int nslab, int K,
                                                           double *__restrict__ out) {
  __shared__ OrdShared<1> sh;
  const int k = blockIdx.x * 32 + threadIdx.x % 32, at = min(k, K - 1);
  double S[1];
  ordered_sums<1>(nslab, [&](int sl, int) { return part[(i64)sl * K + at]; }, sh, S);
  if (threadIdx.x < 32 && k < K) out[k] = S[0];
}

template <typename T>
__global__ void k_restart_split(T *__restrict__ q, const T *__restrict__ X, i64 N, int K, int D,
                                int icl, int best, int dim, T cut) {
  i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  T p = q[i * K + best], r = q[i * K + icl];
  if (X[i * D + dim] < cut) {
    q[i * K + icl] = p + r;
    q[i * K + best] = 0;
  } else {
    q[i * K + icl] = 0;
    q[i * K + best] = p + r;
  }
}

// ------------------------------------------------------------ Fisher
// Fisher statistics of one segment for TKC components and a block of
// 8*JMAX dimensions (vl/fisher.c:419-449): for pi_k >= 1e-6 and q >= 1e-6,
// u += q (x-mu) s, v += q ((x-mu)^2 s^2 - 1); counts the accumulated terms.
template <typename T, int TKC, int RC, int JMAX>
__global__ void __launch_bounds__(kThreads) k_fisher_stats(
    const T *__restrict__ X, const T *__restrict__ q, i64 qbase, int K, int D,
    const Segment *__restrict__ segs, const T *__restrict__ means, const T *__restrict__ sis,
    const T *__restrict__ priors, double *__restrict__ pu, double *__restrict__ pv,
    unsigned long long *__restrict__ pnt) {
  constexpr int DB = 8 * JMAX;
  __shared__ __align__(16) T sx[RC][DB];
  __shared__ T sq[RC][TKC];
  __shared__ T smu[DB][TKC + 1];
  __shared__ T ssi[DB][TKC + 1];
  const int tid = threadIdx.x, c = tid % TKC, dg = tid / TKC;
  const int sidx = blockIdx.x, k0 = blockIdx.y * TKC, dbase = blockIdx.z * DB;
  const Segment sg = segs[sidx];
  for (int e = tid; e < TKC * DB; e += kThreads) {
    int cc = e / DB, dd = e % DB;
    int k = k0 + cc, d = dbase + dd;
    bool ok = (k < K && d < D);
    smu[dd][cc] = ok ? means[(i64)k * D + d] : (T)0;
    ssi[dd][cc] = ok ? sis[(i64)k * D + d] : (T)0;
  }
  const int k = k0 + c;
  const bool active = (k < K) && ((double)priors[k] >= 1e-6);
  T u[JMAX], v[JMAX];
#pragma unroll
  for (int j = 0; j < JMAX; ++j) u[j] = v[j] = 0;
  unsigned long long nt = 0;
  for (i64 rb = sg.row0; rb < sg.row1; rb += RC) {
    const int rc = (int)min((i64)RC, sg.row1 - rb);
    __syncthreads();
    for (int e = tid; e < RC * DB; e += kThreads) {
      int r = e / DB, dd = e % DB, d = dbase + dd;
      sx[r][dd] = (r < rc && d < D) ? X[(rb + r) * D + d] : (T)0;
    }
    for (int e = tid; e < RC * TKC; e += kThreads) {
      int r = e / TKC, cc = e % TKC, kk = k0 + cc;
      T val = (r < rc && kk < K) ? q[(rb + r - qbase) * K + kk] : (T)0;
      sq[r][cc] = ((double)val < 1e-6) ? (T)0 : val;
    }
    __syncthreads();
    if (!active) continue;
    if constexpr (sizeof(T) == 4 && JMAX % 2 == 0) {
      // Packed fp32x2 over dimension pairs (j, j + 1): each half is the
      // scalar (x - mu) sigma^-1, p df + u and p (df^2 - 1) + v.
      constexpr unsigned long long kNeg = 0x8000000080000000ull, kMinus1 = 0xbf800000bf800000ull;
      unsigned long long mn[JMAX / 2], si[JMAX / 2], au[JMAX / 2], av[JMAX / 2];
#pragma unroll
      for (int j = 0; j < JMAX; j += 2) {
        mn[j / 2] = tc::f2u(smu[dg * JMAX + j][c], smu[dg * JMAX + j + 1][c]) ^ kNeg;
        si[j / 2] = tc::f2u(ssi[dg * JMAX + j][c], ssi[dg * JMAX + j + 1][c]);
        au[j / 2] = tc::f2u(u[j], u[j + 1]);
        av[j / 2] = tc::f2u(v[j], v[j + 1]);
      }
      for (int r = 0; r < rc; ++r) {
        const T p = sq[r][c];
        if (p == (T)0) continue;
        ++nt;
        const unsigned long long pp = tc::f2u(p, p);
        const unsigned long long *xr = reinterpret_cast<const unsigned long long *>(&sx[r][dg * JMAX]);
#pragma unroll
        for (int j = 0; j < JMAX; j += 2) {
          const unsigned long long xp = xr[j / 2];
          const unsigned long long df = tc::mul2(tc::add2(xp, mn[j / 2]), si[j / 2]);
          au[j / 2] = tc::fma2(pp, df, au[j / 2]);
          av[j / 2] = tc::fma2(pp, tc::fma2(df, df, kMinus1), av[j / 2]);
        }
      }
#pragma unroll
      for (int j = 0; j < JMAX; j += 2) {
        u[j] = tc::lo32(au[j / 2]);
        u[j + 1] = tc::hi32(au[j / 2]);
        v[j] = tc::lo32(av[j / 2]);
        v[j + 1] = tc::hi32(av[j / 2]);
      }
    } else {
      for (int r = 0; r < rc; ++r) {
        const T p = sq[r][c];
        if (p == (T)0) continue;
        ++nt;
#pragma unroll
        for (int j = 0; j < JMAX; ++j) {
          const int dd = dg * JMAX + j;
          const T df = (sx[r][dd] - smu[dd][c]) * ssi[dd][c];
          u[j] += p * df;
          v[j] += p * (df * df - (T)1);
        }
      }
    }
  }
  if (k < K) {
    const i64 base = ((i64)sidx * K + k) * D;
#pragma unroll
    for (int j = 0; j < JMAX; ++j) {
      const int d = dbase + dg * JMAX + j;
      if (d < D) {
        pu[base + d] = (double)u[j];
        pv[base + d] = (double)v[j];
      }
    }
    if (dg == 0 && blockIdx.z == 0) pnt[(i64)sidx * K + k] = nt;
  }
}

// Thresholded statistics visiting only the (row, component) pairs that pass
// the skip, for data of up to 128 dimensions:
//  - kSpFisher: k_fisher_stats' statistics (vl/fisher.c:419-449): per segment,
//    for pi_k >= 1e-6 and q >= 1e-6, u += q df, v += q (df^2 - 1) with
//    df = (x - mu) s, and the term counts;
//  - kSpMstep: k_mstep_stats' statistics (vl/gmm.c:1093-1149): per slab, for
//    q >= 1e-2/K, mass += q, S1 += q x, S2 += q (x - mu_old)^2.
// A block takes one segment (or slab) and 16 CPW components, all dimensions;
// chunks of R rows of x and of the block's posterior columns are
// double-buffered in shared memory.  Warp w owns CPW neighbouring components:
// a lane reads its rows' CPW posteriors, ballots list the rows that pass per
// component, and the warp walks the list in row order, four rows in flight,
// lanes over pairs of dimensions, the component's constants and sums in
// registers.  Per (component, dimension) the operations and their order are
// the dense kernels' (fused multiply-adds as there, rows ascending), so the
// partials are the same bits; the dense kernels spend their time on the pairs
// the skip removes (about 94% of them on typical posteriors).
// Bound by issue: packed operations hold the port two clocks, about 25 clocks
// a passing pair at D = 80 beside the ballots, and by the blocks' barriers
// (warps' lists differ in length).  1.04 M rows, K = 256, D = 80, about 21
// passing components a row: 0.96 ms; a kernel that took one passing row at a
// time from each ballot, over chunks of 32 rows, took 1.83.
constexpr int kFsThreads = 512;
enum { kSpFisher = 0, kSpMstep = 1 };

template <typename T>
struct SparseStatsArgs {
  const T *X;            // rows indexed from the call's first row
  const T *q;            // N x K posteriors, row (r - qbase)
  i64 qbase;
  T thr;                 // the smallest value of the type >= the skip threshold
  int K, D;
  const Segment *segs;   // kSpFisher: the segments
  i64 N, rowsPerSlab;    // kSpMstep: slab s is rows [s rps, min(N, (s + 1) rps))
  const T *mu;           // means (kSpFisher) or old means (kSpMstep)
  const T *sis;          // kSpFisher: 1 / sigma
  const T *priors;       // kSpFisher
  double *p1, *p2;       // u, v (kSpFisher) or S1, S2 (kSpMstep): [block][K][D]
  unsigned long long *pnt;  // kSpFisher: term counts [segment][K]
  double *pmass;            // kSpMstep: [slab][K]
  int xvec, qvec;           // bytes per copied piece of X and q
};

// Two dimensions of one row: packed for float, two values for double.
struct PairF {
  unsigned long long v;
};
struct PairD {
  double a, b;
};
template <typename T>
using PairOf = typename std::conditional<sizeof(T) == 4, PairF, PairD>::type;
__device__ __forceinline__ PairF ld_pair(const float *p) { return {*(const unsigned long long *)p}; }
__device__ __forceinline__ PairD ld_pair(const double *p) {
  const double2 d = *(const double2 *)p;
  return {d.x, d.y};
}
__device__ __forceinline__ PairF mk_pair(float a, float b) { return {tc::f2u(a, b)}; }
__device__ __forceinline__ PairD mk_pair(double a, double b) { return {a, b}; }
__device__ __forceinline__ PairF p_add(PairF a, PairF b) { return {tc::add2(a.v, b.v)}; }
__device__ __forceinline__ PairD p_add(PairD a, PairD b) { return {a.a + b.a, a.b + b.b}; }
__device__ __forceinline__ PairF p_mul(PairF a, PairF b) { return {tc::mul2(a.v, b.v)}; }
__device__ __forceinline__ PairD p_mul(PairD a, PairD b) { return {a.a * b.a, a.b * b.b}; }
__device__ __forceinline__ PairF p_fma(PairF a, PairF b, PairF c) { return {tc::fma2(a.v, b.v, c.v)}; }
__device__ __forceinline__ PairD p_fma(PairD a, PairD b, PairD c) { return {fma(a.a, b.a, c.a), fma(a.b, b.b, c.b)}; }
__device__ __forceinline__ double p_lo(PairF a) { return (double)tc::lo32(a.v); }
__device__ __forceinline__ double p_hi(PairF a) { return (double)tc::hi32(a.v); }
__device__ __forceinline__ double p_lo(PairD a) { return a.a; }
__device__ __forceinline__ double p_hi(PairD a) { return a.b; }

template <typename T, int CPW>
__host__ __device__ constexpr int fs_rows() { return sizeof(T) == 4 ? 128 : 64; }
// Posterior columns of a row in shared memory: 16 bytes of padding keep the
// rows 16-byte aligned and, with 64 float columns, eight lanes' 16-byte reads
// on distinct banks.
template <typename T, int CPW>
__host__ __device__ constexpr int fs_qpitch() { return 16 * CPW + 16 / (int)sizeof(T); }
// A passing row: its posterior and its offset in the chunk's x rows.
template <typename T>
struct __align__(2 * sizeof(T)) RowEntry {
  T p;
  int off;
};
template <typename T, int CPW>
size_t sparse_stats_smem(int D) {
  return sizeof(T) * (size_t)2 * fs_rows<T, CPW>() * ((D + 1) / 2 * 2 + fs_qpitch<T, CPW>()) +
         sizeof(RowEntry<T>) * (size_t)(kFsThreads / 32) * fs_rows<T, CPW>();
}

// NP: pairs of dimensions per lane (dimensions up to 64 NP); NS: single
// dimensions per lane after them (0 or 1, up to 32 more).
template <typename T, int MODE, int NP, int NS, int CPW>
__global__ void __launch_bounds__(kFsThreads, 1) k_stats_sparse(const SparseStatsArgs<T> a) {
  constexpr int NW = kFsThreads / 32, KB = NW * CPW, R = fs_rows<T, CPW>(), QP = fs_qpitch<T, CPW>(), NWD = R / 32;
  using P = PairOf<T>;
  extern __shared__ __align__(16) unsigned char fs_smem[];
  const int K = a.K, D = a.D, Dp = (D + 1) / 2 * 2;
  const T *__restrict__ X = a.X;
  const T *__restrict__ q = a.q;
  T *sx = (T *)fs_smem;        // [2][R][Dp]
  T *sq = sx + 2 * R * Dp;     // [2][R][QP]
  const int tid = threadIdx.x, w = tid / 32, lane = tid % 32;
  using Entry = RowEntry<T>;
  constexpr int U = 4;         // rows of a list in flight
  Entry *list = (Entry *)(sq + 2 * R * QP) + w * R;  // this warp's passing rows of one component
  const unsigned below = (1u << lane) - 1u;
  const int sidx = blockIdx.x, k0 = (blockIdx.z * gridDim.y + blockIdx.y) * KB;
  if (k0 >= K) return;
  i64 row0, row1;
  if constexpr (MODE == kSpFisher) {
    const Segment sg = a.segs[sidx];
    row0 = sg.row0;
    row1 = sg.row1;
  } else {
    row0 = (i64)sidx * a.rowsPerSlab;
    row1 = min(a.N, row0 + a.rowsPerSlab);
  }
  const i64 rows = row1 - row0;
  const int nch = (int)((rows + R - 1) / R);
  const i64 qbase = a.qbase;

  auto issue = [&](int ch) {
    const int b = ch & 1;
    const i64 rb = row0 + (i64)ch * R;
    const int rc = (int)min((i64)R, row1 - rb);
    const uint32_t bx = tc::smem_u32(sx + b * R * Dp), bq = tc::smem_u32(sq + b * R * QP);
    const T *xs = X + rb * D;
    // The chunk's x rows are one contiguous range (rows past rc are never
    // used), except that rows of an odd dimension are padded to an even one.
    if (a.xvec == 16) {
      for (int e = tid; e < rc * D * (int)sizeof(T) / 16; e += kFsThreads) cp_async16(bx + 16 * e, (const char *)xs + 16 * e, 16u);
    } else if (a.xvec == 8 && D == Dp) {
      for (int e = tid; e < rc * D * (int)sizeof(T) / 8; e += kFsThreads) cp_async8(bx + 8 * e, (const char *)xs + 8 * e, 8u);
    } else {
      for (int r = w; r < rc; r += NW)
        for (int d = lane; d < D; d += 32)
          cp_async_piece<(int)sizeof(T)>(bx + (uint32_t)sizeof(T) * (r * Dp + d), xs + r * D + d, true);
    }
    if (a.qvec == 16) {
      constexpr int V = 16 / (int)sizeof(T);
      for (int e = tid; e < R * (KB / V); e += kFsThreads) {
        const int r = e / (KB / V), c = e % (KB / V) * V, kk = k0 + c;
        const bool ok = r < rc && kk < K;
        cp_async16(bq + (uint32_t)sizeof(T) * (r * QP + c), ok ? q + (rb + r - qbase) * K + kk : q, ok ? 16u : 0u);
      }
    } else {
      for (int e = tid; e < R * KB; e += kFsThreads) {
        const int r = e / KB, c = e % KB, kk = k0 + c;
        const bool ok = r < rc && kk < K;
        cp_async_piece<(int)sizeof(T)>(bq + (uint32_t)sizeof(T) * (r * QP + c), ok ? q + (rb + r - qbase) * K + kk : q, ok);
      }
    }
    cp_async_commit();
  };

  if (nch > 0) issue(0);
  // This lane's dimension pairs 2 (lane + 32 j), 2 (lane + 32 j) + 1; lanes
  // past the last pair read pair 0 and write nothing.
  int off[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const int d = 2 * (lane + 32 * j);
    off[j] = d < D ? d : 0;
  }
  const int ds = 64 * NP + lane, offs = NS && ds < D ? ds : 0;
  // The skip: values below thr (compared in double, i.e. below a.thr in the
  // data type; NaN passes in both, zeros and rows past the end do not).
  const T thr = a.thr;
  bool act[CPW];
  P mn[CPW][NP], si[CPW][NP], u[CPW][NP], v[CPW][NP];
  T smn[CPW], ssi[CPW], su[CPW], sv[CPW];  // the single dimension's
  T mass[CPW];
  unsigned nt[CPW];  // at most the segment's rows
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int k = k0 + w * CPW + c;
    if constexpr (MODE == kSpFisher) act[c] = k < K && (double)a.priors[k] >= 1e-6;
    else act[c] = k < K;
    nt[c] = 0;
    mass[c] = su[c] = sv[c] = (T)0;
    if constexpr (NS > 0) {
      smn[c] = act[c] ? a.mu[(i64)k * D + offs] : (T)0;
      if constexpr (MODE == kSpFisher) ssi[c] = act[c] ? a.sis[(i64)k * D + offs] : (T)0;
    }
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      u[c][j] = v[c][j] = mk_pair((T)0, (T)0);
      const bool o0 = act[c], o1 = act[c] && off[j] + 1 < D;
      const i64 e = (i64)k * D + off[j];
      mn[c][j] = mk_pair(o0 ? -a.mu[e] : (T)0, o1 ? -a.mu[e + 1] : (T)0);
      if constexpr (MODE == kSpFisher) si[c][j] = mk_pair(o0 ? a.sis[e] : (T)0, o1 ? a.sis[e + 1] : (T)0);
    }
  }
  const P minus1 = mk_pair((T)-1, (T)-1);
  for (int ch = 0; ch < nch; ++ch) {
    if (ch + 1 < nch) {
      issue(ch + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const T *bx = sx + (ch & 1) * R * Dp, *bq = sq + (ch & 1) * R * QP + w * CPW;
    T val[NWD][CPW];
#pragma unroll
    for (int wd = 0; wd < NWD; ++wd) {
      if constexpr (sizeof(T) == 4 && CPW == 4) {
        const float4 f = *(const float4 *)(bq + (32 * wd + lane) * QP);
        val[wd][0] = f.x; val[wd][1] = f.y; val[wd][2] = f.z; val[wd][3] = f.w;
      } else {
#pragma unroll
        for (int c = 0; c < CPW; ++c) val[wd][c] = bq[(32 * wd + lane) * QP + c];
      }
    }
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
      if (!act[c]) continue;  // warp-uniform
      // The chunk's passing rows of this component, in row order.
      int n = 0;
#pragma unroll
      for (int wd = 0; wd < NWD; ++wd) {
        const bool pass = !(val[wd][c] < thr);
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (pass) list[n + __popc(m & below)] = Entry{val[wd][c], (32 * wd + lane) * Dp};
        n += __popc(m);
      }
      __syncwarp();
      nt[c] += (unsigned)n;
      auto add = [&](T p, const P(&x)[NP], T xs) {
        const P pp = mk_pair(p, p);
        if constexpr (MODE == kSpMstep) mass[c] += p;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          if constexpr (MODE == kSpFisher) {
            const P df = p_mul(p_add(x[j], mn[c][j]), si[c][j]);
            u[c][j] = p_fma(pp, df, u[c][j]);
            v[c][j] = p_fma(pp, p_fma(df, df, minus1), v[c][j]);
          } else {
            const P df = p_add(x[j], mn[c][j]);
            u[c][j] = p_fma(pp, x[j], u[c][j]);
            v[c][j] = p_fma(pp, p_mul(df, df), v[c][j]);
          }
        }
        if constexpr (NS > 0) {
          if constexpr (MODE == kSpFisher) {
            const T df = (xs - smn[c]) * ssi[c];
            su[c] = fma(p, df, su[c]);
            sv[c] = fma(p, fma(df, df, (T)-1), sv[c]);
          } else {
            const T df = xs - smn[c];
            su[c] = fma(p, xs, su[c]);
            sv[c] = fma(p, df * df, sv[c]);
          }
        }
      };
      int i = 0;
#pragma unroll 1
      for (; i + U <= n; i += U) {
        Entry en[U];
        P x[U][NP];
        T xs[U];
#pragma unroll
        for (int g = 0; g < U; ++g) en[g] = list[i + g];
#pragma unroll
        for (int g = 0; g < U; ++g)
#pragma unroll
          for (int j = 0; j < NP; ++j) x[g][j] = ld_pair(bx + en[g].off + off[j]);
#pragma unroll
        for (int g = 0; g < U; ++g) xs[g] = NS > 0 ? bx[en[g].off + offs] : (T)0;
#pragma unroll
        for (int g = 0; g < U; ++g) add(en[g].p, x[g], xs[g]);
      }
#pragma unroll 1
      for (; i < n; ++i) {
        const Entry en = list[i];
        P x[NP];
#pragma unroll
        for (int j = 0; j < NP; ++j) x[j] = ld_pair(bx + en.off + off[j]);
        add(en.p, x, NS > 0 ? bx[en.off + offs] : (T)0);
      }
      __syncwarp();  // the list is read before the next component's is written
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int k = k0 + w * CPW + c;
    if (k >= K) continue;
    const i64 base = ((i64)sidx * K + k) * D;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int d = 2 * (lane + 32 * j);
      if (d < D) {
        a.p1[base + d] = p_lo(u[c][j]);
        a.p2[base + d] = p_lo(v[c][j]);
      }
      if (d + 1 < D) {
        a.p1[base + d + 1] = p_hi(u[c][j]);
        a.p2[base + d + 1] = p_hi(v[c][j]);
      }
    }
    if (NS > 0 && ds < D) {
      a.p1[base + ds] = (double)su[c];
      a.p2[base + ds] = (double)sv[c];
    }
    if (lane == 0) {
      if constexpr (MODE == kSpFisher) a.pnt[(i64)sidx * K + k] = (unsigned long long)nt[c];
      else a.pmass[(i64)sidx * K + k] = (double)mass[c];
    }
  }
}

template <typename T, int MODE, int NP, int NS, int CPW>
void launch_stats_sparse_as(const SparseStatsArgs<T> &a, i64 nblk, cudaStream_t s) {
  auto kern = k_stats_sparse<T, MODE, NP, NS, CPW>;
  const size_t smem = sparse_stats_smem<T, CPW>(a.D);
  VLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int kb = kFsThreads / 32 * CPW;
  const unsigned nb = (unsigned)((a.K + kb - 1) / kb), nz = (nb + 65534) / 65535;  // a grid has 65,535 rows at most
  kern<<<dim3((unsigned)nblk, (nb + nz - 1) / nz, nz), kFsThreads, smem, s>>>(a);
}

// Launches k_stats_sparse over nblk segments (or slabs); false when the shape
// is outside it (the dense kernel runs instead).
template <int MODE, typename T>
bool launch_stats_sparse(SparseStatsArgs<T> a, i64 nblk, cudaStream_t s) {
  if (a.D > 128 || nblk <= 0) return false;
  const int VE = 16 / (int)sizeof(T);
  const uintptr_t xa = (uintptr_t)a.X, qa = (uintptr_t)a.q;
  a.xvec = a.D % VE == 0 && xa % 16 == 0 ? 16 : a.D % 2 == 0 && xa % 8 == 0 ? 8 : (int)sizeof(T);
  a.qvec = a.K % VE == 0 && qa % 16 == 0 ? 16 : (int)sizeof(T);
  // (double)v < t for a value v of the type exactly when v < tf, tf the
  // smallest such value >= t.
  const double t = MODE == kSpFisher ? 1e-6 : 1e-2 / (double)a.K;
  T tf = (T)t;
  if ((double)tf < t) tf = std::nextafter(tf, (T)INFINITY);
  a.thr = tf;
  // Four components per warp read x a quarter as often; with too few segments
  // to give every SM a block that way, one per warp spreads the components
  // over four times the blocks.  One image of 500 rows, K = 64, D = 64: 15 us
  // with one, 27 with four; 1.04 M rows in 256 images, K = 256, D = 80: 1485 and
  // 965 us.  In double four components' constants and sums do not fit in
  // registers.
  // Up to 96 dimensions the ones past 64 are single dimensions: half the issue
  // time of a second, mostly empty round of pairs.
  auto go = [&](auto cpw) {
    constexpr int C = decltype(cpw)::value;
    if (a.D <= 64) launch_stats_sparse_as<T, MODE, 1, 0, C>(a, nblk, s);
    else if (a.D <= 96) launch_stats_sparse_as<T, MODE, 1, 1, C>(a, nblk, s);
    else launch_stats_sparse_as<T, MODE, 2, 0, C>(a, nblk, s);
  };
  if constexpr (sizeof(T) == 4) {
    if (nblk * ((a.K + 63) / 64) >= (i64)sm_count()) {
      go(std::integral_constant<int, 4>());
      return true;
    }
  }
  go(std::integral_constant<int, 1>());
  return true;
}

// Per-image Fisher finalisation (vl/fisher.c:450-485): sum the image's
// segment partials, scale u by 1/(N sqrt pi) and v by 1/(N sqrt(2 pi)),
// signed square root, global L2 normalisation.  A cluster of kFvCluster blocks
// per image: each forms its part of the vector in shared memory, the partial
// norms and term counts go through distributed shared memory (added in rank
// order, so every block scales by the same bits), and each part is written
// once.  Bound by the latency of a block's loads and divisions; 256 images of
// K = 256, D = 80: 0.133 ms (one block per image, the vector written, read back
// and divided: 0.49); one image of K = 64, D = 64: 10 us against 25.
constexpr int kFvCluster = 8;
// Elements of each half (u and v) per block.
__host__ __device__ inline i64 fv_part(i64 KD) { return (KD + kFvCluster - 1) / kFvCluster; }
// Components that a part of E elements of dimension D touches, at most.  Their
// factors are tabulated in shared memory up to kFvTable of them (64 KB); above
// that, from 32,752 components on, each element forms its own.
__host__ __device__ inline i64 fv_part_comps(i64 E, i64 D) { return E / D + 2; }
constexpr i64 kFvTable = 4096;

// cached: the block's part fits in shared memory; else it is formed in place
// in the output and scaled there.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_fisher_finalize(
    int K, int D, const int *__restrict__ imgSegBegin, const i64 *__restrict__ imgRows,
    const double *__restrict__ pu, const double *__restrict__ pv,
    const unsigned long long *__restrict__ pnt, const T *__restrict__ priors, int flags,
    i64 imgBase, T *__restrict__ enc, unsigned long long *__restrict__ nterms, int cached) {
  constexpr int NW = kThreads / 32;
  extern __shared__ __align__(16) unsigned char fin_smem[];
  __shared__ double sh[NW], part, total;
  __shared__ unsigned long long shn[NW], partn;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x;
  const int img = blockIdx.x / kFvCluster;
  const int s0 = imgSegBegin[img], s1 = imgSegBegin[img + 1];
  const i64 n = imgRows[img];
  const i64 KD = (i64)K * D, E = fv_part(KD), lo = min(KD, rank * E), hi = min(KD, lo + E);
  T *out = enc + (imgBase + img) * 2 * KD;
  // Per-component factors 1 / (n sqrt(pi_k)) and 1 / (n sqrt(2 pi_k)) of this
  // part's components (-1: the component is skipped, its entries are 0).
  const int ka = (int)(lo / D), nk = hi > lo ? (int)((hi - 1) / D) - ka + 1 : 0;
  const i64 ncomp = fv_part_comps(E, D);
  const bool table = ncomp <= kFvTable;
  double *sfu = (double *)fin_smem, *sfv = sfu + (table ? ncomp : 0);
  T *zu = (T *)(sfv + (table ? ncomp : 0)), *zv = zu + E;
  auto factor = [&](int k, double c) -> double {  // 1 / (n sqrt(c pi_k))
    const double pk = (double)priors[k];
    return pk >= 1e-6 && n > 0 ? 1.0 / ((double)n * sqrt(c * pk)) : -1.0;
  };
  if (table) {
    for (int k = tid; k < nk; k += kThreads) {
      sfu[k] = factor(ka + k, 1.0);
      sfv[k] = factor(ka + k, 2.0);
    }
    __syncthreads();
  }
  double sq = 0;
  // For float, sqrtf is the float rounding of the double square root (double
  // rounding is innocuous for sqrt with 53 >= 2 x 24 + 2 bits).
  auto finish = [&](double acc, double f) -> T {
    T zt = (T)(f >= 0.0 ? acc * f : 0.0);
    if (flags & 1) {
      if constexpr (sizeof(T) == 4) zt = zt >= 0.f ? sqrtf(zt) : -sqrtf(-zt);
      else zt = zt >= (T)0 ? (T)sqrt((double)zt) : -(T)sqrt(-(double)zt);
    }
    sq += (double)zt * (double)zt;
    return zt;
  };
  for (i64 e = lo + tid; e < hi; e += kThreads) {
    const int k = (KD <= (i64)INT32_MAX ? (int)((unsigned)e / (unsigned)D) : (int)(e / D)) - ka;
    double au = 0, av = 0;
#pragma unroll 4
    for (int s = s0; s < s1; ++s) {
      au += pu[(i64)s * KD + e];
      av += pv[(i64)s * KD + e];
    }
    const T u = finish(au, table ? sfu[k] : factor(ka + k, 1.0));
    const T v = finish(av, table ? sfv[k] : factor(ka + k, 2.0));
    if (cached) {
      zu[e - lo] = u;
      zv[e - lo] = v;
    } else {
      out[e] = u;
      out[KD + e] = v;
    }
  }
  unsigned long long nt = 0;
  for (i64 e = rank * kThreads + tid; e < K; e += kThreads * kFvCluster)
    for (int s = s0; s < s1; ++s) nt += pnt[(i64)s * K + e];
  sq = warp_sum(sq);
  nt = warp_sum(nt);
  if (tid % 32 == 0) {
    sh[tid / 32] = sq;
    shn[tid / 32] = nt;
  }
  __syncthreads();
  if (tid == 0) {
    double t = 0;
    unsigned long long c = 0;
    for (int w = 0; w < NW; ++w) {
      t += sh[w];
      c += shn[w];
    }
    part = t;
    partn = c;
  }
  cluster.sync();  // every block's partials are written
  if (tid == 0) {
    double t = 0;
    unsigned long long c = 0;
    for (int r = 0; r < kFvCluster; ++r) {
      t += *cluster.map_shared_rank(&part, r);
      c += *cluster.map_shared_rank(&partn, r);
    }
    total = t;
    if (rank == 0 && nterms) nterms[imgBase + img] = c;
  }
  __syncthreads();
  const bool scale = (flags & 2) != 0;
  double nrm = sqrt(total);
  if (nrm < 1e-12) nrm = 1e-12;
  const T nf = (T)nrm;
  if (cached) {
    for (i64 e = lo + tid; e < hi; e += kThreads) {
      out[e] = scale ? zu[e - lo] / nf : zu[e - lo];
      out[KD + e] = scale ? zv[e - lo] / nf : zv[e - lo];
    }
  } else if (scale) {
    for (i64 e = lo + tid; e < hi; e += kThreads) {
      out[e] = out[e] / nf;
      out[KD + e] = out[KD + e] / nf;
    }
  }
  cluster.sync();  // the partials stay readable until every block has read them
}

template <typename T>
void launch_fisher_finalize(i64 nimg, i64 K, i64 D, const int *imgSegBegin, const i64 *imgRows, const double *pu,
                            const double *pv, const unsigned long long *pnt, const T *priors, int flags, i64 imgBase,
                            T *enc, unsigned long long *nterms, cudaStream_t s) {
  const i64 E = fv_part(K * D);
  const i64 ncomp = fv_part_comps(E, D);
  size_t smem = ncomp <= kFvTable ? sizeof(double) * 2 * (size_t)ncomp : 0;
  const int cached = smem + 2 * sizeof(T) * (size_t)E <= 200 * 1024;
  if (cached) smem += 2 * sizeof(T) * (size_t)E;
  auto kern = k_fisher_finalize<T>;
  VLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kFvCluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(nimg * kFvCluster));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  VLB_CUDA(cudaLaunchKernelEx(&cfg, kern, (int)K, (int)D, imgSegBegin, imgRows, pu, pv, pnt, priors, flags, imgBase,
                              enc, nterms, cached));
}

template <typename T>
T half_dim_log_2pi(i64 D) {
  return (T)(((double)D / 2.0) * log(2.0 * 3.141592653589793));
}

inline unsigned grid1(i64 n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

// ================================================================ launchers

// Elements of the E-step's model image for K components of dimension D.
template <typename T>
size_t exact_image_elems(i64 K, i64 D) {
  return (size_t)es_blocks(K) * 64 * es_half_nj(K) * 2 * es_dpad<T>(D);
}

namespace {
template <typename T>
unsigned prepare_grid(i64 K) {
  return (unsigned)((es_blocks(K) * 64 * es_half_nj(K) * 32 + 127) / 128);
}
}  // namespace

template <typename T>
void exact_prepare(const DevModel<T> &m, DevDerived<T> &der, cudaStream_t s) {
  VLB_LAUNCH("exact_prepare", s,
             k_prepare<T><<<prepare_grid<T>(m.K), 128, 0, s>>>(m.priors, m.means, m.covs, (int)m.K, (int)m.D,
                                                               half_dim_log_2pi<T>(m.D), der.inv, der.cst,
                                                               der.sis, der.img));
}

// Capacity bound for any E-step kernel: the exact kernels write one partial
// per 8 rows (4 for double with more than 128 components); the tensor-core
// E-step 8 per 128-row tile.
i64 estep_ll_parts(i64 N) { return std::max<i64>((N + 3) / 4 + 1, 8 * ((N + 127) / 128) + 8); }

template <typename T>
i64 exact_estep(const T *X, i64 N, const DevModel<T> &m, const DevDerived<T> &der, T *q,
                double *ll_part, bool fast, cudaStream_t s) {
  if (N <= 0) return 0;
  int per = 0;
  VLB_LAUNCH("exact_estep", s,
             per = launch_estep<T>(X, N, m.D, m.K, der.img, der.cst, q, fast, ll_part, s));
  if (per > 0) return (N + per - 1) / per;
  VLB_LAUNCH("exact_normalize", s,
             k_normalize<T><<<grid1(N, 8), kThreads, 0, s>>>(q, N, (int)m.K, fast ? 1 : 0,
                                                             ll_part));
  return (i64)grid1(N, 8);
}

void sum_doubles(const double *part, i64 n, double *out, cudaStream_t s) {
  VLB_LAUNCH("sum_doubles", s, k_sum_doubles<<<1, kThreads, 0, s>>>(part, n, out));
}

namespace {
i64 pick_slab_rows(i64 N) {
  // About 2 slabs per SM for large N; at least 256 rows per slab.
  i64 slabs = 296;
  i64 r = (N + slabs - 1) / slabs;
  if (r < 256) r = 256;
  return r;
}
}  // namespace

// The M-step statistics of nslab slabs of rows by the sparse kernel (up to 128
// dimensions); false when the dense kernel is to run.
template <typename T>
bool mstep_stats_sparse(const T *X, const T *q, i64 N, i64 K, i64 D, i64 rps, i64 nslab, const T *oldMeans,
                        double *pmass, double *ps1, double *ps2, cudaStream_t s) {
  if (D > 128) return false;
  SparseStatsArgs<T> a{};
  a.X = X; a.q = q; a.qbase = 0; a.K = (int)K; a.D = (int)D; a.N = N; a.rowsPerSlab = rps;
  a.mu = oldMeans; a.p1 = ps1; a.p2 = ps2; a.pmass = pmass;
  bool done = false;
  VLB_LAUNCH("exact_mstep_stats", s, done = launch_stats_sparse<kSpMstep>(a, nslab, s));
  return done;
}

template <typename T>
void exact_mstep(const T *X, i64 N, const T *q, T *means, T *covs, T *priors, i64 K, i64 D,
                 const double *lb, cudaStream_t s) {
  constexpr int TKC = 32, RC = 32, JMAX = sizeof(T) == 8 ? 8 : 16, DB = 8 * JMAX;
  const i64 rps = pick_slab_rows(N > 0 ? N : 1);
  const int nslab = (int)((N + rps - 1) / rps > 0 ? (N + rps - 1) / rps : 1);
  Scratch &sc = thread_scratch(kArenaExact);
  double *pmass = sc.slot[10].get<double>((size_t)nslab * K);
  double *ps1 = sc.slot[11].get<double>((size_t)nslab * K * D);
  double *ps2 = sc.slot[12].get<double>((size_t)nslab * K * D);
  if (N > 0) {
    if (!mstep_stats_sparse<T>(X, q, N, K, D, rps, nslab, means, pmass, ps1, ps2, s)) {
      dim3 g(nslab, grid1(K, TKC), grid1(D, DB));
      VLB_LAUNCH("exact_mstep_stats", s,
                 (k_mstep_stats<T, TKC, RC, JMAX><<<g, kThreads, 0, s>>>(
                     X, q, N, (int)K, (int)D, rps, means, pmass, ps1, ps2)));
    }
  } else {
    VLB_CUDA(cudaMemsetAsync(pmass, 0, sizeof(double) * nslab * K, s));
    VLB_CUDA(cudaMemsetAsync(ps1, 0, sizeof(double) * nslab * K * D, s));
    VLB_CUDA(cudaMemsetAsync(ps2, 0, sizeof(double) * nslab * K * D, s));
  }
  VLB_LAUNCH("exact_mstep_finalize", s,
             k_mstep_finalize<T><<<grid1(K * D, 32), kOrdThreads, 0, s>>>(
                 nslab, (int)K, (int)D, pmass, ps1, ps2, lb, means, covs, priors));
  VLB_LAUNCH("normalize_priors", s, k_normalize_priors<T><<<1, kThreads, 0, s>>>(priors, (int)K));
}

i64 exact_mstep_slab_rows(i64 N) { return pick_slab_rows(N > 0 ? N : 1); }

template <typename T>
void exact_mstep_stats_rows(const T *X, i64 row0, i64 n, i64 rps, const T *q, const T *oldMeans, i64 K,
                            i64 D, double *pmass, double *ps1, double *ps2, cudaStream_t s) {
  constexpr int TKC = 32, RC = 32, JMAX = sizeof(T) == 8 ? 8 : 16, DB = 8 * JMAX;
  if (n <= 0) return;
  VLB_CHECK(row0 % rps == 0, VL_ERR_BAD_ARG, "M-step chunk must start on a slab boundary");
  const i64 s0 = row0 / rps, nslab = (n + rps - 1) / rps;
  if (mstep_stats_sparse<T>(X + row0 * D, q, n, K, D, rps, nslab, oldMeans, pmass + s0 * K, ps1 + s0 * K * D,
                            ps2 + s0 * K * D, s))
    return;
  dim3 g((unsigned)nslab, grid1(K, TKC), grid1(D, DB));
  VLB_LAUNCH("exact_mstep_stats", s,
             (k_mstep_stats<T, TKC, RC, JMAX><<<g, kThreads, 0, s>>>(
                 X + row0 * D, q, n, (int)K, (int)D, rps, oldMeans, pmass + s0 * K, ps1 + s0 * K * D,
                 ps2 + s0 * K * D)));
}

template <typename T>
void exact_mstep_finalize_slabs(int nslab, const double *pmass, const double *ps1, const double *ps2,
                                const double *lb, T *means, T *covs, T *priors, i64 K, i64 D,
                                cudaStream_t s) {
  VLB_LAUNCH("exact_mstep_finalize", s,
             k_mstep_finalize<T><<<grid1(K * D, 32), kOrdThreads, 0, s>>>(
                 nslab, (int)K, (int)D, pmass, ps1, ps2, lb, means, covs, priors));
  VLB_LAUNCH("normalize_priors", s, k_normalize_priors<T><<<1, kThreads, 0, s>>>(priors, (int)K));
}

// Slab partials summed into slab 0 in slab order (the order the finalize
// kernel uses), so that the finalize over one slab gives the same values.
__global__ void k_sum_slabs(int nslab, i64 K, i64 KD, double *__restrict__ pmass, double *__restrict__ ps1,
                            double *__restrict__ ps2) {
  const i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= KD) return;
  double a = 0, b = 0, c = 0;
  for (int sl = 0; sl < nslab; ++sl) {
    if (i < K) a += pmass[(i64)sl * K + i];
    b += ps1[(i64)sl * KD + i];
    c += ps2[(i64)sl * KD + i];
  }
  if (i < K) pmass[i] = a;
  ps1[i] = b;
  ps2[i] = c;
}

void exact_sum_slabs(int nslab, double *pmass, double *ps1, double *ps2, i64 K, i64 D, cudaStream_t s) {
  VLB_LAUNCH("sum_slabs", s,
             k_sum_slabs<<<grid1(K * D, kThreads), kThreads, 0, s>>>(nslab, K, K * D, pmass, ps1, ps2));
}

template <typename T>
void normalize_priors(T *priors, i64 K, cudaStream_t s) {
  VLB_LAUNCH("normalize_priors", s, k_normalize_priors<T><<<1, kThreads, 0, s>>>(priors, (int)K));
}

template <typename T>
void column_mass(const T *q, i64 N, i64 K, double *mass, cudaStream_t s) {
  const i64 rps = pick_slab_rows(N > 0 ? N : 1);
  const int nslab = (int)((N + rps - 1) / rps > 0 ? (N + rps - 1) / rps : 1);
  double *part = thread_scratch(kArenaExact).slot[13].get<double>((size_t)nslab * K);
  if (N > 0) {
    bool done = false;
    if constexpr (sizeof(T) == 4) {
      if (K % 4 == 0 && K <= 4 * kThreads) {
        VLB_LAUNCH("column_mass", s, k_colmass4<<<nslab, kThreads, 0, s>>>((const float *)q, N, (int)K, rps, part));
        done = true;
      }
    }
    if (!done) VLB_LAUNCH("column_mass", s, k_colmass<T><<<nslab, kThreads, 0, s>>>(q, N, (int)K, rps, part));
  } else {
    VLB_CUDA(cudaMemsetAsync(part, 0, sizeof(double) * nslab * K, s));
  }
  VLB_LAUNCH("sum_slabs", s, k_sum_slabs<<<grid1(K, 32), kOrdThreads, 0, s>>>(part, nslab, (int)K, mass));
}

template <typename T>
void restart_split(T *q, const T *X, i64 N, i64 K, i64 D, i64 icl, i64 best, i64 dim, T cut,
                   cudaStream_t s) {
  if (N <= 0) return;
  VLB_LAUNCH("restart_split", s,
             k_restart_split<T><<<grid1(N, kThreads), kThreads, 0, s>>>(
                 q, X, N, (int)K, (int)D, (int)icl, (int)best, (int)dim, cut));
}

template <typename T>
void apply_bounds(T *covs, i64 K, i64 D, const double *lb, cudaStream_t s) {
  VLB_LAUNCH("apply_bounds", s,
             k_apply_bounds<T><<<grid1(K * D, kThreads), kThreads, 0, s>>>(covs, K * D, (int)D, lb));
}

// Batched Fisher encoding with the exact kernels.  Images are processed in
// chunks bounded by a row budget; each image is cut into segments of at most
// kSegRows rows so long images still spread over many blocks.
template <typename T>
void exact_fisher_batch(const T *X, const i64 *h_offsets, i64 numImages, const DevModel<T> &m,
                        T *enc, unsigned long long *nterms, int flags, cudaStream_t s,
                        bool use_router) {
  const i64 K = m.K, D = m.D;
  constexpr int TKC = 32, RC = 32, JMAX = sizeof(T) == 8 ? 5 : 10, DB = 8 * JMAX;
  constexpr i64 kSegRows = 2048;
  const i64 kRowBudget = std::max<i64>(4096, (i64)(1u << 30) / (K * (i64)sizeof(T)));
  const i64 kSegBudget = std::max<i64>(64, (i64)(256u << 20) / (2 * K * D * 8));
  Scratch &sc = thread_scratch(kArenaExact);
  DevDerived<T> der;
  der.img = sc.slot[0].get<T>(exact_image_elems<T>(K, D));
  der.sis = sc.slot[1].get<T>(K * D);
  der.cst = sc.slot[2].get<double>(K);
  exact_prepare(m, der, s);

  i64 img = 0;
  while (img < numImages) {
    // Form one chunk of images.
    std::vector<Segment> segs;
    std::vector<int> segBegin;
    std::vector<i64> rows;
    const i64 chunkImg0 = img, row0 = h_offsets[img];
    while (img < numImages) {
      const i64 a = h_offsets[img], b = h_offsets[img + 1];
      const i64 nseg = std::max<i64>(1, (b - a + kSegRows - 1) / kSegRows);
      if (!segs.empty() && ((b - row0) > kRowBudget || (i64)segs.size() + nseg > kSegBudget)) break;
      segBegin.push_back((int)segs.size());
      rows.push_back(b - a);
      for (i64 j = 0; j < nseg; ++j) {
        i64 s0 = a + j * kSegRows, s1 = std::min(b, s0 + kSegRows);
        segs.push_back({img - chunkImg0, s0, s1});
      }
      ++img;
    }
    segBegin.push_back((int)segs.size());
    const i64 nimg = img - chunkImg0;
    const i64 row1 = h_offsets[img];
    const i64 nrows = row1 - row0;
    const i64 nseg = (i64)segs.size();

    T *q = sc.slot[3].get<T>(std::max<i64>(1, nrows) * K);
    double *llp = sc.slot[4].get<double>(estep_ll_parts(nrows));
    if (nrows > 0) {
      if constexpr (sizeof(T) == 4) {
        if (use_router) {
          router_default_posteriors(X + row0 * D, nrows, m, q, s);
          if (flags & 4) {  // FAST: one-hot of each row's arg-max
            VLB_LAUNCH("exact_onehot", s,
                       k_onehot<<<grid1(nrows, 8), kThreads, 0, s>>>(q, nrows, (int)K));
          }
        } else {
          exact_estep(X + row0 * D, nrows, m, der, q, llp, (flags & 4) != 0, s);
        }
      } else {
        exact_estep(X + row0 * D, nrows, m, der, q, llp, (flags & 4) != 0, s);
      }
    }

    Segment *dsegs = sc.slot[5].get<Segment>(nseg);
    int *dbeg = sc.slot[6].get<int>(nimg + 1);
    i64 *drows = sc.slot[7].get<i64>(nimg);
    double *pu = sc.slot[8].get<double>(nseg * K * D);
    double *pv = sc.slot[9].get<double>(nseg * K * D);
    unsigned long long *pnt = sc.slot[14].get<unsigned long long>(nseg * K);
    VLB_CUDA(cudaMemcpyAsync(dsegs, segs.data(), sizeof(Segment) * nseg, cudaMemcpyHostToDevice, s));
    VLB_CUDA(cudaMemcpyAsync(dbeg, segBegin.data(), sizeof(int) * (nimg + 1), cudaMemcpyHostToDevice, s));
    VLB_CUDA(cudaMemcpyAsync(drows, rows.data(), sizeof(i64) * nimg, cudaMemcpyHostToDevice, s));
    SparseStatsArgs<T> a{};
    a.X = X; a.q = q; a.qbase = row0; a.K = (int)K; a.D = (int)D; a.segs = dsegs;
    a.mu = m.means; a.sis = der.sis; a.priors = m.priors; a.p1 = pu; a.p2 = pv; a.pnt = pnt;
    bool sparse = false;
    if (D <= 128) VLB_LAUNCH("exact_fisher_stats", s, sparse = launch_stats_sparse<kSpFisher>(a, nseg, s));
    if (!sparse) {
      dim3 g((unsigned)nseg, grid1(K, TKC), grid1(D, DB));
      VLB_LAUNCH("exact_fisher_stats", s,
                 (k_fisher_stats<T, TKC, RC, JMAX><<<g, kThreads, 0, s>>>(
                     X, q, row0, (int)K, (int)D, dsegs, m.means, der.sis, m.priors, pu, pv, pnt)));
    }
    VLB_LAUNCH("exact_fisher_finalize", s,
               launch_fisher_finalize<T>(nimg, K, D, dbeg, drows, pu, pv, pnt, m.priors, flags, chunkImg0, enc,
                                         nterms, s));
  }
}

namespace {
constexpr i64 kFixedSegRows = 2048;

// Segment tables of one image, written on the device so a call needs no
// host-to-device copy.
__global__ void k_single_segments(i64 N, i64 nseg, Segment *segs, int *segBegin, i64 *rows) {
  for (i64 j = threadIdx.x; j < nseg; j += blockDim.x) {
    const i64 a = j * kFixedSegRows;
    segs[j] = Segment{0, a, a + kFixedSegRows < N ? a + kFixedSegRows : N};
  }
  if (threadIdx.x == 0) {
    segBegin[0] = 0;
    segBegin[1] = (int)nseg;
    rows[0] = N;
  }
}
}  // namespace

i64 exact_fv_segments(i64 N) { return N > 0 ? (N + kFixedSegRows - 1) / kFixedSegRows : 1; }

void exact_fisher_single_fixed(const float *X, i64 N, const DevModel<float> &m, float *enc,
                               unsigned long long *nterms, int flags, const ExactFvScratch &sc,
                               cudaStream_t s) {
  const i64 K = m.K, D = m.D, nseg = exact_fv_segments(N);  // D <= 128 here
  VLB_LAUNCH_PLAIN(s, k_single_segments<<<1, 32, 0, s>>>(N, nseg, sc.segs, sc.segBegin, sc.rows));
  VLB_LAUNCH_PLAIN(s, k_prepare<float><<<prepare_grid<float>(K), 128, 0, s>>>(
                          m.priors, m.means, m.covs, (int)K, (int)D, half_dim_log_2pi<float>(D), nullptr,
                          sc.cst, sc.sis, sc.img));
  if (N > 0)  // numClusters <= 256 here: one kernel
    VLB_LAUNCH_PLAIN(s, launch_estep<float>(X, N, D, K, sc.img, sc.cst, sc.q, (flags & 4) != 0, nullptr, s));
  SparseStatsArgs<float> a{};
  a.X = X; a.q = sc.q; a.qbase = 0; a.K = (int)K; a.D = (int)D; a.segs = sc.segs;
  a.mu = m.means; a.sis = sc.sis; a.priors = m.priors; a.p1 = sc.pu; a.p2 = sc.pv; a.pnt = sc.pnt;
  VLB_LAUNCH_PLAIN(s, launch_stats_sparse<kSpFisher>(a, nseg, s));
  VLB_LAUNCH_PLAIN(s, launch_fisher_finalize<float>(1, K, D, sc.segBegin, sc.rows, sc.pu, sc.pv, sc.pnt, m.priors,
                                                    flags, 0, enc, nterms, s));
}

// ------------------------------------------------- Rand initialisation
// The reference's Rand initialisation (vl/gmm.c:1376-1443, vl/kmeans.c:
// 588-649) reproduced operation for operation: every sum runs in the data
// type and in the reference's order, multiplies and adds stay separate (the
// explicitly rounded intrinsics of exact_math.cuh never contract into a fused
// multiply-add), so the centres and variances are the reference's bits.

// Global data variance, vl/gmm.c:1376-1413: per dimension the mean, then the
// sum of squared deviations, each accumulated over the rows in order and
// divided by N and N - 1 (0 when N <= 1).  A block takes 32 dimensions: one
// warp adds, a lane per dimension, out of a shared-memory ring of row tiles
// that the other warps fill asynchronously several tiles ahead.  Bound by the
// addition's latency, two chains of N additions: 100,000 rows take 0.76 ms
// of 64 dimensions (a thread per dimension reading the rows from memory: 5.35).
constexpr int kGvStages = 4, kGvUnroll = 32;
template <typename T>
__host__ __device__ constexpr int gv_rows() { return 1024 / (int)sizeof(T); }  // rows per tile

// A shared-memory load that stays where it is written.
__device__ __forceinline__ float ld_volatile(const float *p) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(tc::smem_u32(p)));
  return v;
}
__device__ __forceinline__ double ld_volatile(const double *p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(tc::smem_u32(p)));
  return v;
}

// n rows of a tile added to acc: the values, or with SQ their squared
// deviations from mean.
template <bool SQ, typename T>
__device__ __forceinline__ T gv_add(T acc, T mean, const T *__restrict__ src, int n) {
  auto term = [&](T x) {
    if constexpr (!SQ) return x;
    const T diff = sub_rn(x, mean);
    return mul_rn(diff, diff);
  };
  int r = 0;
  // A group's loads beside the additions of the group before, in a loop short
  // enough for the instruction cache.
  if (n >= kGvUnroll) {
    T v[kGvUnroll];
#pragma unroll
    for (int u = 0; u < kGvUnroll; ++u) v[u] = ld_volatile(src + u * 32);
#pragma unroll 1
    for (r = kGvUnroll; r + kGvUnroll <= n; r += kGvUnroll) {
#pragma unroll
      for (int u = 0; u < kGvUnroll; ++u) {
        acc = add_rn(acc, term(v[u]));
        v[u] = ld_volatile(src + (r + u) * 32);
      }
    }
#pragma unroll
    for (int u = 0; u < kGvUnroll; ++u) acc = add_rn(acc, term(v[u]));
  }
  for (; r < n; ++r) acc = add_rn(acc, term(src[r * 32]));
  return acc;
}

// VB: bytes per asynchronous copy (16 when rows are whole 16-byte pieces).
template <typename T, int VB>
__global__ void __launch_bounds__(256) k_global_variance(const T *__restrict__ X, i64 N, int D, T *__restrict__ sigma) {
  extern __shared__ __align__(16) unsigned char gv_smem[];
  constexpr int VE = VB / (int)sizeof(T), PR = 32 / VE;  // pieces per tile row
  T *ring = (T *)gv_smem;  // [stage][row][32]
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int d = blockIdx.x * 32 + lane;
  if (N <= 1) {
    if (w == 0 && d < D) sigma[d] = (T)0;
    return;
  }
  constexpr int R = gv_rows<T>();
  const int nt = (int)((N + R - 1) / R);  // tiles of one pass over the rows
  const int dc = blockIdx.x * 32 + lane % PR * VE;
  int jt = 0, js = 0;  // the next tile to copy, of two passes, and its stage
  i64 jr = 0;          // its first row
  auto issue = [&]() {
    if (jt < 2 * nt) {
      T *dst = ring + js * R * 32 + lane % PR * VE;
      for (int r = (w - 1) * (32 / PR) + lane / PR; r < R; r += 7 * (32 / PR)) {
        const bool in = jr + r < N && dc < D;
        cp_async_piece<VB>(tc::smem_u32(dst + r * 32), in ? X + (jr + r) * D + dc : X, in);
      }
    }
    cp_async_commit();
    ++jt;
    js = js + 1 == kGvStages ? 0 : js + 1;
    jr = jt == nt ? 0 : jr + R;
  };
  if (w > 0) {
    for (int t = 0; t < kGvStages - 1; ++t) issue();
    for (int t = 0; t < 2 * nt; ++t) {
      cp_async_wait<kGvStages - 2>();
      __syncthreads();  // tile t has landed; the adding warp is done with tile t - 1
      issue();
    }
    return;
  }
  T mean = (T)0, acc = (T)0;
  int st = 0;
  auto tile = [&]() {
    __syncthreads();
    const T *src = ring + st * R * 32 + lane;
    st = st + 1 == kGvStages ? 0 : st + 1;
    return src;
  };
  const int last = (int)(N - (i64)(nt - 1) * R);  // rows of the last tile
  for (int t = 0; t < nt; ++t) acc = gv_add<false>(acc, mean, tile(), t + 1 < nt ? R : last);
  mean = div_rn(acc, (T)N);
  acc = (T)0;
  for (int t = 0; t < nt; ++t) acc = gv_add<true>(acc, mean, tile(), t + 1 < nt ? R : last);
  if (d < D) sigma[d] = div_rn(acc, (T)(N - 1));
}

// minDist[x] = min(minDist[x], ||c - x||^2) with the reference's VL_MIN, c the
// row *xDev (or xHost when xDev is null, the first centre, whose distances
// start minDist); block 0 copies the row to dst.  A row per thread, read 16
// bytes at a time when VEC (D a multiple of 16 bytes, aligned data).
template <typename T, int L, bool VEC>
__global__ void __launch_bounds__(kThreads) k_kpp_update(const T *__restrict__ X, i64 N, int D,
                                                         const i64 *__restrict__ xDev, i64 xHost, T *__restrict__ dst,
                                                         T *__restrict__ minDist) {
  extern __shared__ __align__(16) unsigned char kpp_smem[];
  T *c = (T *)kpp_smem;
  const i64 row = xDev ? *xDev : xHost;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const T v = X[row * D + d];
    c[d] = v;
    if (blockIdx.x == 0) dst[d] = v;
  }
  __syncthreads();
  const i64 x = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= N) return;
  T dist;
  if constexpr (VEC) {
    // l2_ordered's lane sums with the row in registers one group at a time.
    constexpr int VE = 16 / (int)sizeof(T);
    using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
    constexpr int G = L > VE ? L : VE;  // elements per step: whole lane groups and whole vectors
    T v[L];
#pragma unroll
    for (int l = 0; l < L; ++l) v[l] = (T)0;
    const T *xr = X + x * D;
    int i = 0;
#pragma unroll 4
    for (; i + G <= D; i += G) {
#pragma unroll
      for (int g = 0; g < G / VE; ++g) {
        const V w = __ldg((const V *)(xr + i) + g);
        const T *wp = (const T *)&w;
#pragma unroll
        for (int e = 0; e < VE; ++e) {
          const T dl = sub_rn(c[i + g * VE + e], wp[e]);
          v[(g * VE + e) % L] = add_rn(v[(g * VE + e) % L], mul_rn(dl, dl));
        }
      }
    }
    dist = l2_ordered_tail<T, L>(v, c, 1, xr, i, D);
  } else {
    dist = l2_ordered<T, L>(c, X + x * D, D);
  }
  if (!xDev) {
    minDist[x] = dist;
  } else {
    const T m = minDist[x];
    minDist[x] = m < dist ? m : dist;
  }
}

constexpr int kKppStages = 4;

// The next centre, vl/kmeans.c:631-641: the energy (sum of minDist in order),
// then the first x whose prefix sum is >= thresh * energy, or N - 1 (a NaN
// energy fails every test).  The prefixes are the energy's own, so the energy
// pass keeps one per tile (8192 terms, 4096 in double) and only the tile that holds the answer
// is scanned again.  One block: 100,000 terms take 28 us, 1 M 138 us; a
// thread that adds in order takes 290 and 2,900 (7 clocks a term).
template <typename T>
__global__ void __launch_bounds__(kSeqThreads) k_kpp_select(const T *__restrict__ minDist, i64 N, T thresh,
                                                            T *__restrict__ ck, i64 *__restrict__ xOut) {
  constexpr int EPT = seq_ept<T>(), kTile = seq_tile<T>();
  __shared__ SeqShared<T> sh;
  __shared__ int s_tile;
  extern __shared__ __align__(16) unsigned char kps_smem[];
  constexpr int VE = 16 / (int)sizeof(T), P = EPT + VE;  // a thread's terms and 16 bytes, so that its reads spread over the banks
  T *ring = (T *)kps_smem;                               // [stage][thread][P]
  const int tid = threadIdx.x;
  const i64 ntile = (N + kTile - 1) / kTile;
  int pb = 0;
  // Terms of a tile to its stage, zeros past the end; and this thread's terms from there.
  auto issue = [&](i64 tile, int stage) {
    if (tile < ntile)
#pragma unroll
      for (int u = 0; u < kTile / VE / kSeqThreads; ++u) {
        const int e = (u * kSeqThreads + tid) * VE;
        const i64 i = tile * kTile + e;
        const i64 left = N - i;
        const uint32_t bytes = left >= VE ? 16u : left > 0 ? (uint32_t)(left * (i64)sizeof(T)) : 0u;
        cp_async16(tc::smem_u32(ring + ((size_t)stage * kSeqThreads + e / EPT) * P + e % EPT),
                   bytes ? minDist + i : minDist, bytes);
      }
    cp_async_commit();
  };
  auto load = [&](int stage, T(&v)[EPT]) {
    const T *src = ring + ((size_t)stage * kSeqThreads + tid) * P;
#pragma unroll
    for (int u = 0; u < EPT; u += VE) {
      using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
      const V x = *(const V *)(src + u);
#pragma unroll
      for (int e = 0; e < VE; ++e) v[u + e] = ((const T *)&x)[e];
    }
  };
  T v[EPT];
  T acc = (T)0;
  for (int t = 0; t < kKppStages - 1; ++t) issue(t, t);
  for (i64 tile = 0; tile < ntile; ++tile) {
    cp_async_wait<kKppStages - 2>();
    __syncthreads();  // the tile has landed; every thread has read the one before
    load((int)(tile % kKppStages), v);
    issue(tile + kKppStages - 1, (int)((tile + kKppStages - 1) % kKppStages));
    seq_add<T, false>(v, acc, (T)0, 0, sh, pb);
    if (tid == 0) ck[tile] = acc;
  }
  cp_async_wait<0>();
  // The first tile whose last prefix reaches the threshold.
  const T t = mul_rn(thresh, acc);
  if (tid == 0) s_tile = 0x7fffffff;
  __syncthreads();
  for (i64 j = tid; j < ntile; j += kSeqThreads)
    if (ck[j] >= t) {
      atomicMin(&s_tile, (int)j);
      break;
    }
  __syncthreads();
  const int tile = s_tile;
  if (tile == 0x7fffffff) {
    if (tid == 0) *xOut = N - 1;
    return;
  }
  acc = tile > 0 ? ck[tile - 1] : (T)0;
  issue(tile, 0);
  cp_async_wait<0>();
  __syncthreads();
  load(0, v);
  const bool found = seq_add<T, true>(v, acc, t, (i64)tile * kTile, sh, pb);
  if (tid == 0) *xOut = found ? min((i64)sh.x, N - 1) : N - 1;
}

template <typename T>
__global__ void k_kpp_copy(const T *__restrict__ X, int D, const i64 *__restrict__ xDev, i64 xHost,
                           T *__restrict__ dst) {
  const i64 x = xDev ? *xDev : xHost;
  for (int d = threadIdx.x; d < D; d += blockDim.x) dst[d] = X[x * D + d];
}

template <typename T>
void global_variance(const T *X, i64 N, i64 D, T *sigma, cudaStream_t s) {
  constexpr size_t smem = sizeof(T) * kGvStages * gv_rows<T>() * 32;
  const bool vec = D % (16 / (i64)sizeof(T)) == 0 && ((uintptr_t)X & 15) == 0;
  auto kern = vec ? k_global_variance<T, 16> : k_global_variance<T, (int)sizeof(T)>;
  VLB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  VLB_LAUNCH("global_variance", s, kern<<<grid1(D, 32), 256, smem, s>>>(X, N, (int)D, sigma));
}

namespace {
template <typename T, int L>
void launch_kpp_update(const T *X, i64 N, i64 D, const i64 *xDev, i64 x0, T *dst, T *minDist, cudaStream_t s) {
  const bool vec = D % (16 / (i64)sizeof(T)) == 0 && ((uintptr_t)X & 15) == 0;
  auto kern = vec ? k_kpp_update<T, L, true> : k_kpp_update<T, L, false>;
  VLB_LAUNCH("kpp_update", s, kern<<<grid1(N, kThreads), kThreads, sizeof(T) * D, s>>>(X, N, (int)D, xDev, x0, dst, minDist));
}
}  // namespace

template <typename T>
void kmeanspp(const T *X, i64 N, i64 D, i64 K, T *centers, i64 x0, const std::vector<T> &thresh, int lanes,
              cudaStream_t s) {
  VLB_CHECK((i64)thresh.size() >= K && N > 0 && K > 0 && x0 >= 0 && x0 < N, VL_ERR_BAD_ARG,
            "kmeans++: bad arguments");
  Scratch &sc = thread_scratch(kArenaExact);
  T *minDist = sc.slot[20].get<T>(N);
  i64 *xdev = sc.slot[21].get<i64>(1);
  T *ck = sc.slot[22].get<T>(N / seq_tile<T>() + 1);
  constexpr size_t ssmem = (size_t)kKppStages * kSeqThreads * (seq_ept<T>() * sizeof(T) + 16);
  VLB_CUDA(cudaFuncSetAttribute(k_kpp_select<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssmem));
  for (i64 c = 0; c < K; ++c) {
    const i64 *xp = c == 0 ? nullptr : xdev;
    if (c + 1 == K) {
      VLB_LAUNCH("kpp_copy", s, k_kpp_copy<T><<<1, 128, 0, s>>>(X, (int)D, xp, x0, centers + c * D));
      break;
    }
    switch (lanes) {
      case 8: launch_kpp_update<T, 8>(X, N, D, xp, x0, centers + c * D, minDist, s); break;
      case 4: launch_kpp_update<T, 4>(X, N, D, xp, x0, centers + c * D, minDist, s); break;
      case 2: launch_kpp_update<T, 2>(X, N, D, xp, x0, centers + c * D, minDist, s); break;
      default: launch_kpp_update<T, 1>(X, N, D, xp, x0, centers + c * D, minDist, s); break;
    }
    VLB_LAUNCH("kpp_select", s, k_kpp_select<T><<<1, kSeqThreads, ssmem, s>>>(minDist, N, thresh[c], ck, xdev));
  }
}

// ------------------------------------------------------ instantiations
#define VLB_INST(T)                                                                          \
  template void exact_prepare<T>(const DevModel<T> &, DevDerived<T> &, cudaStream_t);        \
  template size_t exact_image_elems<T>(i64, i64);                                            \
  template i64 exact_estep<T>(const T *, i64, const DevModel<T> &, const DevDerived<T> &,    \
                              T *, double *, bool, cudaStream_t);                            \
  template void exact_mstep<T>(const T *, i64, const T *, T *, T *, T *, i64, i64,           \
                               const double *, cudaStream_t);                                \
  template void column_mass<T>(const T *, i64, i64, double *, cudaStream_t);                 \
  template void exact_mstep_stats_rows<T>(const T *, i64, i64, i64, const T *, const T *, i64, i64, \
                                          double *, double *, double *, cudaStream_t);       \
  template void exact_mstep_finalize_slabs<T>(int, const double *, const double *, const double *, \
                                              const double *, T *, T *, T *, i64, i64, cudaStream_t); \
  template void normalize_priors<T>(T *, i64, cudaStream_t);                                 \
  template void global_variance<T>(const T *, i64, i64, T *, cudaStream_t);                  \
  template void kmeanspp<T>(const T *, i64, i64, i64, T *, i64, const std::vector<T> &, int,  \
                            cudaStream_t);                                                   \
  template void restart_split<T>(T *, const T *, i64, i64, i64, i64, i64, i64, T,           \
                                 cudaStream_t);                                              \
  template void apply_bounds<T>(T *, i64, i64, const double *, cudaStream_t);                \
  template void exact_fisher_batch<T>(const T *, const i64 *, i64, const DevModel<T> &, T *, \
                                      unsigned long long *, int, cudaStream_t, bool);
VLB_INST(float)
VLB_INST(double)

}  // namespace vlb
