// A sequential floating-point sum of non-negative terms, formed in parallel with
// the bits of the loop that adds them in order.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "exact_math.cuh"

namespace vlb {

// The sum acc = rn(acc + v_i), in order, of non-negative terms: while acc stays
// in one binade [2^e, 2^(e+1)) it is an integer A times the binade's ulp u, and
// an addition adds to A the term rounded to a multiple of u; only an exact tie
// depends on acc, through A's parity (round half to even).  So a run of terms
// maps A's parity to an increment, such maps compose associatively, and a
// block scans them; the term that takes acc past the binade (or is not a
// finite non-negative number) is added by its thread as it is, and the scan
// goes on from there with the next binade.  Zero and subnormal acc count as
// the lowest binade, whose ulp they share.  Every prefix has the bits of the
// loop's.
template <typename T>
struct SeqFloat;
template <>
struct SeqFloat<float> {
  using U = uint32_t;
  static constexpr int kMant = 23, kExpMax = 255;
  static __device__ __forceinline__ U bits(float v) { return __float_as_uint(v); }
  static __device__ __forceinline__ float value(U b) { return __uint_as_float(b); }
};
template <>
struct SeqFloat<double> {
  using U = unsigned long long;
  static constexpr int kMant = 52, kExpMax = 2047;
  static __device__ __forceinline__ U bits(double v) { return (U)__double_as_longlong(v); }
  static __device__ __forceinline__ double value(U b) { return __longlong_as_double((long long)b); }
};
template <typename T>
struct Seq {
  using F = SeqFloat<T>;
  using U = typename F::U;
  static constexpr U kOne = (U)1 << F::kMant, kLim = kOne * 2, kSat = kOne * 4;
  // A map is 4 i + (d + 1): i is the increment of an even A (at most kSat), d in
  // {-1, 0, 1} how much more an odd A gains.  (A tie sends one of the two
  // starts up and the other down; from then on both have the same parity, so
  // d stays.)
  static constexpr U kIdentity = 1;
  static __device__ __forceinline__ U pack(U i, int d) { return ((i < kSat ? i : kSat) << 2) | (U)(d + 1); }
  static __device__ __forceinline__ int diff(U m) { return (int)(m & 3) - 1; }
  static __device__ __forceinline__ U gain(U m, bool odd) { return (m >> 2) + (U)(odd ? diff(m) : 0); }
  static __device__ __forceinline__ U then(U a, U b) {
    const bool odd = ((a >> 2) & 1) != 0;
    const int da = diff(a), db = diff(b);
    return pack((a >> 2) + gain(b, odd), da ? da : odd ? -db : db);
  }
  // Biased exponent (at least 1) and integer of a finite non-negative value.
  static __device__ __forceinline__ int exponent(U b) { return max(1, (int)(b >> F::kMant)); }
  static __device__ __forceinline__ U integer(U b) { return (b & (kOne - 1)) | (b >> F::kMant ? kOne : (U)0); }
  static __device__ __forceinline__ T value(int be, U A) {
    return F::value(A < kOne ? A : ((U)be << F::kMant) + (A - kOne));  // A < kOne only in the lowest binade
  }
  // The map of a run of terms, acc in the binade with biased exponent be: the
  // run added to the binade's first value (an even A) and to the next (odd).
  // A sum that leaves the binade, or is not a number, saturates: whatever A it
  // starts from, its thread adds the terms as they are.
  template <int EPT>
  static __device__ __forceinline__ U run(const T (&v)[EPT], int be) {
    const U b0 = (U)be << F::kMant;
    T x0 = F::value(b0), x1 = F::value(b0 + 1);
    const T lim = add_rn(x0, x0);
#pragma unroll
    for (int u = 0; u < EPT; ++u) {
      x0 = add_rn(x0, v[u]);
      x1 = add_rn(x1, v[u]);
    }
    if (!(x0 < lim && x1 < lim && x0 >= F::value(b0))) return pack(kSat, 0);
    const U i = F::bits(x0) - b0;
    return pack(i, (int)(F::bits(x1) - b0 - 1 - i));
  }
};

constexpr int kSeqThreads = 256;  // threads of a block that adds a tile
template <typename T>
__host__ __device__ constexpr int seq_ept() { return 128 / (int)sizeof(T); }  // terms per thread and tile
template <typename T>
__host__ __device__ constexpr int seq_tile() { return kSeqThreads * seq_ept<T>(); }

template <typename T>
struct SeqShared {
  typename Seq<T>::U warp[2][kSeqThreads / 32];
  T acc;
  int next;
  long long x;
};

// Inclusive scan of the maps over the first `width` lanes of a warp.
template <typename T>
__device__ __forceinline__ typename Seq<T>::U seq_scan(typename Seq<T>::U m, int width) {
  using S = Seq<T>;
  using U = typename S::U;
  const int lane = threadIdx.x % 32;
  if (!__any_sync(0xffffffffu, S::diff(m) != 0)) {  // no ties: plain saturating sums
    U i = m >> 2;
#pragma unroll
    for (int o = 1; o < width; o <<= 1) {
      const U p = __shfl_up_sync(0xffffffffu, i, o);
      if (lane >= o) i = min(i + p, S::kSat);
    }
    return S::pack(i, 0);
  }
#pragma unroll
  for (int o = 1; o < width; o <<= 1) {
    const U p = __shfl_up_sync(0xffffffffu, m, o);
    if (lane >= o) m = S::then(p, m);
  }
  return m;
}

// Adds a tile's terms (thread i's are terms seq_ept i ..) to acc, which all
// threads of the block hold alike.  With FIND it stops at the first prefix >= t
// and returns true, sh.x the term's index plus base.  pb, kept by the caller
// across calls, is the buffer of warp totals: a pass writes the one that the
// pass before did not.
template <typename T, bool FIND>
__device__ __forceinline__ bool seq_add(const T (&v)[seq_ept<T>()], T &acc, T t, long long base, SeqShared<T> &sh,
                                        int &pb) {
  using S = Seq<T>;
  using U = typename S::U;
  constexpr int NW = kSeqThreads / 32, EPT = seq_ept<T>();
  const int tid = threadIdx.x, lane = tid % 32, w = tid / 32;
  int from = 0;  // first thread whose terms are not in acc
  while (from < kSeqThreads) {
    if (!(acc < (T)INFINITY)) {
      // NaN stays; infinity turns into NaN at a NaN or -infinity.
      bool nan = false;
#pragma unroll
      for (int u = 0; u < EPT; ++u) nan |= tid >= from && !(v[u] > -(T)INFINITY);
      if (__syncthreads_or(nan)) acc = add_rn(acc, (T)NAN);
      return false;
    }
    const U ab = S::F::bits(acc), A = S::integer(ab);
    const int be = S::exponent(ab);
    const bool odd = (A & 1) != 0;
    const U m = seq_scan<T>(tid >= from ? S::run(v, be) : S::kIdentity, 32);
    if (lane == 31) sh.warp[pb][w] = m;
    __syncthreads();
    const U x = seq_scan<T>(lane < NW ? sh.warp[pb][lane] : S::kIdentity, NW);  // inclusive over the warps, in every warp
    pb ^= 1;
    auto stops = [&](U end) { return end >= S::kLim || (FIND && S::value(be, end) >= t); };
    const unsigned at = __ballot_sync(0xffffffffu, lane < NW && stops(A + S::gain(x, odd)));
    if (!at) {
      acc = S::value(be, A + S::gain(__shfl_sync(0xffffffffu, x, NW - 1), odd));
      return false;
    }
    // The first thread whose terms leave the binade (or reach t) adds them.
    const U before = __shfl_sync(0xffffffffu, x, max(w - 1, 0));
    if (w == __ffs(at) - 1) {
      const U prev = w > 0 ? before : S::kIdentity;
      const U incl = S::then(prev, m), up = __shfl_up_sync(0xffffffffu, incl, 1);
      const unsigned in = __ballot_sync(0xffffffffu, stops(A + S::gain(incl, odd)));
      if (lane == __ffs(in) - 1) {
        T y = S::value(be, A + S::gain(lane > 0 ? up : prev, odd));
        long long hit = -1;
#pragma unroll
        for (int u = 0; u < EPT; ++u) {
          y = add_rn(y, v[u]);
          if (FIND && hit < 0 && y >= t) hit = base + tid * EPT + u;
        }
        sh.acc = y;
        sh.next = tid + 1;
        sh.x = hit;
      }
    }
    __syncthreads();
    acc = sh.acc;
    from = sh.next;
    if (FIND && sh.x >= 0) return true;
  }
  return false;
}

}  // namespace vlb
