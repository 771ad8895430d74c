// Sums of many partials per element in index order (the order fixes the
// rounding), with the loads of 64 partials in flight at a time.
#pragma once
#include <cuda_runtime.h>

namespace vlb {

constexpr int kOrdThreads = 256;  // 8 rows of 32 elements
constexpr int kOrdItems = 64;     // partials staged per round

template <int NV>
struct OrdShared {
  double v[NV][kOrdItems][32];
};

// out[q] = sum over items 0 .. n - 1 of load(item, q), added in item order,
// for this lane's element; valid in every warp.  A block of kOrdThreads
// threads takes 32 elements (the lanes): its eight warps fetch eight items
// each, and warp q adds value q out of shared memory while the next round's
// loads are in flight.  The chain of one thread per element that this replaces
// had a few loads in flight and waited for memory at each group.
template <int NV, typename Load>
__device__ __forceinline__ void ordered_sums(int n, Load load, OrdShared<NV> &sh, double (&out)[NV]) {
  constexpr int W = kOrdThreads / 32, J = kOrdItems / W;
  const int lane = threadIdx.x % 32, y = threadIdx.x / 32;
  double v[J][NV];
  auto fetch = [&](int base) {
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int item = base + y + W * j;
#pragma unroll
      for (int q = 0; q < NV; ++q) v[j][q] = item < n ? load(item, q) : 0.0;
    }
  };
  double s = 0;
  fetch(0);
  for (int base = 0; base < n; base += kOrdItems) {
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
      for (int q = 0; q < NV; ++q) sh.v[q][y + W * j][lane] = v[j][q];
    __syncthreads();
    if (base + kOrdItems < n) fetch(base + kOrdItems);
    if (y < NV) {
      const int cnt = min(kOrdItems, n - base);
#pragma unroll 8
      for (int i = 0; i < cnt; ++i) s += sh.v[y][i][lane];
    }
    __syncthreads();
  }
  if (y < NV) sh.v[y][0][lane] = s;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) out[q] = sh.v[q][0][lane];
}

}  // namespace vlb
