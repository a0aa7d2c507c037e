// Device helpers on sinogram bins shared by the kernels' translation units:
// bin numbers, count loads, the likelihood term, block sums.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "internal.h"
#include "../../include/apirl_b200.h"

namespace apirl {

struct BinPos {
  int g, k, l, a;  // sinogram, subset angle, r, full angle
};

__device__ __forceinline__ BinPos decode(int64_t b, const LorTable& t, const SubsetSel& s) {
  BinPos p;
  const int64_t per = (int64_t)s.nk * t.n_r;
  const int gl = (int)(b / per);  // sinogram within the shard
  const int rem = (int)(b - (int64_t)gl * per);
  p.g = t.g0 + gl;
  p.k = rem / t.n_r;
  p.l = rem - p.k * t.n_r;
  p.a = s.subset < 0 ? p.k : s.subset + s.nsub * p.k;
  return p;
}

template <typename CT> __device__ __forceinline__ float load_count(const CT* p, int64_t i);
template <> __device__ __forceinline__ float load_count<float>(const float* p, int64_t i) { return __ldg(p + i); }
template <> __device__ __forceinline__ float load_count<uint32_t>(const uint32_t* p, int64_t i) {
  return (float)__ldg(p + i);
}
template <> __device__ __forceinline__ float load_count<uint16_t>(const uint16_t* p, int64_t i) {
  return (float)__ldg(p + i);
}

// A walked bin's likelihood term (Sinogram3D::getLikelihoodValue,
// data/src/Sinogram3D.cpp:584-606: m log e - e over e != 0).  skip_zero:
// 0 = every bin walked; 1 = zero-count bins not walked, their -e supplied by
// -x . Z_s (Z_s = A_s^T 1[m == 0]); 2 = zero-count bins not walked and the
// -e of every bin supplied by -x . G_s - sum(add) (G_s = A_s^T 1, a
// geometry image), so a walked bin adds m log e alone.
__device__ __forceinline__ double lik_term(float m, float e, int skip_zero) {
  return skip_zero == 2 ? (double)m * log((double)e) : (double)m * log((double)e) - (double)e;
}

__device__ __forceinline__ float load_count_any(const void* p, int dtype, int64_t i) {
  if (dtype == APIRL_U32) return (float)__ldg((const uint32_t*)p + i);
  if (dtype == APIRL_U16) return (float)__ldg((const uint16_t*)p + i);
  return __ldg((const float*)p + i);
}

// The last of n entries whose first (block, tile or chunk) key(e) is <= k;
// entries are ordered by key.
template <typename J, class Key>
__device__ __forceinline__ int find_entry(const J* __restrict__ e, int n, int64_t k, Key key) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (key(e[mid]) <= k) lo = mid; else hi = mid - 1;
  }
  return lo;
}

}  // namespace apirl
