// Sums whose order is part of the result: count values `stride` apart, added one after the other.
// By one thread that is a chain of loads; here a CTA of 256 threads takes LANES sums, all of them
// bring the next (256 / LANES) EACH values of each to shared memory, and one thread a sum adds those.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace sma {

template <int LANES, int EACH>
struct OrderedSum {
  static constexpr int kGroups = 256 / LANES;
  double sh[kGroups * EACH][LANES + 1];

  // p: the first value of the sum of lane threadIdx.x % LANES (null: none).  For all threads of the
  // CTA; the sum is the result of the first LANES of them.
  __device__ __forceinline__ double operator()(const double *p, int64_t stride, int64_t count) {
    const int lane = threadIdx.x % LANES, group = threadIdx.x / LANES;
    double s = 0.0;
    for (int64_t z0 = 0; z0 < count; z0 += kGroups * EACH) {
      const int here = (int)min((int64_t)(kGroups * EACH), count - z0);
      if (p) {
        double v[EACH];
#pragma unroll
        for (int u = 0; u < EACH; ++u) {
          const int z = group + u * kGroups;
          v[u] = z < here ? p[(z0 + z) * stride] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < EACH; ++u) sh[group + u * kGroups][lane] = v[u];
      }
      __syncthreads();
      if (p && group == 0) {
#pragma unroll 8
        for (int z = 0; z < here; ++z) s += sh[z][lane];
      }
      __syncthreads();
    }
    return s;
  }
};

}  // namespace sma
