// The scalar half of the k-means assignment, for host and device.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace qcp {

// The first of the centres [ka, kb) whose squared distance from x, evaluated
// term by term without contraction, is `best`, which another evaluation found
// to be the least of theirs.  The two agree by the rules of rounding; where a
// compiler made them differ the answer is ka, so that it is a centre whatever
// `best` is.
template <int D>
__host__ __device__ __forceinline__ uint32_t first_at_distance(const float (&x)[D], const float* centres, uint32_t K,
                                                               uint32_t ka, uint32_t kb, float best) {
  for (uint32_t k = ka; k < kb; ++k) {
    float dist = 0.f;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int d = 0; d < D; ++d) {
#ifdef __CUDA_ARCH__
      const float t = __fsub_rn(x[d], __ldg(centres + (uint64_t)d * K + k));
      dist = __fadd_rn(dist, __fmul_rn(t, t));
#else
      const float t = x[d] - centres[(uint64_t)d * K + k], s = t * t;
      dist = dist + s;
#endif
    }
    if (dist == best) return k;
  }
  return ka;
}

}  // namespace qcp
