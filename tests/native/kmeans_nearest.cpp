// first_at_distance (csrc/qcp_kmeans.cuh) on the host: prints, for the object
// (0, 0) and the centres (k, 0), the centre found in [ka, kb) at the distance
// given, for every argument "ka kb distance".
#include <cuda_runtime.h>

#include <cstdio>

#include "qcp_kmeans.cuh"

int main() {
  constexpr uint32_t K = 20;
  float centres[2 * K];
  // centres 3 and 5 are the same
  for (uint32_t k = 0; k < K; ++k) centres[k] = k == 5 ? 3.f : (float)k, centres[K + k] = 0.f;
  const float x[2] = {0.f, 0.f};
  unsigned ka, kb;
  float best;
  while (scanf("%u %u %f", &ka, &kb, &best) == 3)
    printf("%u\n", qcp::first_at_distance<2>(x, centres, K, ka, kb, best));
  return 0;
}
