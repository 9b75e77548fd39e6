// The reference's momentum stream (main.h:207-213): a fresh Thrust engine advanced by n, one N(0,1) draw.  Thrust's
// own code does the work, as it does in the reference.
#pragma once
#include <thrust/random.h>

namespace mcmc_b200 {

__device__ __forceinline__ float refstream_normal(unsigned long long n) {
  thrust::default_random_engine engine;
  engine.discard(n);
  thrust::normal_distribution<float> unit_normal(0.f, 1.f);
  return unit_normal(engine);
}
constexpr unsigned long long REF_DRAWS_PER_ITER = 962;  // 961 momenta + 1 accept draw (main.h:216,237)

}  // namespace mcmc_b200
