// Near-field instances of the summation by transforms.
#include "sr_fast_sum.cuh"

namespace sr {

int launch_uneven_near(const FarMixedParams &p, int n_sm, cudaStream_t s) {
  return launch_uneven<true>(p, n_sm, s);
}

int launch_fast_near(const FarMixedParams &p, const FastLayout &l, cudaStream_t s) {
  return launch_fast<true>(p, l, s);
}

}  // namespace sr
