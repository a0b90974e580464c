// Batched propagation with vectors per lane group by mesh.
#include "mg_batched_small.cuh"

namespace mg {
cudaError_t batched_small_fwd(const LaunchCfg& lc, const BatchedSmall& b) { return launch_batched_small<OP_FWD>(lc, b); }
}  // namespace mg
