// Launches of the batched kernels with vectors per lane group by mesh (mg_batched_small.cuh), one translation unit per op.
#pragma once
#include "../../include/meshes_gb300.h"
#include "mg_launch.h"

namespace mg {

constexpr int kSmallWarps = 8;
struct BatchedSmall {
  const mg_batch_framed* meshes;
  int n_meshes;
  const mg_batch_item* items;
  int n_items;
  int* head;
  int* status;
};
cudaError_t batched_small_fwd(const LaunchCfg& lc, const BatchedSmall& b);
cudaError_t batched_small_bwd(const LaunchCfg& lc, const BatchedSmall& b);

}  // namespace mg
