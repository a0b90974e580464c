// Launch of one framed instantiation (included by the mg_prop_framed_*.cu units).
#pragma once
#include "mg_framed.cuh"
#include "mg_launch.h"

namespace mg {

template <int OP, int M, int V, int GT, bool MIX>
cudaError_t launch_one_framed(const LaunchCfg& lc, const FramedArgs& a) {
  static std::atomic<unsigned long long> done{0};
  auto k = framed_kernel<OP, M, V, GT, MIX>;
  const cudaError_t e = ensure_smem_attr(k, done);
  if (e != cudaSuccess) return e;
  k<<<lc.grid, lc.block, lc.smem, lc.stream>>>(a);
  return cudaGetLastError();
}

}  // namespace mg

// the launches of one unit: X(M, V, mixed warps)
#define MG_FRAMED_UNIT(NAME, OP, LIST)                                                                \
  namespace mg {                                                                                      \
  cudaError_t NAME(int M, int V, bool mix, const LaunchCfg& lc, const FramedArgs& a) {                \
    LIST(MG_FRAMED_CASE_##OP)                                                                         \
    return cudaErrorInvalidConfiguration;                                                             \
  }                                                                                                   \
  }
#define MG_FRAMED_CASE_OP_FWD(M_, V_, MIX_) \
  if (M == M_ && V == V_ && mix == MIX_) return launch_one_framed<OP_FWD, M_, V_, 32, MIX_>(lc, a);
#define MG_FRAMED_CASE_OP_BWD(M_, V_, MIX_) \
  if (M == M_ && V == V_ && mix == MIX_) return launch_one_framed<OP_BWD, M_, V_, 32, MIX_>(lc, a);
