// Butterfly kernels, op BWD.
#include "mg_fft.cuh"
#include "mg_launch.h"

namespace mg {
namespace {
template <int M, int G>
cudaError_t launch(const LaunchCfg& lc, const FftArgs& a) {
  static std::atomic<unsigned long long> done{0};
  const cudaError_t e = ensure_smem_attr(fft_kernel<OP_BWD, M, G>, done);
  if (e != cudaSuccess) return e;
  fft_kernel<OP_BWD, M, G><<<lc.grid, lc.block, lc.smem, lc.stream>>>(a);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_fft_bwd(const LaunchCfg& lc, const FftArgs& a) {
  switch (a.N) {
    case 64: return launch<8, 8>(lc, a);
    case 128: return launch<16, 8>(lc, a);
    case 256: return launch<16, 16>(lc, a);

    default: return cudaErrorInvalidConfiguration;
  }
}
}  // namespace mg
