// mg_l2_loss: J = sum |y - t|^2 over n floats (complex fields: their real and imaginary parts), the loss whose gradient
// mg_propagate_l2 forms on load.
//
// What bounds it: HBM or L2 for a large batch (8 bytes per float), latency for a small one, which takes one launch of a cluster up to
// kOneCluster floats.  A thread adds its squares in float over 32 values at a time and those sums in double; the
// CTAs' sums are added in order, so J is the same from run to run.  Measured on GB300 against difference, square and sum as
// three passes: N = 256, B = 4096 13.8 -> 8.8 us, N = 128, B = 128 8.7 -> 4.2 us (one CTA: 6.6).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/meshes_gb300.h"
#include "mg_launch.h"

namespace mg {
namespace {

constexpr int kLossThreads = 512;
constexpr int kCluster = 8;
constexpr size_t kOneCluster = 1 << 18;    // floats
constexpr size_t kPerCta = 1 << 14;        // floats per CTA, at least

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double warps[kLossThreads / 32];
  for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kLossThreads / 32; ++w) s += warps[w];
  return s;   // of thread 0
}

// The thread's part of n floats.  VEC: y and t 16-byte aligned, the last n % 4 floats by themselves
template <bool VEC>
__device__ __forceinline__ double l2_part(const float* __restrict__ y, const float* __restrict__ t, size_t n) {
  double sum = 0;
  const size_t first = (size_t)blockIdx.x * kLossThreads + threadIdx.x, step = (size_t)gridDim.x * kLossThreads;
  auto sq = [](float a, float b, float s) {
    const float d = a - b;
    return fmaf(d, d, s);
  };
  if (VEC) {
    const float4* y4 = reinterpret_cast<const float4*>(y);
    const float4* t4 = reinterpret_cast<const float4*>(t);
    const size_t m = n / 4;
    for (size_t i0 = first; i0 < m; i0 += 8 * step) {
      float4 a[8], b[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const size_t i = i0 + k * step;
        a[k] = b[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < m) {
          a[k] = __ldg(y4 + i);
          b[k] = __ldg(t4 + i);
        }
      }
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) s = sq(a[k].w, b[k].w, sq(a[k].z, b[k].z, sq(a[k].y, b[k].y, sq(a[k].x, b[k].x, s))));
      sum += s;
    }
    if (first < n - 4 * m) sum += sq(y[4 * m + first], t[4 * m + first], 0.f);
  } else {
    for (size_t i0 = first; i0 < n; i0 += 8 * step) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const size_t i = i0 + k * step;
        if (i < n) s = sq(y[i], t[i], s);
      }
      sum += s;
    }
  }
  return sum;
}

template <bool VEC>
__global__ void __launch_bounds__(kLossThreads) l2_loss_kernel(const float* __restrict__ y, const float* __restrict__ t, size_t n,
                                                               double* part) {
  const double s = block_sum(l2_part<VEC>(y, t, n));
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// one cluster: the CTAs' sums are added, in order, through distributed shared memory
template <bool VEC>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kLossThreads)
l2_loss_cluster_kernel(const float* __restrict__ y, const float* __restrict__ t, size_t n, float* out) {
  __shared__ double sum;
  auto cluster = cooperative_groups::this_cluster();
  const double s = block_sum(l2_part<VEC>(y, t, n));
  if (threadIdx.x == 0) sum = s;
  cluster.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    double all = 0;
    for (int k = 0; k < kCluster; ++k) all += *cluster.map_shared_rank(&sum, k);
    *out = (float)all;
  }
  cluster.sync();
}

__global__ void __launch_bounds__(kLossThreads) l2_loss_sum_kernel(const double* part, int n, float* out) {
  double v = 0;
  for (int i = threadIdx.x; i < n; i += kLossThreads) v += part[i];
  const double s = block_sum(v);
  if (threadIdx.x == 0) *out = (float)s;
}

}  // namespace
}  // namespace mg

using namespace mg;

extern "C" int mg_l2_loss(const float* y, const float* t, size_t n, float* out, double* scratch, int scratch_doubles,
                          void* stream) {
  if (!out || (n && (!y || !t))) return set_last_error(MG_E_ARG, "mg_l2_loss: NULL argument");
  if ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(t)) & 3) return set_last_error(MG_E_ARG, "mg_l2_loss: fields not 4-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec = ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(t)) & 15) == 0;
  if (n <= kOneCluster || !scratch || scratch_doubles < 1) {
    if (vec) l2_loss_cluster_kernel<true><<<kCluster, kLossThreads, 0, st>>>(y, t, n, out);
    else l2_loss_cluster_kernel<false><<<kCluster, kLossThreads, 0, st>>>(y, t, n, out);
  } else {
    const int grid = (int)std::min<size_t>((n + kPerCta - 1) / kPerCta, scratch_doubles);
    if (vec) l2_loss_kernel<true><<<grid, kLossThreads, 0, st>>>(y, t, n, scratch);
    else l2_loss_kernel<false><<<grid, kLossThreads, 0, st>>>(y, t, n, scratch);
    l2_loss_sum_kernel<<<1, kLossThreads, 0, st>>>(scratch, grid, out);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MG_OK : set_last_error(MG_E_CUDA, "l2_loss_kernel: %s", cudaGetErrorString(e));
}
