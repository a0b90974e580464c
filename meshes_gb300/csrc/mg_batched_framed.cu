// Batched propagation of meshes on framed tiles: the persistent launch of mg_batched.cu with the framed body
// (mg_framed.cuh) for nearest-neighbour MZI meshes of 129 to 256 modes.
//
// What bounds it: as the one-mesh kernel, the FMA pipe's register operands.  An item is 32 vectors (8 warps of 4), what a
// full wave of the one-mesh kernel gives a CTA; items are drained longest first.
#include "mg_batched_framed.cuh"
#include "mg_batched_small.h"

namespace mg {
namespace {

constexpr int kBFWarps = 8, kBFM = 8, kBFV = 4;

template <int OP>
__global__ void __launch_bounds__(kBFWarps * 32, 1)
batched_framed_kernel(const mg_batch_framed* __restrict__ meshes, int n_meshes, const mg_batch_item* __restrict__ items,
                      int n_items, int* head, int* status) {
  extern __shared__ __align__(128) unsigned char smem[];
  // in shared memory: the body's registers hold the fields, and what it asks of its arguments it asks per chunk
  __shared__ FramedArgs args;
  __shared__ int next;
  for (;;) {
    __syncthreads();                       // the item before is done (barriers, shared memory)
    if (threadIdx.x == 0) {
      const int i = atomicAdd(head, 1);
      next = i >= n_items ? -1 : 0;
      if (i < n_items) {
        const mg_batch_item it = items[i];
        args = FramedArgs{};
        if (it.mesh >= 0 && it.mesh < n_meshes && framed_item<OP>(meshes[it.mesh], it, kBFM, kBFWarps, status, args)) next = 1;
        else set_status(status, ST_BAD_WORK);
      }
    }
    __syncthreads();
    if (next < 0) return;
    if (next) framed_run<OP, kBFM, kBFV, 32, false>(args, smem);
  }
}

// grid (columns, meshes): a mesh's CTAs stride over the blocks of its columns; meshes on plain tiles have no main
__global__ void __launch_bounds__(256) batched_framed_reduce_kernel(const mg_batch_framed* __restrict__ meshes) {
  __shared__ float4 acc[kFReduceRows][kFReduceCols];
  const mg_batch_framed f = meshes[blockIdx.y];
  const mg_batch_mesh& md = f.mesh;
  if (!md.dp || !md.partial || md.n_items <= 0) return;
  if (!f.main) {
    batch_reduce(md, blockIdx.x, gridDim.x);
    return;
  }
  const int M = batch_framed_M(md.N), np2 = 16 * M;
  const FramedReduceArgs a{static_cast<const float2*>(md.partial), md.n_items, md.L, np2, M, 32, md.N, md.dp, md.ldp, 0,
                           md.kinds + md.L, static_cast<const float2*>(f.wts), f.count, f.refuse,
                           f.scales};
  for (int blk = blockIdx.x; 2 * blk * kFReduceCols < md.L * np2; blk += gridDim.x) {
    framed_reduce_block(a, blk, acc);
    __syncthreads();
  }
}

template <int OP>
cudaError_t launch(const mg_batch_framed* meshes, int n_meshes, const mg_batch_item* items, int n_items, int* head, int grid,
                   size_t smem, int* status, cudaStream_t st) {
  static std::atomic<unsigned long long> done{0};
  const cudaError_t e = ensure_smem_attr(batched_framed_kernel<OP>, done);
  if (e != cudaSuccess) return e;
  batched_framed_kernel<OP><<<grid, kBFWarps * 32, smem, st>>>(meshes, n_meshes, items, n_items, head, status);
  return cudaGetLastError();
}

}  // namespace
}  // namespace mg

using namespace mg;

extern "C" int mg_batched_framed(int op, const mg_batch_framed* meshes, int n_meshes, const mg_batch_item* items, int n_items,
                                 int* head, int grid, size_t smem, int* status, void* stream) {
  if (op != MG_OP_FWD && op != MG_OP_BWD) return set_last_error(MG_E_ARG, "batched op must be fwd or bwd");
  if (!meshes || n_meshes < 0 || (!items && n_items > 0) || !head || grid < 1)
    return set_last_error(MG_E_ARG, "batched launch: bad arguments");
  if (n_items == 0) return MG_OK;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem + 1024 > (size_t)optin) return set_last_error(MG_E_CONFIG, "batched smem %zu above %d", smem, optin);
  (void)cudaGetLastError();   // start from a clean error state: launch errors below are this call's
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const cudaError_t e = op == MG_OP_FWD ? launch<OP_FWD>(meshes, n_meshes, items, n_items, head, grid, smem, status, st)
                                        : launch<OP_BWD>(meshes, n_meshes, items, n_items, head, grid, smem, status, st);
  return e == cudaSuccess ? MG_OK : set_last_error(MG_E_CUDA, "batched_framed_kernel: %s", cudaGetErrorString(e));
}

extern "C" int mg_batched_small(int op, const mg_batch_framed* meshes, int n_meshes, const mg_batch_item* items, int n_items,
                                int* head, int grid, size_t smem, int* status, void* stream) {
  if (op != MG_OP_FWD && op != MG_OP_BWD) return set_last_error(MG_E_ARG, "batched op must be fwd or bwd");
  if (!meshes || n_meshes < 0 || (!items && n_items > 0) || !head || grid < 1)
    return set_last_error(MG_E_ARG, "batched launch: bad arguments");
  if (n_items == 0) return MG_OK;
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem + 1024 > (size_t)optin) return set_last_error(MG_E_CONFIG, "batched smem %zu above %d", smem, optin);
  (void)cudaGetLastError();   // start from a clean error state: launch errors below are this call's
  const BatchedSmall b{meshes, n_meshes, items, n_items, head, status};
  LaunchCfg lc;
  lc.grid = dim3(grid);
  lc.block = dim3(32 * kSmallWarps);
  lc.smem = smem;
  lc.stream = static_cast<cudaStream_t>(stream);
  const cudaError_t e = op == MG_OP_FWD ? batched_small_fwd(lc, b) : batched_small_bwd(lc, b);
  return e == cudaSuccess ? MG_OK : set_last_error(MG_E_CUDA, "batched_small_kernel: %s", cudaGetErrorString(e));
}

extern "C" int mg_batched_framed_reduce(const mg_batch_framed* meshes, int n_meshes, void* stream) {
  if (!meshes || n_meshes < 0) return set_last_error(MG_E_ARG, "batched reduce: bad arguments");
  if (n_meshes == 0) return MG_OK;
  batched_framed_reduce_kernel<<<dim3(256, n_meshes), 256, 0, static_cast<cudaStream_t>(stream)>>>(meshes);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MG_OK : set_last_error(MG_E_CUDA, "batched_framed_reduce_kernel: %s", cudaGetErrorString(e));
}
