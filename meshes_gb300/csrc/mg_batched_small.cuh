// Batched propagation with a number of vectors per lane group of each mesh's own (mg_batch_framed.V), every class of mesh in
// one persistent launch, those of 65 to 256 modes on framed tiles where they have some.
//
// What bounds it: the latency of a mesh's layers, which is that of the deepest mesh in the launch.  An item of
// mg_batched.cu is 8 warps of 4 vectors, so a few requests leave most SMs idle and take 99 us forward through a 256-mode
// mesh; items of one vector per warp spread over the SMs, and a framed layer of theirs takes a third of that.
#pragma once
#include "mg_batched_framed.cuh"
#include "mg_batched_small.h"

namespace mg {

// bodies: a class and its vectors per lane group
enum { ITEM_NONE = 0, ITEM_BAD = 1, ITEM_FRAMED_8 = 8, ITEM_FRAMED_4 = 16, ITEM_PLAIN = 24 };

// An item on plain tiles: on arguments of its own, in which the compiler knows what is null; with those in shared memory it
// kept the body's branches for permutations, targets and stored fields (GB300: a tick's forward launch, 64 modes, 24.7 -> 22.2 us).
template <int OP, int M, int V, bool REAL, int GR>
__device__ __forceinline__ void plain_item(const BatchedSmall& b, int item, unsigned char* smem) {
  const mg_batch_item it = b.items[item];
  const mg_batch_mesh md = b.meshes[it.mesh].mesh;
  PropArgs a{};
  batch_args<OP>(a, md, it, md.G * M / 2, kSmallWarps, b.status);
  if constexpr (REAL) prop_body<OP, M, V, true, 0, GR, false, false>(a, smem);
  else prop_body<OP, M, V, false, 0, GR, false, false, false>(a, smem);
}

template <int OP>
__global__ void __launch_bounds__(256, 1) batched_small_kernel(const BatchedSmall b) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ FramedArgs args;
  __shared__ int next, item;
  for (;;) {
    __syncthreads();                       // the item before is done (barriers, shared memory)
    if (threadIdx.x == 0) {
      const int i = atomicAdd(b.head, 1);
      next = ITEM_NONE;
      item = i;
      if (i < b.n_items) {
        const mg_batch_item it = b.items[i];
        next = ITEM_BAD;
        if (it.mesh >= 0 && it.mesh < b.n_meshes) {
          const mg_batch_framed f = b.meshes[it.mesh];
          const mg_batch_mesh& md = f.mesh;
          args = FramedArgs{};
          if (f.V >= 1 && f.V <= 4) {
            if (f.main) {
              const int M = batch_framed_M(md.N);
              if (framed_item<OP>(f, it, M, kSmallWarps, b.status, args)) next = (M == 8 ? ITEM_FRAMED_8 : ITEM_FRAMED_4) + f.V;
            } else if (md.cls >= MG_BCLS_C8 && md.cls <= MG_BCLS_R8 && batch_item_ok(md, it, cls_M(md.cls))) {
              next = ITEM_PLAIN + 8 * md.cls + f.V;
            }
          }
        }
      }
    }
    __syncthreads();
    constexpr int C = OP == OP_BWD ? 1 : 0, R = OP == OP_BWD ? 2 : 0;
    // plain tiles: one-vector crossings, as mg_batched.cu's; back-propagation at the class's own V alone, in whose order
    // the gradients of a request are always summed
    switch (next) {
      case ITEM_NONE: return;
      case ITEM_FRAMED_8 + 1: framed_run<OP, 8, 1, 32, false>(args, smem); break;
      case ITEM_FRAMED_8 + 4: framed_run<OP, 8, 4, 32, false>(args, smem); break;
      case ITEM_FRAMED_4 + 1: framed_run<OP, 4, 1, 32, false>(args, smem); break;
      case ITEM_FRAMED_4 + 4: framed_run<OP, 4, 4, 32, false>(args, smem); break;
      case ITEM_PLAIN + 8 * MG_BCLS_C8 + 4: plain_item<OP, 8, 4, false, C>(b, item, smem); break;
      case ITEM_PLAIN + 8 * MG_BCLS_C16 + 2: plain_item<OP, 16, 2, false, C>(b, item, smem); break;
      case ITEM_PLAIN + 8 * MG_BCLS_R8 + 4: plain_item<OP, 8, 4, true, R>(b, item, smem); break;
      default:
        if constexpr (OP == OP_FWD) {
          if (next == ITEM_PLAIN + 8 * MG_BCLS_C8 + 1) { plain_item<OP, 8, 1, false, 0>(b, item, smem); break; }
          if (next == ITEM_PLAIN + 8 * MG_BCLS_C16 + 1) { plain_item<OP, 16, 1, false, 0>(b, item, smem); break; }
          if (next == ITEM_PLAIN + 8 * MG_BCLS_R8 + 1) { plain_item<OP, 8, 1, true, 0>(b, item, smem); break; }
        } else {
          if (next == ITEM_FRAMED_8 + 2) { framed_run<OP, 8, 2, 32, false>(args, smem); break; }
          if (next == ITEM_FRAMED_4 + 2) { framed_run<OP, 4, 2, 32, false>(args, smem); break; }
        }
        if (threadIdx.x == 0) set_status(b.status, ST_BAD_WORK);
    }
  }
}

template <int OP>
cudaError_t launch_batched_small(const LaunchCfg& lc, const BatchedSmall& b) {
  static std::atomic<unsigned long long> done{0};
  const cudaError_t e = ensure_smem_attr(batched_small_kernel<OP>, done);
  if (e != cudaSuccess) return e;
  batched_small_kernel<OP><<<lc.grid, lc.block, lc.smem, lc.stream>>>(b);
  return cudaGetLastError();
}

}  // namespace mg
