// A work item of a mesh on framed tiles (mg_batch_framed): 65 to 256 modes over the 32 lanes of a warp.
#pragma once
#include "mg_batched.cuh"
#include "mg_framed.cuh"

namespace mg {

// modes per lane of a mesh on framed tiles in a batch
__device__ __forceinline__ int batch_framed_M(int N) { return N > 128 ? 8 : 4; }

// the item's launch arguments for W warps; false: a work item outside its mesh or its batch, or a stage that shared memory
// cannot hold
template <int OP>
__device__ __forceinline__ bool framed_item(const mg_batch_framed& f, const mg_batch_item& it, int M, int W, int* status,
                                            FramedArgs& a) {
  const mg_batch_mesh& md = f.mesh;
  const int np2 = 16 * M;
  if (md.G != 32 || !batch_item_ok(md, it, M) || f.fcl < 1) return false;
  // the mesh's tiles are those of M modes per lane, with gamma (both ops read back-propagation's)
  if (M != batch_framed_M(md.N) || f.flb != framed_layer_bytes(OP_BWD, np2)) return false;
  unsigned dynamic;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dynamic));
  if (framed_smem_bytes(OP, f.flb, np2, W, f.fcl, md.L) > dynamic) return false;
  batch_args<OP>(a, md, it, np2, W, status);
  a.main = static_cast<const float4*>(f.main);
  a.resc = static_cast<const float4*>(f.resc);
  a.dfin = static_cast<const float2*>(f.dfin);
  a.fkinds = f.fkinds;
  a.count = f.count;
  a.scales = OP == OP_BWD && f.scales ? f.scales + it.part : nullptr;
  a.fcl = f.fcl; a.flb = f.flb; a.refuse = f.refuse;
  return true;
}

}  // namespace mg
