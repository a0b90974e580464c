// What the persistent batched kernels share: arguments of a work item, the plain reduction.
#pragma once
#include "../../include/meshes_gb300.h"
#include "mg_prop.cuh"

namespace mg {

__host__ __device__ __forceinline__ int cls_M(int cls) { return cls == MG_BCLS_C16 ? 16 : 8; }

// arguments of one item of a mesh on plain tiles (np2 slots per layer, W warps per CTA)
template <int OP>
__device__ __forceinline__ void batch_args(PropArgs& a, const mg_batch_mesh& md, const mg_batch_item& it, int np2, int W,
                                           int* status) {
  a.N = md.N; a.L = md.L; a.B = md.B; a.ldu = md.ldu;
  a.G = md.G; a.logG = 31 - __clz(md.G); a.W = W; a.CL = md.CL; a.S = md.S;
  a.layer_bytes = md.layer_bytes; a.dlayer_bytes = 0;
  a.tiles = static_cast<const unsigned char*>(md.tiles); a.dtiles = nullptr;
  a.kinds = md.kinds;
  a.in0 = md.in0; a.in1 = md.in1; a.out0 = md.out0; a.out1 = md.out1;
  a.partial = (OP == OP_BWD) ? static_cast<float2*>(md.partial) + (size_t)it.part * md.L * np2 : nullptr;
  a.status = status;
  a.v0 = it.v0; a.vend = it.vend;
  a.target = nullptr;
  a.perm = a.pflags = a.perm_last = a.pflag_last = nullptr;   // batched meshes carry no permutations
}
// whether an item is within a mesh's batch and its lane group holds the mesh
__device__ __forceinline__ bool batch_item_ok(const mg_batch_mesh& md, const mg_batch_item& it, int M) {
  return md.G >= 1 && md.G <= 32 && !(md.G & (md.G - 1)) && md.G * M >= md.N && it.v0 >= 0 && it.vend <= md.B;
}

// dp[l][q][k] = sum over the mesh's items (in item order) of the partials: the ny CTAs of a mesh stride over its slot
// positions, one position per thread at a time, consecutive threads on consecutive positions (coalesced); each thread keeps
// 8 item loads in flight and adds them in item order, so the sums are those of a plain sequential loop.  (One CTA per mesh,
// one load in flight per thread, took 3.85 ms on the 512-mesh benchmark - 23% of its forward + backward step.)
__device__ __forceinline__ void batch_reduce(const mg_batch_mesh& md, int y, int ny) {
  const int M = cls_M(md.cls), G = md.G, np2 = G * M / 2, L = md.L, N = md.N;
  const int* geo = md.kinds + L;
  const float2* part = static_cast<const float2*>(md.partial);
  const size_t stride = (size_t)L * np2;
  const int n = md.n_items;
  for (int idx = y * blockDim.x + threadIdx.x; idx < L * np2; idx += ny * blockDim.x) {
    const int l = idx / np2, pos = idx - l * np2;
    const int q = pos_slot(pos, M, G);
    if (q >= N / 2) continue;
    const int sh = geo[2 * l], ln = geo[2 * l + 1];
    float sx = 0.f, sy = 0.f;
    if (q >= sh / 2 && q < sh / 2 + ln) {
      const float2* p = part + (size_t)l * np2 + pos;
      int k = 0;
      for (; k + 8 <= n; k += 8) {
        float2 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = p[(size_t)(k + i) * stride];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          sx += v[i].x;
          sy += v[i].y;
        }
      }
      for (; k < n; ++k) {
        const float2 v = p[(size_t)k * stride];
        sx += v.x;
        sy += v.y;
      }
    }
    float* o = md.dp + (size_t)l * md.ldp + (size_t)q * md.n_p;
    o[0] = sx;
    if (md.n_p > 1) o[1] = sy;
  }
}

}  // namespace mg
