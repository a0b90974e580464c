// Arguments and sizes of the frame pass (mg_frame.cuh) and the framed kernels (mg_framed.cuh), for the host side.
#pragma once
#include "mg_coeffs.cuh"

namespace mg {

// Frames start at 2^22, are due to start again below 2^-8 and do so at once below 2^-18; a layer may take one down by 2^-30
// (a cross state), so they stay within 2^-48 and 2^22.
constexpr int kFrameTop = 22, kFrameDue = -8, kFrameNow = -18;
// Largest part of a vector as it enters, 2^22: with its 640 modes' energy in one (2^28) the products of two framed fields stay
// below 2^102 and the sum of 2^20 vectors' below 2^122; behind a cross state a product 2^-35 of the largest keeps its bits
constexpr int kFieldTop = 22;
constexpr int kWarpScales = 12;            // ints of shared memory per warp (16-byte steps)
constexpr int kFrameSeg = 16;              // layers per segment, about
constexpr int kFrameBatch = 16;            // layers whose frames are held in shared memory at a time
constexpr int kFrameThreads = 512;
constexpr int kFrameStages = 3;            // pipeline stages and gradient slots: the chunk at work, the one before, the next
constexpr int KIND_RESCALE = 1 << 14;      // OR-ed into a layer's kind: the frames start again behind it

// Planes of one layer, lane j, pair e < M/4 of the lane's crossings (e, e + M/4), values of the two side by side:
//   main [(2e + h) G + j] = (re, re', im, im') of alpha (h = 0), beta (h = 1)
//   gam  [e G + j]          gamma, back-propagation only: behind the layer's main plane (framed_layer_bytes)
//   resc [k G + j], k < M/2 RESCALE layers: the factors of the lane's modes k and k + M/2
// Gradient partials and their weights: float4 (th, th', ph, ph') at [e G + j].
struct FrameArgs {
  int L, M, G;
  int bwd;                       // 1: gam and wts are wanted
  const float4* tdiag;           // [L][modes], CoefArgs
  const float4* toff;
  const float* tmag;
  const float2* tcs;
  const int* kinds;              // [L]
  float4* main;                  // [L][np2, bwd: + np2/2 of gamma]
  float4* resc;                  // [L][np2]
  float4* wts;                   // [L][np2/2]
  float2* dfin;                  // [modes]: frames after the last layer
  int* fkinds;                   // [L] kinds with KIND_RESCALE
  int* count;                    // layers that break a pair of layers up, plus 2^30 for an entry that is NaN (set to 0
                                 // by the coefficient pass)
};
// A CTA of the frame pass takes rows * 32 modes of one segment
constexpr int kFrameMaxRows = 5;
inline size_t frame_smem_bytes(int modes, int rows) {
  return (size_t)(kFrameBatch + 1) * (32 * rows + 2) * 16 + (size_t)(kFrameBatch + 1) * modes * 4;
}

// The PropArgs part describes the unframed launch on the same tiles (tiles, kinds, CL, S), which a mesh that the
// frames do not suit takes inside the same kernel.
struct FramedArgs : PropArgs {
  const float4* main;
  const float4* resc;
  const float2* dfin;
  const int* fkinds;
  const int* count;
  int* scales;                   // back-propagation: the CTA's partials are 2^this of their own size (null: fields as they are)
  int fcl;                       // layers per stage
  unsigned flb;                  // bytes of a layer's tile
  int refuse;                    // count from which on the mesh takes the unframed body
};
// threads per CTA the kernels are compiled for
__host__ __device__ constexpr int framed_max_threads(int M, int V) { return M * V <= 16 ? 512 : 256; }
// vectors of one CTA: W warps of V per lane group (R groups per warp), mix: every second four warps V - 1
__host__ __device__ constexpr int framed_cta_vectors(int W, int R, int V, bool mix) {
  return R * (W * V - (mix ? W / 8 * 4 : 0));
}
// rows of resc staged with CL layers (few layers have one: each segment's last and those that bound the frames; more are
// read from global memory)
__host__ __device__ constexpr int framed_resc_rows(int CL) { return CL / 8 > 1 ? CL / 8 : 1; }
// one layer's tile (op: that the tiles are built for); one pipeline stage: CL tiles of lb bytes and the rows of resc
__host__ __device__ constexpr unsigned framed_layer_bytes(int op, int np2) { return (unsigned)np2 * (op == OP_BWD ? 24 : 16); }
__host__ __device__ constexpr size_t framed_stage_bytes(unsigned lb, int np2, int CL) { return (size_t)CL * lb + (size_t)framed_resc_rows(CL) * np2 * 16; }
// shared memory of a launch: [stages][a layer of zeros][BWD: per slot the W warps' gradients of CL layers, one layer beyond
// the last][2 mbarriers per stage][state][warps' scales][step codes][RESCALEs per chunk]
__host__ __device__ constexpr size_t framed_bars_offset(int op, unsigned lb, int np2, int W, int CL) {
  return kFrameStages * framed_stage_bytes(lb, np2, CL) + lb +
         (op == OP_BWD ? ((size_t)kFrameStages * W * CL + 1) * np2 * 8 : 0);
}
__host__ __device__ constexpr size_t framed_smem_bytes(int op, unsigned lb, int np2, int W, int CL, int L) {
  return framed_bars_offset(op, lb, np2, W, CL) + 16 * kFrameStages + 16 + 4 * (size_t)kWarpScales * W + 4 * (size_t)(L + 8) + 4 * (size_t)((L + CL) / CL) * framed_resc_rows(CL);
}

}  // namespace mg
