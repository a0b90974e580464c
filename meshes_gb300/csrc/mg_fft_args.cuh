// Arguments and sizes of the butterfly kernels (mg_fft.cuh), for the host side.
#pragma once
#include "mg_prop.cuh"

namespace mg {

constexpr int kFftThreads = 256;
constexpr int kFftVectors = 2;      // per lane group: packed
struct FftArgs : PropArgs {
  int M;                            // of the tiles (G too)
};
// modes per lane for N modes, 0: no kernel
__host__ __device__ constexpr int fft_modes(int op, int N) {
  return N == 64 ? 8 : N == 128 || N == 256 ? 16 : N == 512 && op == OP_FWD ? 32 : 0;
}
// forward: 64 registers of fields, two CTAs per SM
__host__ __device__ constexpr int fft_ctas_per_sm(int op, int M) { return op == OP_FWD && M <= 16 ? 2 : 1; }
// shared memory: the tiles (T by rows; back-propagation: the splitter pairs), per warp a buffer to turn the fields in and
// (back-propagation) its gradient sums, the layers' codes
struct FftLayout {
  uint32_t tiles, cs, turn, acc, codes, total;
};
__host__ __device__ constexpr FftLayout fft_layout(int op, int M, int G, int L) {
  const uint32_t N = M * G, W = kFftThreads / 32, l = L;
  FftLayout o{};
  o.cs = o.tiles + l * N * 16;
  o.turn = o.cs + (op == OP_BWD ? l * N * 4 : 0);
  o.acc = o.turn + W * (32 / G) * (N + G) * 16;
  o.codes = o.acc + (op == OP_BWD ? W * l * N * 4 : 0);
  o.total = o.codes + l * 4;
  return o;
}

}  // namespace mg
