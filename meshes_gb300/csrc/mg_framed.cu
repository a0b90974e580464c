// Dispatch of the framed kernels, the frame pass and the framed gradient reduction.
#include <algorithm>

#include "../../include/meshes_gb300.h"
#include "mg_framed.cuh"
#include "mg_framed_list.h"
#include "mg_launch.h"

namespace mg {

#define MG_UNIT(NAME) cudaError_t NAME(int M, int V, bool mix, const LaunchCfg& lc, const FramedArgs& a);
MG_UNIT(framed_fwd_a) MG_UNIT(framed_fwd_b) MG_UNIT(framed_fwd_c) MG_UNIT(framed_fwd_d)
MG_UNIT(framed_bwd_a) MG_UNIT(framed_bwd_b1) MG_UNIT(framed_bwd_b2) MG_UNIT(framed_bwd_c) MG_UNIT(framed_bwd_d)
#undef MG_UNIT

bool framed_instantiated(int op, int M, int V, bool full, bool mix) {
  if (!full) return false;
#define MG_X(M_, V_, MIX_) if (M == M_ && V == V_ && mix == MIX_) return true;
  if (op == OP_FWD) { MG_FRAMED_FWD_A(MG_X) MG_FRAMED_FWD_B(MG_X) MG_FRAMED_FWD_C(MG_X) MG_FRAMED_FWD_D(MG_X) }
  if (op == OP_BWD) { MG_FRAMED_BWD_A(MG_X) MG_FRAMED_BWD_B1(MG_X) MG_FRAMED_BWD_B2(MG_X) MG_FRAMED_BWD_C(MG_X) MG_FRAMED_BWD_D(MG_X) }
#undef MG_X
  return false;
}

// The launch of a batch: warps per CTA and vectors per lane such that waves x (vectors per scheduler + 4) is least.
// Measured on GB300 over one-wave batches, a launch takes time proportional to n + 4 for n vectors per scheduler: the
// layers' latency is worth about four vectors (M = 8, L = 256, back-propagation: 87 us at n = 1, 160 at 4, 236 at 8;
// forward 36, 53, 79).  Two vectors per scheduler go as V = 2 in 4 warps rather than V = 1 in 8 where that is faster (each
// coefficient serves two vectors): forward at N = 256 44 -> 40 us, N = 400 97 -> 86, N = 600 171 -> 148; back-propagation at
// N = 400 314 -> 267, but at N = 256 101 -> 105 and at N = 600 531 -> 580 (it spills).
bool framed_pick(int op, int M, int B, int sms, mg_config* out) {
  long best = 0;
  auto consider = [&](int V, bool mix, int W) {
    const int cap = framed_cta_vectors(W, 1, V, mix);
    const long ctas = std::max(1, (B + cap - 1) / cap), waves = (ctas + sms - 1) / sms;
    const bool pairs = op == OP_FWD || M == 16;   // V = 2 in 4 warps before V = 1 in 8
    const long cost = 2 * waves * (cap / 4 + 4) + (W == 8 && V == 1 && pairs ? 1 : 0);
    if (W == 4 && V > 1 && !(V == 2 && !mix && pairs)) return;
    if (best != 0 && cost >= best) return;
    best = cost;
    *out = mg_config{M, V, W, 0, 0, mix ? 6 : 5};
  };
#define MG_X(M_, V_, MIX_)                            \
  if (M == M_) {                                      \
    if (!MIX_) consider(V_, MIX_, 4);                 \
    consider(V_, MIX_, 8);                            \
    if (M_ == 4 && V_ > 1) consider(V_, MIX_, 16);    \
  }
  if (op == OP_FWD) { MG_FRAMED_FWD_A(MG_X) MG_FRAMED_FWD_B(MG_X) MG_FRAMED_FWD_C(MG_X) MG_FRAMED_FWD_D(MG_X) }
  if (op == OP_BWD) { MG_FRAMED_BWD_A(MG_X) MG_FRAMED_BWD_B1(MG_X) MG_FRAMED_BWD_B2(MG_X) MG_FRAMED_BWD_C(MG_X) MG_FRAMED_BWD_D(MG_X) }
#undef MG_X
  return best != 0;
}

// Whether the framed launch repays the frame pass.  The pass takes about 8 us and 6e-5 us per slot (tiles with it and without:
// N = 128 17 and 9 us, N = 256 19 and 11, N = 600 42 and 22).  With n vectors per scheduler a framed layer saves, per M modes
// of a lane, forward 0.0018 n us up to M = 8, where the general kernel has a tile for every n (N = 256: 46 -> 40 us at n = 2,
// 64 -> 50 at 4, 99 -> 72 at 7; N = 128: 60 -> 44 at 16), and 0.006 (1 + (n-1)/4) us beyond; in back-propagation about
// 0.018 (1 + (n-1)/8) us (N = 256: 122 -> 75 us at n = 1, 265 -> 199 at 7), of which a forward launch on the same tiles can lose
// some at n = 1 (N = 128, B = 128: 38.6 -> 30.4 us, forward 19.1 -> 21.2, tiles 8.9 -> 17.1: not framed).
bool framed_pays(int op, int M, int L, int np2, int B, int sms) {
  const double n = std::max(1.0, (double)B / (4.0 * sms));
  const double layer = op == OP_BWD ? 0.018 * (1 + (n - 1) / 8) : M <= 8 ? 0.0018 * n : 0.006 * (1 + (n - 1) / 4);
  return L * M * layer > (op == OP_BWD ? 1.15 : 1.0) * (8.0 + 6e-5 * L * np2);
}

cudaError_t launch_prop_framed(int op, int M, int V, bool mix, const LaunchCfg& lc, const FramedArgs& a) {
  if (op == OP_FWD)
    return M == 4 ? framed_fwd_a(M, V, mix, lc, a) : M == 8 ? framed_fwd_b(M, V, mix, lc, a)
         : M == 16 ? framed_fwd_c(M, V, mix, lc, a) : framed_fwd_d(M, V, mix, lc, a);
  return M == 4 ? framed_bwd_a(M, V, mix, lc, a) : M == 16 ? framed_bwd_c(M, V, mix, lc, a)
       : M == 20 ? framed_bwd_d(M, V, mix, lc, a)
       : V <= 2 ? framed_bwd_b1(M, V, mix, lc, a) : framed_bwd_b2(M, V, mix, lc, a);
}

template <int ROWS>
static cudaError_t launch_frames_rows(const FrameArgs& a, int nseg, cudaStream_t stream) {
  static std::atomic<unsigned long long> done{0};
  const cudaError_t e = ensure_smem_attr(frame_kernel<ROWS>, done);
  if (e != cudaSuccess) return e;
  const int modes = a.G * a.M;
  const dim3 grid(nseg, (modes + 32 * ROWS - 1) / (32 * ROWS));
  frame_kernel<ROWS><<<grid, kFrameThreads, frame_smem_bytes(modes, ROWS), stream>>>(a);
  return cudaGetLastError();
}

// Modes per CTA: as few (32 to 160) as keep the pass to one wave, since every CTA of a segment looks through all of its
// modes for where the frames start again.  Measured at N = 600, L = 600: 52 us at 32 modes per CTA, five waves.
cudaError_t launch_frames(const FrameArgs& a, int sms, cudaStream_t stream) {
  const int nseg = (a.L + kFrameSeg - 1) / kFrameSeg, modes = a.G * a.M;
  int rows = 1;
  while (rows < kFrameMaxRows && nseg * ((modes + 32 * rows - 1) / (32 * rows)) > sms) ++rows;
  switch (rows) {
    case 1: return launch_frames_rows<1>(a, nseg, stream);
    case 2: return launch_frames_rows<2>(a, nseg, stream);
    case 3: return launch_frames_rows<3>(a, nseg, stream);
    case 4: return launch_frames_rows<4>(a, nseg, stream);
    default: return launch_frames_rows<5>(a, nseg, stream);
  }
}

cudaError_t launch_framed_reduce(const float2* partial, int nC, int L, int np2, int M, int G, int N, float* dp, int ldp,
                                 int accumulate, const int* geo, const float2* wts, const int* count, int refuse,
                                 const int* scales, cudaStream_t stream) {
  framed_reduce_kernel<<<(L * np2 / 2 + kFReduceCols - 1) / kFReduceCols, 256, 0, stream>>>(
      FramedReduceArgs{partial, nC, L, np2, M, G, N, dp, ldp, accumulate, geo, wts, count, refuse, scales});
  return cudaGetLastError();
}

}  // namespace mg
