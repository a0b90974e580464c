// Back-propagation of nearest-neighbour complex meshes through dJ/dT (GR 0: symmetric and generic crossings), a vector over
// the 32 lanes of a warp.  The general kernel's 8- or 16-mode lane groups with 2 or 4 vectors leave a small batch
// on few warps: 474 modes and layers, 2 vectors 1241 us, here 589; 372, 66 vectors 980 and 463; 128, 2000 vectors 192 and
// 67 us (GB300).
#include "mg_launch.h"

namespace mg {

#define MG_RAW_NN(X) X(2, 1) X(2, 2) X(2, 4) X(4, 1) X(4, 2) X(4, 4) X(8, 1) X(8, 2) X(8, 4) X(16, 1) X(16, 2)

bool nn_raw_instantiated(int M, int V) {
#define MG_X(M_, V_) if (M == M_ && V == V_) return true;
  MG_RAW_NN(MG_X)
#undef MG_X
  return false;
}

cudaError_t launch_prop_nn_raw(int M, int V, const LaunchCfg& lc, const PropArgs& a) {
#define MG_X(M_, V_) if (M == M_ && V == V_) return launch_one<OP_BWD, M_, V_, false, 32, 0, false, true>(lc, a);
  MG_RAW_NN(MG_X)
#undef MG_X
  return cudaErrorInvalidConfiguration;
}

}  // namespace mg
