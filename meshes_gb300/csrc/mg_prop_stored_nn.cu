// Stored-activation kernels (GR 4: the forward pass writes every layer's input, back-propagation reads them) of
// nearest-neighbour meshes with a vector over the 32 lanes of a warp.  A lossy mesh's
// segments are short launches one after another (N = 132, B = 694: forward 78 -> 44 us, back-propagation 200 -> 191 with these
// tiles): at N = 128 and B = 1024 the default tile (8 modes and 4 vectors per
// lane) runs 128 warps on 608 schedulers, 23 us for twelve layers of back-propagation.
#include "mg_launch.h"

namespace mg {

#define MG_STORED_NN(X) \
  X(OP_FWD, 2, 1) X(OP_FWD, 2, 2) X(OP_FWD, 2, 4) X(OP_FWD, 4, 1) X(OP_FWD, 4, 2) X(OP_FWD, 8, 1) X(OP_FWD, 8, 2) X(OP_FWD, 8, 4) \
  X(OP_BWD, 2, 4) X(OP_BWD, 4, 4) X(OP_BWD, 8, 4)

bool stored_nn_instantiated(int op, int M, int V) {
#define MG_X(OP_, M_, V_) if (op == OP_ && M == M_ && V == V_) return true;
  MG_STORED_NN(MG_X)
#undef MG_X
  return false;
}

cudaError_t launch_prop_stored_nn(int op, int M, int V, const LaunchCfg& lc, const PropArgs& a) {
#define MG_X(OP_, M_, V_) \
  if (op == OP_ && M == M_ && V == V_) return launch_one<OP_, M_, V_, false, 32, 4, false, true>(lc, a);
  MG_STORED_NN(MG_X)
#undef MG_X
  return cudaErrorInvalidConfiguration;
}

}  // namespace mg
