// Nearest-neighbour instantiations for small meshes and batches (Clements or Reck, complex, a vector over the 32
// lanes of a warp): forward with 2 to 16 modes and 1 to 4 vectors per lane, and back-propagation with 2 or 4 modes
// and 1 or 2 vectors per lane (through dJ/dT: mg_prop_nn_raw.cu).  A call on a small mesh is latency-bound - at
// N=64, B=1024 the default 2-mode x 4-vector forward tile gives 256 warps for 608 schedulers, one warp per busy
// scheduler - so fewer vectors per lane put more warps on more schedulers.
#include "mg_launch.h"

namespace mg {

namespace {
// (op, gr, M, V)
constexpr int kSmall[][4] = {{OP_FWD, 0, 2, 1}, {OP_FWD, 0, 2, 2}, {OP_FWD, 0, 2, 4}, {OP_FWD, 0, 4, 1},
                             {OP_FWD, 0, 4, 2}, {OP_FWD, 0, 8, 1}, {OP_FWD, 0, 8, 2}, {OP_FWD, 0, 16, 1}, {OP_BWD, 1, 4, 1}, {OP_BWD, 1, 4, 2}, {OP_BWD, 1, 2, 1},
                             {OP_BWD, 1, 2, 2}};
}  // namespace

bool nn_small_instantiated(int op, bool real, int M, int V, int gr, bool full) {
  if (real || !full) return false;
  if (op == OP_BWD && gr == 0) return nn_raw_instantiated(M, V);
  for (const auto& k : kSmall)
    if (k[0] == op && k[1] == gr && k[2] == M && k[3] == V) return true;
  return false;
}

cudaError_t launch_prop_nn_small(int op, int gr, int M, int V, const LaunchCfg& lc, const PropArgs& a) {
  if (op == OP_BWD && gr == 0) return launch_prop_nn_raw(M, V, lc, a);
  switch (op * 10000 + M * 10 + V) {
    case 21: return launch_one<OP_FWD, 2, 1, false, 32, 0, false, true>(lc, a);
    case 22: return launch_one<OP_FWD, 2, 2, false, 32, 0, false, true>(lc, a);
    case 24: return launch_one<OP_FWD, 2, 4, false, 32, 0, false, true>(lc, a);
    case 41: return launch_one<OP_FWD, 4, 1, false, 32, 0, false, true>(lc, a);
    case 81: return launch_one<OP_FWD, 8, 1, false, 32, 0, false, true>(lc, a);
    case 161: return launch_one<OP_FWD, 16, 1, false, 32, 0, false, true>(lc, a);
    case 82: return launch_one<OP_FWD, 8, 2, false, 32, 0, false, true>(lc, a);
    case 42: return launch_one<OP_FWD, 4, 2, false, 32, 0, false, true>(lc, a);
    case OP_BWD * 10000 + 41: return launch_one<OP_BWD, 4, 1, false, 32, 1, false, true>(lc, a);
    case OP_BWD * 10000 + 21: return launch_one<OP_BWD, 2, 1, false, 32, 1, false, true>(lc, a);
    case OP_BWD * 10000 + 22: return launch_one<OP_BWD, 2, 2, false, 32, 1, false, true>(lc, a);
    case OP_BWD * 10000 + 42: return launch_one<OP_BWD, 4, 2, false, 32, 1, false, true>(lc, a);
    default: return cudaErrorInvalidConfiguration;
  }
}

}  // namespace mg
