// Framed propagation kernels of list MG_FRAMED_FWD_D.
#include "mg_framed_launch.cuh"
#include "mg_framed_list.h"

MG_FRAMED_UNIT(framed_fwd_d, OP_FWD, MG_FRAMED_FWD_D)
