// Framed propagation kernels of list MG_FRAMED_FWD_C.
#include "mg_framed_launch.cuh"
#include "mg_framed_list.h"

MG_FRAMED_UNIT(framed_fwd_c, OP_FWD, MG_FRAMED_FWD_C)
