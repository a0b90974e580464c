// Framed propagation kernels of list MG_FRAMED_BWD_B2.
#include "mg_framed_launch.cuh"
#include "mg_framed_list.h"

MG_FRAMED_UNIT(framed_bwd_b2, OP_BWD, MG_FRAMED_BWD_B2)
