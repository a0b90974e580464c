// Framed propagation kernels of list MG_FRAMED_BWD_C.
#include "mg_framed_launch.cuh"
#include "mg_framed_list.h"

MG_FRAMED_UNIT(framed_bwd_c, OP_BWD, MG_FRAMED_BWD_C)
