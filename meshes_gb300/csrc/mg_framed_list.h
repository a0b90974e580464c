// The framed kernels' instantiations, (modes per lane, vectors per lane, mixed warps), for lane groups that fill the warp.
// The fields of back-propagation fill the registers at M V = 32; vectors per lane below that spread smaller batches.
#pragma once
#define MG_FRAMED_FWD_A(X) X(4, 1, false) X(4, 2, false) X(4, 2, true) X(4, 4, false) X(4, 4, true)
#define MG_FRAMED_FWD_B(X) X(8, 1, false) X(8, 2, false) X(8, 2, true) X(8, 3, false) X(8, 4, false) X(8, 4, true)
#define MG_FRAMED_FWD_C(X) X(16, 1, false) X(16, 2, false) X(16, 2, true) X(16, 3, false) X(16, 4, false)
#define MG_FRAMED_FWD_D(X) X(20, 1, false) X(20, 2, false) X(20, 2, true) X(20, 3, false)
#define MG_FRAMED_BWD_A(X) X(4, 1, false) X(4, 2, false) X(4, 2, true) X(4, 4, false) X(4, 4, true)
#define MG_FRAMED_BWD_B1(X) X(8, 1, false) X(8, 2, false) X(8, 2, true)
#define MG_FRAMED_BWD_B2(X) X(8, 3, false) X(8, 4, false) X(8, 4, true)
#define MG_FRAMED_BWD_C(X) X(16, 1, false) X(16, 2, false) X(16, 2, true)
#define MG_FRAMED_BWD_D(X) X(20, 1, false) X(20, 2, false) X(20, 2, true)
