"""The bounded waits of the framed pipeline (tests/test_wait_timeout.py runs the general one): a chunk of coefficients is never
copied, the 1 ms limit runs out, MG_ST_TIMEOUT is recorded, and the same workspace then serves a normal call."""
import ctypes
import time

import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O
from test_framed import _mesh

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("where", ["first", "second", "in the ring", "last"])
@pytest.mark.parametrize("op", [0, 2])
@pytest.mark.parametrize("N,L,B", [(256, 200, 4096), (130, 130, 4000), (600, 100, 900)])     # mixed warps and uniform ones, 8 and 20 modes
def test_expired_wait(N, L, B, op, where):
    from meshes_gb300 import _lib
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(N + op)
    om = _mesh(rng, N, "clements", L)
    info = _lib.mg_plan_info()
    assert lib.mg_plan(op, N, L, B, 0, 0, None, ctypes.byref(info)) == 0
    n = -(-L // info.CL)
    assert info.S == 3 and info.CL != 16 and n >= 5      # (the framed pipeline's stages; general forward launches have 2)
    chunk = {"first": 0, "second": 1, "in the ring": 4, "last": n - 1}[where]
    d = [torch.tensor(np.asarray(a), device="cuda") for a in (np.int32(om.lens), np.int32(om.shifts), om.p, om.s)]
    nb = lib.mg_workspace_bytes(op, N, L, B, 0, 0, None)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    _lib.check(lib.mg_workspace_init(ws.data_ptr(), nb, st), "init")
    _lib.check(lib.mg_build_tiles(op, N, L, 0, d[0].data_ptr(), d[1].data_ptr(), None, 0, d[2].data_ptr(), N, d[3].data_ptr(), N,
                                  None, None, None, B, None, ws.data_ptr(), nb, st), "mg_build_tiles")
    x, g = O.unit_columns(rng, N, B), O.unit_columns(rng, N, B)
    y = O.propagate(om, x)
    a, b = (torch.tensor(t, dtype=torch.complex64, device="cuda") for t in ((x, x) if op == 0 else (y, g)))
    out, dp = torch.zeros_like(a), torch.zeros(om.p.shape, device="cuda")
    args = (a.data_ptr(), None, out.data_ptr(), None) if op == 0 else (a.data_ptr(), b.data_ptr(), None, out.data_ptr())
    t0 = time.perf_counter()
    _lib.check(lib.mg_propagate_wait_test(op, N, L, B, 0, *args, N, 1000000, chunk, ws.data_ptr(), nb, st), "wait test")
    assert lib.mg_read_status(ws.data_ptr(), 1, st) == 1
    assert time.perf_counter() - t0 < 5.0
    _lib.check(lib.mg_propagate(op, N, L, B, 0, 0, *args, N, dp.data_ptr() if op else None, N, 0, None, ws.data_ptr(), nb, st),
               "mg_propagate")
    assert lib.mg_read_status(ws.data_ptr(), 0, st) == 0
    if op == 0:
        assert O.rel_err(out.cpu().numpy(), y) < TOL
    else:
        G, _, gin = O.vjp_unitary(om, y, g)
        assert O.rel_err(out.cpu().numpy(), gin) < TOL and O.rel_err(dp.cpu().numpy(), O.contract_dp(om, G)) < TOL
