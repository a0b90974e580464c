"""Gradients of symmetric crossings (back-propagation through dJ/dT) with a vector over the whole warp, 2 to 16 modes per lane
and 1 to 4 vectors, against the complex128 oracle and the general kernel on its own configuration.  Tolerance: the
library's 1e-5 relative Frobenius error."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _run(om, B, cfg, y, g):
    from meshes_gb300 import _lib
    lib, st, c = _lib.load(), torch.cuda.current_stream().cuda_stream, _lib.cfg_ptr(cfg) if cfg is not None else None
    N, L = om.N, om.L
    nb = lib.mg_workspace_bytes(2, N, L, B, 1, 0, c)
    assert nb, _lib.last_error()
    ws = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
    _lib.check(lib.mg_workspace_init(ws.data_ptr(), nb, st), "init")
    geo = [torch.tensor(a, dtype=torch.int32, device="cuda") for a in (om.lens, om.shifts)]
    p = torch.tensor(om.p.reshape(-1), device="cuda")
    s = None if om.s is None else torch.tensor(om.s.reshape(-1), device="cuda")
    _lib.check(lib.mg_build_tiles(2, N, L, 0, geo[0].data_ptr(), geo[1].data_ptr(), None, 1, p.data_ptr(), N,
                                  None if s is None else s.data_ptr(), N // 2, None, None, None, B, c, ws.data_ptr(), nb, st),
               "tiles")
    x, gx, dp = torch.zeros_like(y), torch.zeros_like(y), torch.zeros(L, N, device="cuda")
    _lib.check(lib.mg_propagate(2, N, L, B, 1, 0, y.data_ptr(), g.data_ptr(), x.data_ptr(), gx.data_ptr(), N, dp.data_ptr(), N,
                                0, c, ws.data_ptr(), nb, st), "propagate")
    assert lib.mg_read_status(ws.data_ptr(), 1, st) == 0
    f = None
    if cfg is None:                                      # forward on the same tiles
        f = torch.zeros_like(y)
        _lib.check(lib.mg_propagate(3, N, L, B, 1, 0, x.data_ptr(), None, f.data_ptr(), None, N, None, 0, 0, c, ws.data_ptr(),
                                    nb, st), "forward")
    return x, gx, dp, f


@pytest.mark.parametrize("B", [1, 700, 1300, 2500])      # 1, 2 and 4 vectors per lane
@pytest.mark.parametrize("N,geo", [(34, "reck"), (64, "clements"), (66, "clements"), (128, "reck"), (130, "clements"),
                                   (256, "clements"), (258, "reck"), (512, "clements")])
def test_gradients(N, geo, B):
    from meshes_gb300 import _lib
    rng = np.random.default_rng(N + B)
    om = O.random_mesh(rng, N, geo, "sym", 0.02 if N % 4 else 0.0)
    L = min(om.L, 17)
    om = O.OracleMesh(N=N, L=L, crossing="sym", lens=list(om.lens[:L]), shifts=list(om.shifts[:L]),
                      p=np.ascontiguousarray(om.p[:L]), s=None if om.s is None else np.ascontiguousarray(om.s[:L]))
    y, g = (torch.tensor(O.unit_columns(rng, N, B), dtype=torch.complex64, device="cuda") for _ in range(2))
    x, gx, dp, f = _run(om, B, None, y, g)
    G, xin, gin = O.vjp_unitary(om, y.cpu().numpy(), g.cpu().numpy())
    dp_ref = O.contract_dp(om, G)
    assert O.rel_err(gx.cpu().numpy(), gin) < TOL
    assert O.rel_err(dp.cpu().numpy().reshape(dp_ref.shape), dp_ref) < TOL
    assert O.rel_err(f.cpu().numpy(), y.cpu().numpy()) < TOL
    x2, gx2, dp2, _ = _run(om, B, _lib.config(8 if N <= 256 else 16, 4 if N <= 256 else 2, 0, 0, 0, 2), y, g)
    assert torch.equal(x, x2) and torch.equal(gx, gx2)
    assert O.rel_err(dp.cpu().numpy(), dp2.cpu().numpy()) < TOL
