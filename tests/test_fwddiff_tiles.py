"""Forward derivatives of nearest-neighbour complex meshes with a vector over the whole warp (2 to 16 modes per lane, 6 and 12
among them) against the general kernel on its own configuration - the same operations, so the same bits - and its
forward part against the complex128 oracle (the library's 1e-5 relative Frobenius error), at the edges of the widths."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O
from test_framed import _mesh

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _run(om, crossing, B, cfg, x, dx, dp):
    from meshes_gb300 import _lib
    lib, st, c = _lib.load(), torch.cuda.current_stream().cuda_stream, _lib.cfg_ptr(cfg) if cfg is not None else None
    N, L = om.N, om.L
    nb = lib.mg_workspace_bytes(1, N, L, B, crossing, 0, c)
    assert nb, _lib.last_error()
    ws = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
    _lib.check(lib.mg_workspace_init(ws.data_ptr(), nb, st), "init")
    geo = [torch.tensor(a, dtype=torch.int32, device="cuda") for a in (om.lens, om.shifts)]
    p, s = torch.tensor(om.p.reshape(-1), device="cuda"), torch.tensor(om.s.reshape(-1), device="cuda")
    _lib.check(lib.mg_build_tiles(1, N, L, 0, geo[0].data_ptr(), geo[1].data_ptr(), None, crossing, p.data_ptr(), N, s.data_ptr(),
                                  om.s.shape[1] * om.s.shape[2], dp.data_ptr(), None, None, B, c, ws.data_ptr(), nb, st), "tiles")
    y, dy = torch.zeros_like(x), torch.zeros_like(x)
    _lib.check(lib.mg_propagate(1, N, L, B, crossing, 0, x.data_ptr(), dx.data_ptr(), y.data_ptr(), dy.data_ptr(), N, None, 0,
                                0, c, ws.data_ptr(), nb, st), "propagate")
    assert lib.mg_read_status(ws.data_ptr(), 1, st) == 0
    return y, dy


@pytest.mark.parametrize("kind", ["clements", "irregular"])
@pytest.mark.parametrize("N", [34, 64, 66, 128, 130, 192, 194, 256, 258, 384, 386, 512])
@pytest.mark.parametrize("B", [1, 333, 1300, 5003])      # 1, 2 and 4 vectors per lane
def test_same_bits_as_the_general_kernel(N, B, kind):
    from meshes_gb300 import _lib
    if B > 2000 and N > 256:
        B = 2500
    rng = np.random.default_rng(N + B)
    om = _mesh(rng, N, kind, 19)
    x, dx = (torch.tensor(O.unit_columns(rng, N, B), dtype=torch.complex64, device="cuda") for _ in range(2))
    dp = torch.tensor(rng.normal(size=om.p.size).astype(np.float32), device="cuda")
    got = _run(om, 0, B, None, x, dx, dp)
    want = _run(om, 0, B, _lib.config(8 if N <= 256 else 16, 2 if N <= 256 else 1, 0, 0, 0, 2), x, dx, dp)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    if B <= 333:
        assert O.rel_err(got[0].cpu().numpy(), O.propagate(om, x.cpu().numpy())) < TOL


def test_sym_crossings():
    from meshes_gb300 import _lib
    rng = np.random.default_rng(3)
    om = O.random_mesh(rng, 150, "clements", "sym", 0.02)
    B = 700
    x, dx = (torch.tensor(O.unit_columns(rng, 150, B), dtype=torch.complex64, device="cuda") for _ in range(2))
    dp = torch.tensor(rng.normal(size=om.p.size).astype(np.float32), device="cuda")
    got, want = _run(om, 1, B, None, x, dx, dp), _run(om, 1, B, _lib.config(8, 2, 0, 0, 0, 2), x, dx, dp)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
