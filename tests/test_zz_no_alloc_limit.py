"""mg_fwdprop_noalloc on meshes whose framed launch does not fit its fixed scratch array but whose plain one does, against the
complex128 oracle (the library's 1e-5 relative Frobenius error)."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [400, 600])
def test_plain_launch_where_it_alone_fits(N):
    from meshes_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(N)
    om = O.random_mesh(rng, N, "clements", "mzi", 0.02)
    B = 2000
    assert lib.mg_workspace_bytes(0, N, om.L, B, 0, 0, None) > 8 << 20
    x = O.unit_columns(rng, N, B)
    xd = torch.tensor(x, dtype=torch.complex64, device="cuda")
    y = torch.zeros_like(xd)
    lens, shifts = (torch.tensor(a, dtype=torch.int32, device="cuda") for a in (om.lens, om.shifts))
    p, s = torch.tensor(om.p.reshape(-1), device="cuda"), torch.tensor(om.s.reshape(-1), device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    rc = lib.mg_fwdprop_noalloc(N, om.L, B, lens.data_ptr(), shifts.data_ptr(), p.data_ptr(), N, s.data_ptr(), N, xd.data_ptr(),
                                y.data_ptr(), N, 0, st)
    assert rc == 0, _lib.last_error()
    torch.cuda.synchronize()
    assert O.rel_err(y.cpu().numpy()[:40], O.propagate(om, x[:40])) < 1e-5
    assert O.rel_err(y.cpu().numpy()[-3:], O.propagate(om, x[-3:])) < 1e-5
