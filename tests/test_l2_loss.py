"""mg_l2_loss (J = sum |y - t|^2 in one pass) against 64-bit sums: sizes around its one-cluster limit and the vector width, fields
off 16-byte alignment, no scratch, and through mesh_l2_loss.  Tolerance: the differences and squares round to 2^-24 each and 32
of them are added in float, a relative 2^-22 for sums of squares."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -22 + 2.0 ** -24


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("scratch", [0, 2, 304])
@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 127, 65537, 262143, 262144, 262145, (1 << 20) + 3, 5_000_000])
def test_sum(n, scratch, offset):
    from meshes_gb300 import _lib
    rng = np.random.default_rng(n + offset)
    y, t = (rng.normal(size=n).astype(np.float32) for _ in range(2))
    yd, td = torch.zeros(n + 4, device="cuda"), torch.zeros(n + 4, device="cuda")
    yd[offset:offset + n], td[offset:offset + n] = torch.tensor(y), torch.tensor(t)
    out = torch.full((), float("nan"), device="cuda")
    part = torch.full((max(scratch, 1),), float("nan"), dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    got = []
    for _ in range(2):
        _lib.check(_lib.load().mg_l2_loss(yd.data_ptr() + 4 * offset, td.data_ptr() + 4 * offset, n, out.data_ptr(),
                                          part.data_ptr() if scratch else None, scratch, st), "mg_l2_loss")
        got.append(float(out))
    want = float(((y.astype(np.float64) - t) ** 2).sum())
    assert abs(got[0] - want) <= TOL * want
    assert got[0] == got[1]


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_not_finite(value):
    from meshes_gb300 import _lib
    y, t, out = torch.zeros(1000, device="cuda"), torch.zeros(1000, device="cuda"), torch.zeros((), device="cuda")
    y[777] = value
    _lib.check(_lib.load().mg_l2_loss(y.data_ptr(), t.data_ptr(), 1000, out.data_ptr(), None, 0,
                                      torch.cuda.current_stream().cuda_stream), "mg_l2_loss")
    assert np.isnan(float(out)) if np.isnan(value) else float(out) == float("inf")
