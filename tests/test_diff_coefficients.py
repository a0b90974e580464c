"""The derivative entries of a forward-mode tile (float-float, one lane of a quad per entry): one layer, unit vectors, against
the oracle's complex128 derivatives - phases at their extremes and beyond the float-float range (400), splitters and
none, pairs within a lane, across lanes and odd-shift.  Tolerance: two float32 products and their sum of entries rounded once,
3 x 2^-24 of the direction's size, and 1e-9."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splitters", [True, False])
@pytest.mark.parametrize("N,shift,stride", [(16, 0, None), (16, 1, None), (130, 1, None), (64, 0, 0), (64, 0, 5), (256, 0, 4)])
def test_one_layer(N, shift, stride, splitters):
    from meshes_gb300 import _lib
    rng = np.random.default_rng(N + shift)
    n = N // 2 if stride is not None or shift == 0 else N // 2 - 1
    p = rng.uniform(-7, 7, (1, N // 2, 2)).astype(np.float32)
    special = [0.0, np.pi, np.pi / 2, -np.pi, 399.0, 401.0, 1e4, 1e-20]
    p[0, :len(special), 0] = special
    p[0, :len(special), 1] = special[::-1]
    s = rng.normal(0, 0.3, (1, N // 2, 2)).astype(np.float32) if splitters else None
    kw = dict(strides=[stride]) if stride is not None else dict(lens=[n], shifts=[shift])
    d = rng.normal(size=p.shape).astype(np.float32)
    if stride is None:
        d[0, n:] = 0                                     # (slot q of an odd layer starts at mode 2 q + 1: the last is inactive)
    x = np.eye(N)

    def y(q):
        return O.propagate(O.OracleMesh(N=N, L=1, crossing="mzi", p=q, s=None if s is None else s.astype(np.float64), **kw), x)

    # T is affine in e^{i th} and in e^{i ph}: its derivative is i (T(.) - T(. + pi)) / 2, with no difference quotient (whose
    # step a phase of 1e4 rounds by 1e-6 of itself)
    q, want = p.astype(np.float64), np.zeros((N, N), complex)
    for k in range(2):
        turned = q.copy()
        turned[..., k] += np.pi
        change = 0.5j * (y(q) - y(turned))
        for slot, a, b in O.OracleMesh(N=N, L=1, crossing="mzi", p=q, s=s, **kw).slots(0):
            want[:, [a, b]] += d[0, slot, k] * change[:, [a, b]]
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    geo = 0 if stride is None else 1
    nb = lib.mg_workspace_bytes(1, N, 1, N, 0, geo, None)
    ws = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
    _lib.check(lib.mg_workspace_init(ws.data_ptr(), nb, st), "init")
    g = [torch.tensor([a], dtype=torch.int32, device="cuda") for a in ((n, shift) if geo == 0 else (stride,))]
    ptr = [t.data_ptr() for t in g]
    pd, dd = torch.tensor(p.reshape(-1), device="cuda"), torch.tensor(d.reshape(-1), device="cuda")
    sd = None if s is None else torch.tensor(s.reshape(-1), device="cuda")
    _lib.check(lib.mg_build_tiles(1, N, 1, geo, *((ptr + [None]) if geo == 0 else ([None, None] + ptr)), 0, pd.data_ptr(), N,
                                  None if sd is None else sd.data_ptr(), N, dd.data_ptr(), None, None, N, None, ws.data_ptr(),
                                  nb, st), "tiles")
    xd = torch.tensor(x, dtype=torch.complex64, device="cuda")
    zero, yo, dy = torch.zeros_like(xd), torch.zeros_like(xd), torch.zeros_like(xd)
    _lib.check(lib.mg_propagate(1, N, 1, N, 0, geo, xd.data_ptr(), zero.data_ptr(), yo.data_ptr(), dy.data_ptr(), N, None, 0, 0,
                                None, ws.data_ptr(), nb, st), "propagate")
    assert lib.mg_read_status(ws.data_ptr(), 1, st) == 0
    size = np.abs(d).sum(axis=2).max()
    assert np.abs(dy.cpu().numpy() - want).max() <= 3 * 2.0 ** -24 * size + 1e-9


def test_float_float_is_no_further_off_than_double():
    """dT/dth and T of 131072 slots, alone and rounded once to float32.  Where that is not the nearest float, the value before the
    rounding lay on the wrong side of the middle between two, by as much as the error goes beyond the nearest float's.  Bound:
    two sines or cosines of the product off by 2e-14 (where the double-precision form stops its series, and the float tail of the
    float-float sine ends) and ten operations of 2^-48."""
    from meshes_gb300 import _lib
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    N = L = 256
    h, cfg, info = N // 2, _lib.config(8, 2, 4, 8, 0, 2), _lib.mg_plan_info()
    assert lib.mg_plan(1, N, L, 64, 0, 0, _lib.cfg_ptr(cfg), ctypes.byref(info)) == 0, _lib.last_error()
    M, G = info.M, info.G
    lens, shifts = (torch.full((L,), v, dtype=torch.int32, device="cuda") for v in (h, 0))
    beyond = 0.0
    for seed in (8, 9, 10, 11):
        rng = np.random.default_rng(seed)
        p, s = rng.uniform(-7, 7, (L, h, 2)).astype(np.float32), rng.normal(0, 0.3, (L, h, 2)).astype(np.float32)
        d = np.zeros_like(p)
        d[..., 0] = 1
        pd, sd, dd = (torch.tensor(a.reshape(-1), device="cuda") for a in (p, s, d))
        ws = torch.zeros(info.total, dtype=torch.uint8, device="cuda")
        _lib.check(lib.mg_build_tiles(1, N, L, 0, lens.data_ptr(), shifts.data_ptr(), None, 0, pd.data_ptr(), N, sd.data_ptr(), N,
                                      dd.data_ptr(), None, None, 64, _lib.cfg_ptr(cfg), ws.data_ptr(), info.total, st), "tiles")
        raw = ws.cpu().numpy()[info.off_tiles:info.off_tiles + L * info.layer_bytes]
        tile = raw.copy().view(np.float32).reshape(L, 2, M // 2, 2, G, 2, 2)     # (T or dT), e, row, lane, column
        got = tile.transpose(0, 1, 4, 2, 3, 5, 6).reshape(L, 2, h, 2, 2, 2)
        th, ph, al, be = (a.astype(np.float64) for a in (p[..., 0], p[..., 1], s[..., 0], s[..., 1]))

        def T(th):
            e, f, S, C = np.exp(0.5j * th), np.exp(1j * ph), np.sin(th / 2), np.cos(th / 2)
            Sp, Cp, Sm, Cm = np.sin(al + be), np.cos(al + be), np.sin(al - be), np.cos(al - be)
            return np.stack([e * f * (-C * Sp + 1j * S * Cm), e * (-S * Sm + 1j * C * Cp),
                             e * f * (S * Sm + 1j * C * Cp), e * (-C * Sp - 1j * S * Cm)], -1).reshape(L, h, 2, 2)
        for k, want in enumerate((T(th), 0.5j * (T(th) - T(th + np.pi)))):
            want = np.stack([want.real, want.imag], -1)
            err = np.abs(got[:, k] - want)
            assert err.max() < 1e-6
            beyond = max(beyond, float((err - np.abs(want.astype(np.float32) - want)).max()))
    assert beyond <= 2 * 2e-14 + 10 * 2.0 ** -48
