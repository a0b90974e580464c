"""Framed launches (mg_config.split 5 and 6: crossings with a unit diagonal on the frame pass's tiles) against the
complex128 oracle, through the C ABI, for every instantiated tile: ragged batches, Clements, Reck and irregular
nearest-neighbour layers, ordinary phases, cross states (a diagonal entry of 0) and meshes that the frames do not suit
(the unframed body inside the same kernel).  Tolerance: the library's 1e-5 relative Frobenius error."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

TOL = 1e-5
# (modes per lane, vectors per lane, mixed warps, warps per CTA) per op; N that selects the modes per lane
FWD = [(4, 1, 0, 4), (4, 1, 0, 8), (4, 2, 0, 16), (4, 2, 1, 8), (4, 4, 0, 8), (4, 4, 1, 16), (8, 1, 0, 4), (8, 2, 0, 8),
       (8, 2, 1, 8), (8, 3, 0, 8), (8, 4, 0, 8), (8, 4, 1, 8), (16, 1, 0, 8), (16, 2, 0, 8), (16, 2, 1, 8), (16, 3, 0, 8),
       (16, 4, 0, 8), (20, 1, 0, 8), (20, 2, 0, 8), (20, 2, 1, 8), (20, 3, 0, 8)]
BWD = [(4, 1, 0, 4), (4, 1, 0, 8), (4, 2, 0, 16), (4, 2, 1, 8), (4, 4, 0, 8), (4, 4, 1, 16), (8, 1, 0, 4), (8, 2, 0, 8),
       (8, 2, 1, 8), (8, 3, 0, 8), (8, 4, 0, 8), (8, 4, 1, 8), (16, 1, 0, 4), (16, 1, 0, 8), (16, 2, 0, 8),
       (16, 2, 1, 8), (20, 1, 0, 4), (20, 1, 0, 8), (20, 2, 0, 8), (20, 2, 1, 8)]
SIZES = {4: (66, 128), 8: (130, 256), 16: (258, 400), 20: (514, 640)}


def _mesh(rng, N, kind, L=None):
    """Oracle mesh: geometry and phases of one kind, L layers (the first of the geometry's)."""
    if kind == "irregular":          # runs of equal shifts, layers of any extent, an odd number of them
        L = L or 23
        shifts = rng.integers(0, 2, L) + 2 * rng.integers(0, N // 8, L)
        lens = [int(rng.integers(0, (N - sh) // 2 + 1)) for sh in shifts]
        shifts = shifts.tolist()
    else:
        lens, shifts = O.reck_geometry(N) if kind == "reck" else O.clements_geometry(N)
        L = L or min(len(lens), 61)
        lens, shifts = list(lens[:L]), list(shifts[:L])
    om = O.OracleMesh(N=N, L=L, crossing="mzi", lens=lens, shifts=shifts,
                      p=rng.uniform(0, 2 * np.pi, (L, N // 2, 2)).astype(np.float32),
                      s=rng.normal(0, 0.02, (L, N // 2, 2)).astype(np.float32))
    mask = om.active_mask()
    if kind == "cross":              # theta = 0 and ideal splitters: t00 = t11 = 0
        om.p[..., 0] = 0
        om.s[:] = 0
    if kind == "few_cross":
        pick = rng.random(mask.shape) < 0.03
        om.p[pick] = 0
        om.s[pick] = 0
    if kind == "flat":               # one splitter of beta = pi/4: cos(pi/4 + beta) = 0
        q = np.argwhere(mask)[3]
        om.s[q[0], q[1], 1] = np.pi / 4
    om.p[~mask] = 0
    om.s[~mask] = 0
    return om


class _Run:
    def __init__(self, om, op, B, cfg):
        from meshes_gb300 import _lib
        self.lib, self.check, self.om, self.B = _lib.load(), _lib.check, om, B
        self.c = _lib.cfg_ptr(_lib.config(*cfg)) if cfg else None
        self.st = torch.cuda.current_stream().cuda_stream
        self.nb = self.lib.mg_workspace_bytes(op, om.N, om.L, B, 0, 0, self.c)
        assert self.nb, _lib.last_error()
        self.ws = torch.full((self.nb,), 255, dtype=torch.uint8, device="cuda")     # stale bits must not matter
        self.check(self.lib.mg_workspace_init(self.ws.data_ptr(), self.nb, self.st), "init")
        dev = [torch.tensor(np.asarray(a), device="cuda") for a in
               (np.int32(om.lens), np.int32(om.shifts), om.p.reshape(-1), om.s.reshape(-1))]
        self.check(self.lib.mg_build_tiles(op, om.N, om.L, 0, dev[0].data_ptr(), dev[1].data_ptr(), None, 0,
                                           dev[2].data_ptr(), om.N, dev[3].data_ptr(), om.N, None, None, None, B, self.c,
                                           self.ws.data_ptr(), self.nb, self.st), "mg_build_tiles")

    def propagate(self, op, *args):
        self.check(self.lib.mg_propagate(op, self.om.N, self.om.L, self.B, 0, 0, *args, self.c, self.ws.data_ptr(),
                                         self.nb, self.st), "mg_propagate")
        assert self.lib.mg_read_status(self.ws.data_ptr(), 0, self.st) == 0


def _c64(a):
    return torch.tensor(a, dtype=torch.complex64, device="cuda")


def _forward(om, x, cfg, op=0):
    r = _Run(om, 0 if op == 0 else 2, x.shape[0], cfg)
    xd = _c64(x)
    y = torch.empty_like(xd)
    r.propagate(op, xd.data_ptr(), None, y.data_ptr(), None, om.N, None, 0, 0)
    return y.cpu().numpy()


def _backward(om, y, g, cfg, accumulate=False):
    r = _Run(om, 2, y.shape[0], cfg)
    yd, gd = _c64(y), _c64(g)
    x, gx = torch.empty_like(yd), torch.empty_like(yd)
    dp = torch.full((om.p.size,), 0.25 if accumulate else float("nan"), device="cuda")
    r.propagate(2, yd.data_ptr(), gd.data_ptr(), x.data_ptr(), gx.data_ptr(), om.N, dp.data_ptr(), om.N, int(accumulate))
    return x.cpu().numpy(), gx.cpu().numpy(), dp.cpu().numpy().reshape(om.p.shape)


def _check_backward(om, B, rng, cfg, accumulate=False):
    x = O.unit_columns(rng, om.N, B)
    g = O.unit_columns(rng, om.N, B)
    y = O.propagate(om, x)
    G, _, gin = O.vjp_unitary(om, y, g)
    dp_ref = O.contract_dp(om, G)
    xo, gx, dp = _backward(om, y, g, cfg, accumulate)
    assert O.rel_err(xo, x) < TOL and O.rel_err(gx, gin) < TOL
    mask = om.active_mask()
    assert O.rel_err((dp - (0.25 if accumulate else 0.0))[mask], dp_ref[mask]) < TOL
    assert np.all(dp[~mask] == (0.25 if accumulate else 0.0))


def _cfg(t):
    M, V, mix, W = t
    return (M, V, W, 0, 0, 6 if mix else 5)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", FWD)
@pytest.mark.parametrize("big", [0, 1])
def test_forward_tiles(tile, big):
    rng = np.random.default_rng(100 * tile[0] + 10 * tile[1] + tile[2] + big)
    N = SIZES[tile[0]][big]
    for kind, B in (("clements", 77), ("irregular", 1)):
        om = _mesh(rng, N, kind)
        x = O.unit_columns(rng, N, B)
        assert O.rel_err(_forward(om, x, _cfg(tile)), O.propagate(om, x)) < TOL, kind


@pytest.mark.gpu
@pytest.mark.parametrize("tile", BWD)
@pytest.mark.parametrize("big", [0, 1])
def test_backward_tiles(tile, big):
    rng = np.random.default_rng(1000 + 100 * tile[0] + 10 * tile[1] + tile[2] + big)
    N = SIZES[tile[0]][big]
    for kind, B in (("clements", 77), ("reck", 3)):
        _check_backward(_mesh(rng, N, kind), B, rng, _cfg(tile))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["clements", "reck", "irregular", "cross", "few_cross", "flat"])
@pytest.mark.parametrize("L", [1, 2, 16, 17, 33, 129])
def test_layer_patterns(kind, L):
    """Segment and chunk edges of every layer pattern, forward from its own and from back-propagation tiles, and
    back-propagation overwriting and adding to dJ/dp."""
    rng = np.random.default_rng(L + len(kind))
    N = 130
    om = _mesh(rng, N, kind, L)
    x = O.unit_columns(rng, N, 41)
    y = O.propagate(om, x)
    assert O.rel_err(_forward(om, x, (8, 4, 8, 0, 0, 6)), y) < TOL
    assert O.rel_err(_forward(om, x, (8, 2, 8, 5, 3, 5)), y) < TOL
    assert O.rel_err(_forward(om, x, (8, 4, 8, 0, 0, 6), op=3), y) < TOL
    _check_backward(om, 41, rng, (8, 4, 8, 0, 0, 6))
    _check_backward(om, 41, rng, (8, 1, 4, 3, 2, 5), accumulate=True)


@pytest.mark.gpu
def test_nan_and_infinite_inputs():
    """A NaN phase, and fields that hold NaN or infinity, reach the outputs they reach without frames."""
    rng = np.random.default_rng(5)
    om = _mesh(rng, 130, "clements", 20)
    x = O.unit_columns(rng, 130, 8)
    x[2, 17] = np.nan
    x[5, 3] = np.inf
    a, b = _forward(om, x, (8, 4, 8, 0, 0, 5)), _forward(om, x, (8, 4, 8, 0, 0, 2))
    assert np.array_equal(np.isfinite(a), np.isfinite(b)) and not np.isfinite(a[2]).all()
    om.p[7, 30, 0] = np.nan
    x = O.unit_columns(rng, 130, 8)
    a, b = _forward(om, x, (8, 4, 8, 0, 0, 5)), _forward(om, x, (8, 4, 8, 0, 0, 2))
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isnan(a).any() and not np.isnan(a).all()


def test_framed_plans_on_the_host():
    """Which shapes take the framed launch by default, and that it is refused where no kernel covers it."""
    from meshes_gb300 import _lib
    lib = _lib.load()

    def plan(op, N, L, B, crossing=0, geo=0, cfg=None):
        i = _lib.mg_plan_info()
        rc = lib.mg_plan(op, N, L, B, crossing, geo, _lib.cfg_ptr(_lib.config(*cfg)) if cfg else None, ctypes.byref(i))
        return i if rc == 0 else None

    assert plan(2, 256, 256, 4096, cfg=(8, 4, 8, 0, 0, 6)).grid == 147         # 28 vectors per CTA
    big, small = plan(0, 256, 256, 4096), plan(0, 256, 256, 4096, cfg=(8, 4, 4, 0, 0, 1))
    assert (big.M, big.V, big.W, big.grid) == (8, 4, 8, 147) and big.total > small.total
    for bad in (dict(op=1, N=256), dict(op=0, N=256, crossing=2), dict(op=0, N=256, geo=1), dict(op=2, N=256, crossing=1),
                dict(op=0, N=64)):
        kw = dict(dict(crossing=0, geo=0), **bad)
        assert plan(kw["op"], kw["N"], 16, 64, kw["crossing"], kw["geo"], (8, 4, 8, 0, 0, 5)) is None
    assert plan(0, 256, 256, 64, cfg=(8, 4, 4, 0, 0, 6)) is None               # mixed warps come in eights
    assert plan(2, 600, 600, 2048).total > 0 and plan(2, 2, 1, 1).total > 0


@pytest.mark.gpu
@pytest.mark.parametrize("N,B", [(100, 3000), (128, 9000), (200, 700)])
def test_layer_ranges_of_framed_tiles(N, B):
    """Tiles built for a whole-mesh launch that is framed (other modes per lane than the range's own choice at N <= 128)
    serve mg_propagate_range."""
    rng = np.random.default_rng(N)
    om = _mesh(rng, N, "clements")
    run = _Run(om, 0, B, None)
    x = O.unit_columns(rng, N, B)
    xd = torch.tensor(x, dtype=torch.complex64, device="cuda")
    mid, y = torch.zeros_like(xd), torch.zeros_like(xd)
    for l0, l1, src, dst in ((0, 20, xd, mid), (20, om.L, mid, y)):
        run.check(run.lib.mg_propagate_range(0, N, om.L, l0, l1, B, 0, 0, src.data_ptr(), None, dst.data_ptr(), None, N, None,
                                             None, 0, None, run.ws.data_ptr(), run.nb, run.st), "range")
    assert O.rel_err(y.cpu().numpy(), O.propagate(om, x)) < TOL
