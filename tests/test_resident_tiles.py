"""Tiles that were built once serve every batch: mg_build_tiles runs at one, and calls of batches on both sides of every rule
that picks a launch by its batch (vectors per lane, modes per lane, framed or not) read them, against the complex128
oracle.  Tolerance: the library's 1e-5 relative Frobenius error."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

TOL = 1e-5
FWD, BWD, FWD_BWDTILES, BWD_STORED = 0, 2, 3, 4
ONE_BATCH = 8
BATCHES = (1, 65, 600, 1000, 2500, 4096, 5200, 6000, 9000, 30000)


def _plan(op, N, L, B, X, geo=0):
    from meshes_gb300 import _lib
    i = _lib.mg_plan_info()
    assert _lib.load().mg_plan(op, N, L, B, X, geo, None, ctypes.byref(i)) == 0, _lib.last_error()
    return i


@pytest.mark.parametrize("X", [0, 1, 2, 3])
@pytest.mark.parametrize("op", [FWD, 1, BWD, BWD_STORED])
def test_batch_does_not_enter_the_tiles(op, X):
    """Each set of tiles (by modes per lane) has its place, and the partials begin behind all of them, whatever the batch."""
    if (X == 3 and op == 1) or (X == 2 and op == BWD_STORED):
        pytest.skip("no such launch")
    for N in (8, 34, 64, 66, 100, 128, 130, 256, 300, 512, 640):
        if N == 640 and op == BWD_STORED:
            continue                                     # (not instantiated)
        for L in (1, 8, 40, N):
            plans = [_plan(op, N, L, B, X) for B in BATCHES]
            places = {}
            for p in plans:
                assert places.setdefault(p.M, p.off_tiles) == p.off_tiles
            assert len({p.off_partial for p in plans}) == 1 and len({p.layer_bytes for p in plans}) == 1
            at = sorted(places.values())
            assert all(b - a >= L * plans[0].layer_bytes for a, b in zip(at, at[1:])) and len(at) <= 2
            assert at[-1] + L * plans[0].layer_bytes <= plans[0].off_partial
            if op == BWD_STORED or X == 3:
                continue
            for B in BATCHES:                            # what the entry points that build for each call need
                assert _plan(op, N, L, B, X, ONE_BATCH).total <= _lib_bytes(op, N, L, B, X)


def _lib_bytes(op, N, L, B, X):
    from meshes_gb300 import _lib
    return _lib.load().mg_workspace_bytes(op, N, L, B, X, 0, None)


@pytest.mark.skipif(torch.cuda.is_available(), reason="calls on addresses that nothing may be launched on")
@pytest.mark.parametrize("X", [0, 1])
def test_a_workspace_holds_every_smaller_batch(X):
    """Back-propagation of no batch is refused for want of space (MG_E_WORKSPACE, before the launch that fails here for want of
    a device) in a workspace of a larger one's size."""
    from meshes_gb300 import _lib
    lib = _lib.load()
    Bs = (1, 7, 600, 1216, 2500, 4096, 4864, 4900, 6000, 9000, 19000, 30000, 99000, 100000)
    a = 1 << 20                                          # an aligned address that is not looked at
    for N in (8, 32, 34, 64, 100, 128, 130, 256, 400, 512, 600, 640):
        for L in (1, 20, N):
            sizes = [_lib_bytes(BWD, N, L, B, X) for B in Bs]
            for n, nb in enumerate(sizes):
                for B in Bs[:n + 1]:
                    rcs = [lib.mg_propagate(BWD, N, L, B, X, 0, a, a, None, a, N, a, N, 0, None, a, nb, None),
                           lib.mg_propagate(FWD_BWDTILES, N, L, B, X, 0, a, None, a, None, N, None, 0, 0, None, a, nb, None),
                           lib.mg_propagate_l2(N, L, B, X, 0, a, a, None, a, N, a, N, 0, None, a, nb, None),
                           lib.mg_backdiff(N, L, B, a, a, a, a, N, a, N, a, a, None, a, N, X, 0, a, nb, None)]
                    assert rcs == [-3] * 4, (N, L, Bs[n], B, _lib.last_error())


class _Tiles:
    """op's tiles of om in a workspace for all of Bs, built with B_build."""

    def __init__(self, om, op, B_build, Bs, T=None):
        from meshes_gb300 import _lib
        self.lib, self.check, self.om = _lib.load(), _lib.check, om
        self.X = {"mzi": 0, "sym": 1}[om.crossing] if T is None else 3
        self.st = torch.cuda.current_stream().cuda_stream
        self.nb = max(self.lib.mg_workspace_bytes(op, om.N, om.L, b, self.X, 0, None) for b in (B_build, *Bs))
        self.ws = torch.full((self.nb,), 255, dtype=torch.uint8, device="cuda")     # stale bits must not matter
        self.check(self.lib.mg_workspace_init(self.ws.data_ptr(), self.nb, self.st), "init")
        n_s = 2 if om.crossing == "mzi" else 1
        d = [torch.tensor(np.asarray(a), device="cuda") for a in
             (np.int32(om.lens), np.int32(om.shifts), om.p.reshape(-1), om.s.reshape(-1))]
        h = om.N // 2
        args = (d[2].data_ptr(), 2 * h, d[3].data_ptr(), n_s * h) if T is None else (None, 0, None, 0)
        self.check(self.lib.mg_build_tiles(op, om.N, om.L, 0, d[0].data_ptr(), d[1].data_ptr(), None, self.X, *args, None,
                                           None if T is None else T.data_ptr(), None, B_build, None, self.ws.data_ptr(),
                                           self.nb, self.st), "mg_build_tiles")

    def run(self, op, B, *args):
        self.check(self.lib.mg_propagate(op, self.om.N, self.om.L, B, self.X, 0, *args, None, self.ws.data_ptr(), self.nb,
                                         self.st), "mg_propagate")
        self.ok()

    def ok(self):
        assert self.lib.mg_read_status(self.ws.data_ptr(), 0, self.st) == 0


def _mesh(rng, N, L, crossing="mzi"):
    lens, shifts = O.clements_geometry(N)
    L = min(L, len(lens))
    om = O.OracleMesh(N=N, L=L, crossing=crossing, lens=list(lens[:L]), shifts=list(shifts[:L]),
                      p=rng.uniform(0, 2 * np.pi, (L, N // 2, 2)).astype(np.float32),
                      s=rng.normal(0, 0.02, (L, N // 2, 2 if crossing == "mzi" else 1)).astype(np.float32))
    mask = om.active_mask()
    om.p[~mask] = 0
    om.s[~mask] = 0
    return om


def _c64(a):
    return torch.tensor(a, dtype=torch.complex64, device="cuda")


# (N, L, batches of the build, batches of the calls)
CASES = [(64, 24, (700, 6000), (1, 700, 2600, 6000)), (100, 100, (1, 6000), (1, 1000, 4096, 6000)),
         (128, 60, (128, 9000), (1, 128, 2000, 9000)), (256, 100, (300, 4096), (1, 1000, 4096)),
         (400, 60, (64, 2432), (64, 2432)), (600, 40, (1, 2048), (1, 2048))]


@pytest.mark.gpu
@pytest.mark.parametrize("crossing", ["mzi", "sym"])
@pytest.mark.parametrize("N,L,built,called", CASES)
def test_forward(N, L, built, called, crossing):
    rng = np.random.default_rng(N)
    om = _mesh(rng, N, L, crossing)
    x = O.unit_columns(rng, N, max(called))
    y = O.propagate(om, x)
    xd = _c64(x)
    for b in built:
        for op, src in ((FWD, FWD), (FWD_BWDTILES, BWD)):
            t = _Tiles(om, src, b, called)
            for B in called:
                out = torch.zeros_like(xd[:B])
                t.run(op, B, xd.data_ptr(), None, out.data_ptr(), None, N, None, 0, 0)
                assert O.rel_err(out.cpu().numpy(), y[:B]) < TOL, (b, B, op)


@pytest.mark.gpu
@pytest.mark.parametrize("crossing", ["mzi", "sym"])
@pytest.mark.parametrize("N,L,built,called", CASES)
def test_backward(N, L, built, called, crossing):
    rng = np.random.default_rng(N + 1)
    om = _mesh(rng, N, min(L, 30), crossing)
    x, g = O.unit_columns(rng, N, max(called)), O.unit_columns(rng, N, max(called))
    y = O.propagate(om, x)
    yd, gd = _c64(y), _c64(g)
    refs = {B: O.vjp_unitary(om, y[:B], g[:B]) for B in called}
    for b in built:
        t = _Tiles(om, BWD, b, called)
        for B in called:
            xo, gx = torch.zeros_like(yd[:B]), torch.zeros_like(yd[:B])
            dp = torch.zeros(om.p.shape, device="cuda")
            t.run(BWD, B, yd.data_ptr(), gd.data_ptr(), xo.data_ptr(), gx.data_ptr(), N, dp.data_ptr(), N, 0)
            G, _, gin = refs[B]
            assert O.rel_err(xo.cpu().numpy(), x[:B]) < TOL and O.rel_err(gx.cpu().numpy(), gin) < TOL, (b, B)
            assert O.rel_err(dp.cpu().numpy(), O.contract_dp(om, G)) < TOL, (b, B)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [64, 128, 200])
def test_layer_ranges(N):
    """Generic crossings: forward ranges, with and without stored inputs, and back-propagation from them."""
    rng = np.random.default_rng(N)
    om = _mesh(rng, N, 12)
    T = torch.tensor(np.ascontiguousarray(om.T_grid(), dtype=np.complex64), device="cuda")
    called = (1, 500, 3000, 7000)
    x, g = O.unit_columns(rng, N, max(called)), O.unit_columns(rng, N, max(called))
    y = O.propagate(om, x)
    xd, gd = _c64(x), _c64(g)
    for b in (100, 7000):
        tf, tb = _Tiles(om, FWD, b, called, T), _Tiles(om, BWD_STORED, b, called, T)
        for B in called:
            mid, out, gx = (torch.zeros_like(xd[:B]) for _ in range(3))
            act = torch.zeros((om.L, B, N), dtype=torch.complex64, device="cuda")
            dT = torch.zeros((om.L, N // 2, 2, 2), dtype=torch.complex64, device="cuda")

            def go(t, op, l0, l1, in0, in1, out0, out1, a, d):
                t.check(t.lib.mg_propagate_range(op, N, om.L, l0, l1, B, 3, 0, in0, in1, out0, out1, N, a, d, 0, None,
                                                 t.ws.data_ptr(), t.nb, t.st), "mg_propagate_range")
                t.ok()
            go(tf, FWD, 0, 5, xd.data_ptr(), None, mid.data_ptr(), None, None, None)
            go(tf, FWD, 5, om.L, mid.data_ptr(), None, out.data_ptr(), None, None, None)
            assert O.rel_err(out.cpu().numpy(), y[:B]) < TOL, (b, B)
            go(tf, FWD, 0, om.L, xd.data_ptr(), None, None, None, act.data_ptr(), None)
            go(tb, BWD_STORED, 0, om.L, None, gd.data_ptr(), None, gx.data_ptr(), act.data_ptr(), dT.data_ptr())
            G, _, gin = O.vjp_unitary(om, y[:B], g[:B])
            assert O.rel_err(gx.cpu().numpy(), gin) < TOL, (b, B)
            assert O.rel_err(dT.cpu().numpy(), np.conj(G)) < TOL, (b, B)


@pytest.mark.gpu
@pytest.mark.parametrize("crossing", ["mzi", "sym"])
@pytest.mark.parametrize("N,L,Bmax,called", [(100, 20, 6000, (6000, 4864, 1, 1216)), (256, 128, 4096, (1216, 3000)),
                                             (256, 40, 10000, (9900, 5000)), (64, 20, 6000, (2600, 600)),
                                             (600, 10, 3000, (1900, 100)), (20, 20, 9000, (2500,))])
def test_smaller_batches_in_one_workspace(N, L, Bmax, called, crossing):
    """A workspace of the largest batch's size serves smaller ones, whose launches of their own may leave more partials:
    mg_propagate on resident tiles and the entry points that build for each call."""
    rng = np.random.default_rng(N + L)
    om = _mesh(rng, N, L, crossing)
    x, g = O.unit_columns(rng, N, Bmax), O.unit_columns(rng, N, Bmax)
    y = O.propagate(om, x)
    xd, yd, gd = _c64(x), _c64(y), _c64(g)
    t = _Tiles(om, BWD, Bmax, ())
    n_s = 2 if crossing == "mzi" else 1
    d = [torch.tensor(np.asarray(a), device="cuda") for a in (np.int32(om.lens), np.int32(om.shifts), om.p, om.s)]
    for one in (False, True):
        for B in called:
            out, xo, gx = (torch.zeros_like(yd[:B]) for _ in range(3))
            dp = torch.zeros(om.p.shape, device="cuda")
            if one:
                t.check(t.lib.mg_backdiff(N, om.L, B, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), dp.data_ptr(), N,
                                          d[3].data_ptr(), n_s * N // 2, yd.data_ptr(), gd.data_ptr(), xo.data_ptr(),
                                          gx.data_ptr(), N, t.X, 0, t.ws.data_ptr(), t.nb, t.st), "mg_backdiff")
                t.ok()
            else:
                t.run(FWD_BWDTILES, B, xd.data_ptr(), None, out.data_ptr(), None, N, None, 0, 0)
                assert O.rel_err(out.cpu().numpy(), y[:B]) < TOL, B
                t.run(BWD, B, yd.data_ptr(), gd.data_ptr(), xo.data_ptr(), gx.data_ptr(), N, dp.data_ptr(), N, 0)
            G, _, gin = O.vjp_unitary(om, y[:B], g[:B])
            assert O.rel_err(xo.cpu().numpy(), x[:B]) < TOL and O.rel_err(gx.cpu().numpy(), gin) < TOL, B
            assert O.rel_err(dp.cpu().numpy(), O.contract_dp(om, G)) < TOL, B
