"""Fields with a leading dimension above N: the same bits as with N, and nothing written beyond a vector's modes, for the kernels
that nearest-neighbour and butterfly meshes take by their size, batch and op (framed, full-warp, stored, butterfly)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O
from test_framed import _mesh

pytestmark = pytest.mark.gpu
MARK = 7.0 - 3.0j
PAD = 6


def _field(a, N, ldu):
    f = torch.full((a.shape[0], ldu), MARK, dtype=torch.complex64, device="cuda")
    f[:, :N] = a
    return f


class _Call:
    """Tiles of om and calls on them, with leading dimension ldu."""

    def __init__(self, om, X, geo, ldu, B, cfg=None, T=None):
        from meshes_gb300 import _lib
        self.lib, self.check, self.om, self.X, self.geo, self.ldu, self.B = _lib.load(), _lib.check, om, X, geo, ldu, B
        self.c, self.T = _lib.cfg_ptr(_lib.config(*cfg)) if cfg else None, T
        self.st = torch.cuda.current_stream().cuda_stream
        self.p = torch.tensor(np.asarray(om.p, np.float32).reshape(-1), device="cuda")
        self.s = torch.tensor(np.asarray(om.s, np.float32).reshape(-1), device="cuda")
        g = [om.strides] if geo else [om.lens, om.shifts]
        self.g = [torch.tensor(np.int32(a), device="cuda") for a in g]

    def build(self, op, dp=None):
        N, n_s = self.om.N, 2 if self.X == 0 else 1
        nb = self.lib.mg_workspace_bytes(op, N, self.om.L, self.B, self.X, self.geo, self.c)
        ws = torch.full((nb,), 255, dtype=torch.uint8, device="cuda")
        self.check(self.lib.mg_workspace_init(ws.data_ptr(), nb, self.st), "init")
        geo = [None, None, self.g[0].data_ptr()] if self.geo else [t.data_ptr() for t in self.g] + [None]
        par = [None, 0, None, 0] if self.X == 3 else [self.p.data_ptr(), N, self.s.data_ptr(), n_s * N // 2]
        self.check(self.lib.mg_build_tiles(op, N, self.om.L, self.geo, *geo, self.X, *par, None if dp is None else dp.data_ptr(),
                                           None if self.T is None else self.T.data_ptr(), None, self.B, self.c, ws.data_ptr(),
                                           nb, self.st), "mg_build_tiles")
        return ws, nb

    def out(self):
        return torch.full((self.B, self.ldu), MARK, dtype=torch.complex64, device="cuda")

    def done(self, ws, *fields):
        assert self.lib.mg_read_status(ws.data_ptr(), 0, self.st) == 0
        for f in fields:
            assert bool((f[..., self.om.N:] == MARK).all())
        return [f[..., :self.om.N].clone() for f in fields]

    def propagate(self, op, built, in0, in1=None, dp=None, x=True):
        ws, nb = built
        o0, o1 = self.out() if op != 2 or x else None, None if op in (0, 3) else self.out()
        ptr = (lambda t: None if t is None else t.data_ptr())
        self.check(self.lib.mg_propagate(op, self.om.N, self.om.L, self.B, self.X, self.geo, ptr(in0), ptr(in1), ptr(o0), ptr(o1),
                                         self.ldu, ptr(dp), self.om.N, 0, self.c, ws.data_ptr(), nb, self.st), "mg_propagate")
        return self.done(ws, *[f for f in (o0, o1) if f is not None])


def _both(run):
    a, b = run(0), run(PAD)
    assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b))


# op, N, layers, batch, crossing, configuration (None: the launch of that shape)
NN = [(0, 256, 256, 4096, 0, None), (0, 100, 60, 777, 0, (4, 1, 8, 0, 0, 5)), (0, 600, 40, 300, 0, (20, 3, 8, 0, 0, 5)),
      (0, 400, 40, 300, 0, (16, 2, 8, 0, 0, 6)), (0, 100, 30, 50, 0, None), (0, 50, 30, 700, 0, None), (0, 300, 12, 40, 0, None),
      (2, 256, 60, 2000, 0, None), (2, 100, 60, 777, 0, (4, 4, 16, 0, 0, 6)), (2, 600, 40, 300, 0, (20, 2, 8, 0, 0, 5)),
      (2, 400, 40, 300, 0, (16, 1, 4, 0, 0, 5)), (2, 50, 30, 700, 0, None), (2, 130, 20, 700, 1, None), (2, 34, 20, 100, 1, None),
      (1, 130, 20, 700, 0, None), (1, 300, 20, 300, 0, None), (1, 50, 20, 60, 0, None), (3, 256, 60, 2000, 0, None),
      (3, 100, 30, 50, 0, None)]


@pytest.mark.parametrize("op,N,L,B,X,cfg", NN)
def test_nearest_neighbour(op, N, L, B, X, cfg):
    def run(pad):
        rng = np.random.default_rng(N + op)
        om = _mesh(rng, N, "clements", L)
        if X:
            om.s = om.s[..., :1].copy()
        a, b = (torch.tensor(O.unit_columns(rng, N, B), dtype=torch.complex64, device="cuda") for _ in range(2))
        c = _Call(om, X, 0, N + pad, B, cfg)
        dp = torch.tensor(rng.normal(size=(L, N)).astype(np.float32), device="cuda")
        built = c.build(2 if op == 3 else op, dp if op == 1 else None)
        fields = [_field(t, N, c.ldu) for t in (a, b)]
        got = c.propagate(op, built, fields[0], None if op in (0, 3) else fields[1], dp if op == 2 else None)
        if op == 2:
            got += c.propagate(op, built, *fields, dp, x=False) + [dp]
            gx = c.out()
            c.check(c.lib.mg_propagate_l2(N, L, B, X, 0, fields[0].data_ptr(), fields[1].data_ptr(), None, gx.data_ptr(), c.ldu,
                                          dp.data_ptr(), N, 0, c.c, built[0].data_ptr(), built[1], c.st), "mg_propagate_l2")
            got += c.done(built[0], gx) + [dp]
        return got
    _both(run)


@pytest.mark.parametrize("op,N,B", [(0, 64, 1300), (0, 128, 2000), (0, 256, 900), (0, 512, 700), (2, 64, 77), (2, 128, 500),
                                    (2, 256, 333)])
def test_butterfly(op, N, B):
    def run(pad):
        rng = np.random.default_rng(N + op)
        om = O.random_mesh(rng, N, "fft", "mzi", 0.02)
        a, b = (torch.tensor(O.unit_columns(rng, N, B), dtype=torch.complex64, device="cuda") for _ in range(2))
        c = _Call(om, 0, 1, N + pad, B, (0, 0, 0, 0, 0, 7))
        dp = torch.zeros(om.L, N, device="cuda")
        return c.propagate(op, c.build(op), _field(a, N, c.ldu), _field(b, N, c.ldu) if op else None, dp if op else None) + [dp]
    _both(run)


@pytest.mark.parametrize("N,B", [(64, 300), (128, 700), (200, 100)])
def test_stored_inputs(N, B):
    def run(pad):
        rng = np.random.default_rng(N)
        om = _mesh(rng, N, "clements", 12)
        T = torch.tensor(np.ascontiguousarray(om.T_grid(), dtype=np.complex64), device="cuda")
        a, b = (torch.tensor(O.unit_columns(rng, N, B), dtype=torch.complex64, device="cuda") for _ in range(2))
        c = _Call(om, 3, 0, N + pad, B, None, T)
        (wf, nf), (wb, nb) = c.build(0), c.build(4)
        act = torch.full((om.L, B, c.ldu), MARK, dtype=torch.complex64, device="cuda")
        dT, y, gx = torch.zeros_like(T), c.out(), c.out()
        x, g = _field(a, N, c.ldu), _field(b, N, c.ldu)
        for op, in0, in1, o0, o1, d, ws, n in ((0, x, None, y, None, None, wf, nf), (4, None, g, None, gx, dT, wb, nb)):
            ptr = (lambda t: None if t is None else t.data_ptr())
            c.check(c.lib.mg_propagate_range(op, N, om.L, 0, om.L, B, 3, 0, ptr(in0), ptr(in1), ptr(o0), ptr(o1), c.ldu,
                                             act.data_ptr(), ptr(d), 0, None, ws.data_ptr(), n, c.st), "mg_propagate_range")
        return c.done(wf, y, act) + c.done(wb, gx) + [dT]
    _both(run)


@pytest.mark.parametrize("op", [0, 2])
def test_batched(op):
    """Framed and plain items of the persistent launches."""
    from meshes_gb300 import _lib
    from meshes_gb300.batched import BatchedMeshes, _to_device
    from test_batched import gpu_mesh
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream

    def run(pad):
        rng = np.random.default_rng(5)
        om = _mesh(rng, 256, "clements", 40)
        bm = BatchedMeshes([gpu_mesh(om)], [40])
        a, b = (torch.tensor(O.unit_columns(rng, 256, 40), dtype=torch.complex64, device="cuda") for _ in range(2))
        fields = [_field(t, 256, 256 + pad) for t in (a, b)]
        got = []
        for V, launch in ((4, lib.mg_batched_framed), (1, lib.mg_batched_small), (4, lib.mg_batched_small)):
            ds, smem = bm.states[0].framed_descriptors()
            d, out = ds[op], torch.full((40, 256 + pad), MARK, dtype=torch.complex64, device="cuda")
            n = -(-40 // (8 * V))
            partial, dp = torch.zeros(n, om.L, 128, 2, device="cuda"), torch.zeros(om.p.shape, device="cuda")
            scales = torch.zeros(n, dtype=torch.int32, device="cuda")
            d.V, d.mesh.ldu, d.mesh.n_items, d.mesh.in0 = V, 256 + pad, n, fields[0].data_ptr()
            if op == 0:
                d.mesh.out0 = out.data_ptr()
            else:
                d.mesh.in1, d.mesh.out0, d.mesh.out1 = fields[1].data_ptr(), None, out.data_ptr()
                d.mesh.partial, d.mesh.dp, d.scales = partial.data_ptr(), dp.data_ptr(), scales.data_ptr()
            dev = _to_device((_lib.mg_batch_framed * 1)(d), out.device)
            its = _to_device((_lib.mg_batch_item * n)(*[(0, k * 8 * V, min((k + 1) * 8 * V, 40), k) for k in range(n)]), out.device)
            head, status = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
            _lib.check(launch(op, dev.data_ptr(), 1, its.data_ptr(), n, head.data_ptr(), 3, smem[op], status.data_ptr(), st), "batch")
            if op:
                _lib.check(lib.mg_batched_framed_reduce(dev.data_ptr(), 1, st), "reduce")
            assert int(status) == 0 and bool((out[:, 256:] == MARK).all())
            got += [out[:, :256].clone(), dp]
        return got
    _both(run)


@pytest.mark.parametrize("N,B", [(256, 4096), (100, 50)])
def test_results_into_wider_arrays(N, B):
    """MeshNetworkGPU: fields from and into columns of arrays with a longer column."""
    from test_batched import gpu_mesh
    rng = np.random.default_rng(N)
    mesh = gpu_mesh(_mesh(rng, N, "clements"))
    x = torch.tensor(O.unit_columns(rng, N, B), dtype=torch.complex64, device="cuda")
    y = mesh.dot(x.t())
    wide, out = _field(x, N, N + PAD), torch.full((B, N + PAD), MARK, dtype=torch.complex64, device="cuda")
    got = mesh.dot(wide[:, :N].t(), out=out[:, :N].t())
    assert got.data_ptr() == out.data_ptr() and torch.equal(out[:, :N], y.t()) and bool((out[:, N:] == MARK).all())
