"""Butterfly kernels (FFT meshes of 64 to 512 modes: fields turned between two orders instead of exchanged between lanes)
against the complex128 oracle and the general kernel on the same tiles, through the C ABI: forward from the batch on that
takes them, back-propagation from one vector on; the layers of an FFT mesh, reversed, repeated, in any order, a single
one; phases without splitters; a target instead of a gradient, accumulation, no input field wanted; and bad strides.
Tolerance: the library's 1e-5 relative Frobenius error."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _mesh(rng, N, order, crossing="mzi", splitters=True):
    k = N.bit_length() - 1
    strides = {"fft": list(range(k)), "reversed": list(range(k))[::-1], "one": [k - 1], "first": [0],
               "any": [int(e) for e in rng.integers(0, k, 11)]}[order]
    om = O.random_mesh(rng, N, "fft", crossing, 0.02 if splitters else 0.0)
    L = len(strides)
    p, s = np.asarray(om.p, np.float32), None if om.s is None else np.asarray(om.s, np.float32)
    pick = rng.integers(0, p.shape[0], L)
    return O.OracleMesh(N=N, L=L, crossing=crossing, lens=None, shifts=None, p=p[pick].copy(),
                        s=None if s is None or not splitters else s[pick].copy(), strides=strides)


class _Run:
    def __init__(self, om, op, B, cfg=None, crossing=0):
        from meshes_gb300 import _lib
        self.lib, self.check, self.om, self.B, self.X = _lib.load(), _lib.check, om, B, crossing
        self.c = _lib.cfg_ptr(cfg) if cfg is not None else None
        self.st = torch.cuda.current_stream().cuda_stream
        self.nb = self.lib.mg_workspace_bytes(op, om.N, om.L, B, crossing, 1, self.c)
        self.ws = torch.full((self.nb,), 255, dtype=torch.uint8, device="cuda")
        self.check(self.lib.mg_workspace_init(self.ws.data_ptr(), self.nb, self.st), "init")
        e = torch.tensor(om.strides, dtype=torch.int32, device="cuda")
        p = torch.tensor(np.asarray(om.p).reshape(-1), device="cuda")
        s = None if om.s is None else torch.tensor(np.asarray(om.s).reshape(-1), device="cuda")
        self.check(self.lib.mg_build_tiles(op, om.N, om.L, 1, None, None, e.data_ptr(), crossing, p.data_ptr(), om.N,
                                           s.data_ptr() if s is not None else None,
                                           om.N // 2 * (2 if crossing == 0 else 1), None, None, None, B, self.c,
                                           self.ws.data_ptr(), self.nb, self.st), "tiles")
        torch.cuda.synchronize()

    def __call__(self, op, in0, in1, out0, out1, dp=None, accumulate=0):
        ptr = (lambda t: None if t is None else t.data_ptr())
        self.check(self.lib.mg_propagate(op, self.om.N, self.om.L, self.B, self.X, 1, ptr(in0), ptr(in1), ptr(out0), ptr(out1),
                                         self.om.N, ptr(dp), self.om.N, accumulate, self.c, self.ws.data_ptr(), self.nb,
                                         self.st), "propagate")
        return self.lib.mg_read_status(self.ws.data_ptr(), 1, self.st)


def _dev(a):
    return torch.tensor(a, dtype=torch.complex64, device="cuda")


@pytest.mark.parametrize("order", ["fft", "reversed", "any", "one", "first"])
@pytest.mark.parametrize("N", [64, 128, 256, 512])
def test_forward(N, order):
    rng = np.random.default_rng(N)
    om = _mesh(rng, N, order)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch = {64: 8, 128: 8, 256: 4, 512: 4}[N]
    B = (1 if N == 64 else 8) * sms * batch + 3          # the first batches that take the butterfly kernel
    x = O.unit_columns(rng, N, B)
    y = torch.zeros(B, N, dtype=torch.complex64, device="cuda")
    assert _Run(om, 0, B)(0, _dev(x), None, y, None) == 0
    assert O.rel_err(y.cpu().numpy(), O.propagate(om, x)) < TOL


@pytest.mark.parametrize("crossing,code", [("sym", 1)])
def test_forward_of_other_crossings(crossing, code):
    rng = np.random.default_rng(5)
    om = _mesh(rng, 128, "any", crossing)
    B = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    x = O.unit_columns(rng, 128, B)
    y = torch.zeros(B, 128, dtype=torch.complex64, device="cuda")
    assert _Run(om, 0, B, crossing=code)(0, _dev(x), None, y, None) == 0
    assert O.rel_err(y.cpu().numpy(), O.propagate(om, x)) < TOL


@pytest.mark.parametrize("order", ["fft", "reversed", "any", "one", "first"])
@pytest.mark.parametrize("N,B", [(64, 1), (64, 8 * 152 * 8 + 9), (128, 7), (128, 1300), (256, 3), (256, 777), (256, 5001)])
def test_back_propagation(N, B, order):
    from meshes_gb300 import _lib
    rng = np.random.default_rng(N + B)
    om = _mesh(rng, N, order, splitters=order != "one")
    x, g = O.unit_columns(rng, N, B), O.unit_columns(rng, N, B)
    y_ref = O.propagate(om, x)
    G, _, gin = O.vjp_unitary(om, y_ref, g)
    dp_ref = O.contract_dp(om, G)
    xo, gx = torch.zeros(B, N, dtype=torch.complex64, device="cuda"), torch.zeros(B, N, dtype=torch.complex64, device="cuda")
    dp = torch.zeros(om.L, N, device="cuda")
    run = _Run(om, 2, B)
    assert run(2, _dev(y_ref), _dev(g), xo, gx, dp) == 0
    assert O.rel_err(xo.cpu().numpy(), x) < TOL
    assert O.rel_err(gx.cpu().numpy(), gin) < TOL
    assert O.rel_err(dp.cpu().numpy().reshape(dp_ref.shape), dp_ref) < TOL
    gx2 = torch.zeros_like(gx)                           # no input field wanted; the gradient added to the first
    assert run(2, _dev(y_ref), _dev(g), None, gx2, dp, 1) == 0
    assert torch.equal(gx, gx2)
    assert O.rel_err(dp.cpu().numpy().reshape(dp_ref.shape), 2 * dp_ref) < TOL
    # the general kernel on its own configuration
    gx3, dp3 = torch.zeros_like(gx), torch.zeros_like(dp)
    assert _Run(om, 2, B, _lib.config(8, 4, 0, 0, 0, 0))(2, _dev(y_ref), _dev(g), None, gx3, dp3) == 0
    assert O.rel_err(gx.cpu().numpy(), gx3.cpu().numpy()) < TOL
    # loss to a target formed in the kernel: g = 2 (y - t)
    t = _dev(y_ref) - 0.5 * _dev(g)
    assert run.lib.mg_propagate_l2(N, om.L, B, 0, 1, _dev(y_ref).data_ptr(), t.data_ptr(), None, gx2.data_ptr(), N,
                                   dp.data_ptr(), N, 0, None, run.ws.data_ptr(), run.nb, run.st) == 0
    torch.cuda.synchronize()
    assert O.rel_err(gx2.cpu().numpy(), gin) < TOL
    assert O.rel_err(dp.cpu().numpy().reshape(dp_ref.shape), dp_ref) < TOL


def test_bad_strides_are_reported():
    rng = np.random.default_rng(9)
    om = _mesh(rng, 256, "fft")
    om.strides[3] = 8                                    # pairs 256 apart in 256 modes
    x = _dev(O.unit_columns(rng, 256, 40))
    run = _Run(om, 2, 40)
    assert run(2, x, x, None, torch.zeros_like(x), torch.zeros(om.L, 256, device="cuda")) == 2
