"""Batched meshes on framed tiles (complex, nearest-neighbour, 129 to 256 modes) against the complex128 oracle: batches at
the edges of a work item (32 vectors), few CTAs with many items each, meshes that the frames do not suit between others
(the unframed body in the same launch), and new phases.  Tolerance: the library's 1e-5 relative Frobenius error."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O
from test_batched import gpu_mesh
from test_framed import _mesh

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _check(bm, oms, xs, gs):
    for st, x, g in zip(bm.states, xs, gs):
        st.x.copy_(torch.tensor(x, dtype=st.x.dtype))
        st.gy.copy_(torch.tensor(g, dtype=st.gy.dtype))
    bm.step(True)
    assert bm.check_status() == 0
    for om, st, x, g in zip(oms, bm.states, xs, gs):
        y_ref = O.propagate(om, x)
        G, _, gin = O.vjp_unitary(om, y_ref, g)
        assert O.rel_err(st.y.cpu().numpy(), y_ref) < TOL, om.N
        assert O.rel_err(st.gx.cpu().numpy(), gin) < TOL, om.N
        assert O.rel_err(st.dp.cpu().numpy(), O.contract_dp(om, G)) < TOL, om.N


@pytest.mark.parametrize("grid", [2, None])
@pytest.mark.parametrize("others", [(), (("fft", "mzi", 64, 20), ("clements", "orth", 200, 37))])
def test_framed_batch(grid, others):
    from meshes_gb300.batched import BatchedMeshes
    rng = np.random.default_rng(71)
    kinds = [("clements", 130, 1), ("reck", 200, 33), ("irregular", 256, 32), ("flat", 256, 65), ("few_cross", 190, 31),
             ("clements", 256, 130)]
    oms = [_mesh(rng, N, kind) for kind, N, _ in kinds] + [O.random_mesh(rng, N, g, c, 0.0) for g, c, N, _ in others]
    Bs = [B for _, _, B in kinds] + [B for *_, B in others]
    bm = BatchedMeshes([gpu_mesh(om) for om in oms], Bs, grid=grid)
    assert [st.framed for st in bm.states] == [True] * len(kinds) + [False] * len(others)
    xs = [O.unit_columns(rng, om.N, B, real=om.crossing == "orth") for om, B in zip(oms, Bs)]
    gs = [O.unit_columns(rng, om.N, B, real=om.crossing == "orth") for om, B in zip(oms, Bs)]
    _check(bm, oms, xs, gs)
    for om in oms:                                        # new phases reach both directions
        om.p = np.where(np.asarray(om.p) == 0, 0, rng.uniform(0, 2 * np.pi, np.shape(om.p))).astype(np.float32)
    bm.update_phases([torch.tensor(np.asarray(om.p).reshape(-1), device="cuda") for om in oms])
    _check(bm, oms, xs, gs)


def test_items_outside_the_batch_are_refused():
    from meshes_gb300 import _lib
    from meshes_gb300.batched import BatchedMeshes, _to_device
    rng = np.random.default_rng(72)
    om = _mesh(rng, 256, "clements")
    bm = BatchedMeshes([gpu_mesh(om)], [40])
    x = O.unit_columns(rng, 256, 40)
    bm.states[0].x.copy_(torch.tensor(x, dtype=torch.complex64))
    bm.states[0].y.zero_()
    items = (_lib.mg_batch_item * 4)()
    for it, (mesh, v0, vend) in zip(items, ((0, 0, 32), (0, 32, 64), (1, 0, 32), (0, -32, 0))):
        it.mesh, it.v0, it.vend, it.part = mesh, v0, vend, 0
    dev = _to_device(items, bm.device)
    bm.head.zero_()
    _lib.check(_lib.load().mg_batched_framed(_lib.OP_FWD, bm.fdesc[0].data_ptr(), 1, dev.data_ptr(), 4, bm.head.data_ptr(),
                                             bm.grid, bm.fsmem[0], bm.status.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream), "mg_batched_framed")
    assert bm.check_status() == 3
    y = bm.states[0].y.cpu().numpy()
    assert O.rel_err(y[:32], O.propagate(om, x)[:32]) < TOL
    assert float(np.abs(y[32:]).max()) == 0.0


@pytest.mark.parametrize("op", [0, 2])
def test_tiles_of_four_modes_per_lane_are_refused(op):
    """mg_batched_framed runs 8 modes per lane; a mesh of 65 to 128 modes, whose framed tiles have 4, is not its item."""
    import ctypes
    from meshes_gb300 import _lib
    from meshes_gb300.batched import _to_device
    from meshes_gb300.serve import MeshServer
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    om = _mesh(np.random.default_rng(73), 128, "clements", 24)
    cfg, ws = MeshServer([gpu_mesh(om)]).res[0].framed
    ds, smem = [_lib.mg_batch_framed(), _lib.mg_batch_framed()], [ctypes.c_size_t(), ctypes.c_size_t()]
    _lib.check(lib.mg_batched_framed_desc(128, om.L, 1, 0, 0, _lib.cfg_ptr(cfg), ws.data_ptr(), ws.numel(),
                                          *map(ctypes.byref, ds), *map(ctypes.byref, smem)), "mg_batched_framed_desc")
    u, g, out = (torch.zeros((32, 128), dtype=torch.complex64, device="cuda") for _ in range(3))
    u += 1
    dp = torch.zeros(om.p.shape, device="cuda")
    partial = torch.zeros((om.L, 128, 2), device="cuda")     # of 8 modes per lane
    d = ds[0 if op == 0 else 1]
    d.mesh.B, d.mesh.ldu, d.mesh.n_items, d.mesh.ldp, d.mesh.n_p = 32, 128, 1, 128, 2
    d.mesh.in0, d.mesh.in1 = u.data_ptr(), g.data_ptr()
    d.mesh.out0, d.mesh.out1 = (out.data_ptr(), None) if op == 0 else (None, out.data_ptr())
    d.mesh.dp, d.mesh.partial = dp.data_ptr(), partial.data_ptr()
    dev, item = _to_device((_lib.mg_batch_framed * 1)(d), u.device), _to_device((_lib.mg_batch_item * 1)((0, 0, 32, 0)), u.device)
    head, status = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    _lib.check(lib.mg_batched_framed(op, dev.data_ptr(), 1, item.data_ptr(), 1, head.data_ptr(), 1, 200000, status.data_ptr(),
                                     st), "mg_batched_framed")
    assert int(status) == 3
    assert not out.any() and not partial.any()
