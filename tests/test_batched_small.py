"""Batched launches with vectors per lane group by mesh (mg_batched_small) against the complex128 oracle: every class of mesh
in one launch, on framed and on plain tiles, batches at the edges of an item; a vector's result does not depend on the
shape; and the server's requests of every size.  Tolerance: the library's 1e-5 relative Frobenius error."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O
from test_batched import gpu_mesh
from test_framed import _mesh

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _desc(mesh, st):
    """({op: mg_batch_framed}, smem, lanes, keep-alive) of a mesh: framed where the server would, else the plain tiles of st."""
    from meshes_gb300 import _lib
    from meshes_gb300.serve import MeshServer
    framed = MeshServer([mesh]).res[0].framed
    ds, smem = [_lib.mg_batch_framed(), _lib.mg_batch_framed()], [ctypes.c_size_t(), ctypes.c_size_t()]
    if framed is None:
        for d, op in zip(ds, (0, 2)):
            d.mesh = st.descriptor(op)
        return dict(zip((0, 2), ds)), max(st.info[0].smem, st.info[2].smem), st.G, None
    cfg, ws = framed
    _lib.check(_lib.load().mg_batched_framed_desc(mesh.N, mesh.L, 1, mesh.crossing, mesh.geometry, _lib.cfg_ptr(cfg),
                                                  ws.data_ptr(), ws.numel(), *map(ctypes.byref, ds),
                                                  *map(ctypes.byref, smem)), "mg_batched_framed_desc")
    return dict(zip((0, 2), ds)), max(v.value for v in smem), 32, ws


# vectors per lane group: (framed fwd, framed bwd, plain fwd; None: the class's own, as always in back-propagation)
@pytest.mark.parametrize("shape", [(1, 1, 1), (4, 4, None), (1, 2, 1)])
def test_every_class(shape):
    from meshes_gb300 import _lib
    from meshes_gb300.batched import BatchedMeshes, _to_device
    rng = np.random.default_rng(81)
    oms = [_mesh(rng, 256, "clements"), _mesh(rng, 100, "reck"), _mesh(rng, 130, "irregular"), _mesh(rng, 128, "flat"),
           O.random_mesh(rng, 64, "clements", "mzi", 0.01), O.random_mesh(rng, 8, "reck", "mzi", 0.01),
           O.random_mesh(rng, 256, "fft", "mzi", 0.01), O.random_mesh(rng, 300, "clements", "mzi", 0.01),
           O.random_mesh(rng, 200, "clements", "orth", 0.0)]
    meshes = [gpu_mesh(om) for om in oms]
    Bs = [65, 32, 3, 1, 33, 5, 17, 15, 9]
    bm = BatchedMeshes(meshes, Bs, full_warp=False)
    descs = [_desc(m, st) for m, st in zip(meshes, bm.states)]
    assert [d[3] is not None for d in descs] == [True] * 4 + [False] * 5
    lib, stream, items, keep = _lib.load(), torch.cuda.current_stream().cuda_stream, {0: [], 2: []}, []
    for i, ((ds, _, G, framed), om, st) in enumerate(zip(descs, oms, bm.states)):
        for op, d in ds.items():
            d.V = (shape[0] if op == 0 else shape[1]) if framed is not None else (op == 0 and shape[2]) or st.V
            cap = 8 * (32 // G) * d.V
            n = -(-st.B // cap)
            items[op] += [(i, k * cap, min((k + 1) * cap, st.B), k) for k in range(n)]
            d.mesh.B, d.mesh.ldu, d.mesh.n_items = st.B, om.N, n
            d.mesh.ldp, d.mesh.n_p = om.N // 2 * meshes[i].X_np, meshes[i].X_np
            st._fields(op, d.mesh)
            if op == 2:
                keep.append(torch.empty(n * om.L * 256 * 2, dtype=torch.float32, device="cuda"))
                d.mesh.partial = keep[-1].data_ptr()
    smem = max(d[1] for d in descs)
    xs = [O.unit_columns(rng, om.N, B, real=om.crossing == "orth") for om, B in zip(oms, Bs)]
    gs = [O.unit_columns(rng, om.N, B, real=om.crossing == "orth") for om, B in zip(oms, Bs)]
    for st, x, g in zip(bm.states, xs, gs):
        st.x.copy_(torch.tensor(x, dtype=st.x.dtype))
        st.gy.copy_(torch.tensor(g, dtype=st.gy.dtype))
    for op in (0, 2):
        dev = _to_device((_lib.mg_batch_framed * len(oms))(*[d[0][op] for d in descs]), bm.device)
        its = _to_device((_lib.mg_batch_item * len(items[op]))(*[_lib.mg_batch_item(*t) for t in items[op]]), bm.device)
        keep += [dev, its]
        bm.head.zero_()
        _lib.check(lib.mg_batched_small(op, dev.data_ptr(), len(oms), its.data_ptr(), len(items[op]), bm.head.data_ptr(), 5,
                                        smem, bm.status.data_ptr(), stream), "mg_batched_small")
    _lib.check(lib.mg_batched_framed_reduce(dev.data_ptr(), len(oms), stream), "mg_batched_framed_reduce")
    assert bm.check_status() == 0
    for om, st, x, g in zip(oms, bm.states, xs, gs):
        y_ref = O.propagate(om, x)
        G, _, gin = O.vjp_unitary(om, y_ref, g)
        assert O.rel_err(st.y.cpu().numpy(), y_ref) < TOL, om.N
        assert O.rel_err(st.gx.cpu().numpy(), gin) < TOL, om.N
        assert O.rel_err(st.dp.cpu().numpy(), O.contract_dp(om, G)) < TOL, om.N


def test_a_request_is_the_same_in_every_tick():
    """A forward request's item shape goes by the load of its tick; its result must not.  Each class's vectors through items
    of 1 vector per lane group and of the class's own, alone and in a tick that fills the SMs several times."""
    from meshes_gb300.serve import MeshServer
    rng = np.random.default_rng(82)
    oms = [_mesh(rng, 256, "clements", 24), _mesh(rng, 128, "reck", 24), O.random_mesh(rng, 64, "fft", "mzi", 0.01),
           _mesh(rng, 64, "clements"), O.random_mesh(rng, 300, "clements", "mzi", 0.01),
           O.random_mesh(rng, 200, "clements", "orth", 0.0)]
    real = [om.crossing == "orth" for om in oms]
    dt = [np.float32 if r else np.complex64 for r in real]
    srv = MeshServer([gpu_mesh(om) for om in oms], mem_budget=256 << 20, n_streams=1)
    probes = [(i, O.unit_columns(rng, oms[i].N, b, real=real[i]).astype(dt[i])) for i in range(len(oms)) for b in (1, 13, 70)]
    load = [(i % 2, O.unit_columns(rng, oms[i % 2].N, 900).astype(np.complex64)) for i in range(8)]
    srv.start()
    try:
        alone = [srv.submit(i, x, x).result(timeout=60) for i, x in probes]
        for _ in range(3):
            fs = [srv.submit(i, x) for i, x in load[:4]] + [srv.submit(i, x, x) for i, x in probes]
            fs += [srv.submit(i, x) for i, x in load[4:]]
            mixed = [f.result(timeout=60) for f in fs[4:4 + len(probes)]]
            [f.result(timeout=60) for f in fs]
            for (i, _), a, m in zip(probes, alone, mixed):
                assert all(np.array_equal(u, v) for u, v in zip(a, m)), oms[i].N
    finally:
        srv.stop()


# vectors of a request: framed items of 1, 2 and 4 vectors per lane group, 256 and 128 modes; the plain ones of 128 beyond 32
@pytest.mark.parametrize("b", [1, 8, 9, 16, 17, 32, 33, 65, 600, 2600])
def test_server_shapes(b):
    from meshes_gb300.serve import MeshServer
    rng = np.random.default_rng(83)
    oms = [_mesh(rng, 256, "clements", 24), _mesh(rng, 128, "reck", 24), _mesh(rng, 200, "flat"),
           O.random_mesh(rng, 64, "fft", "mzi", 0.01)]
    srv = MeshServer([gpu_mesh(om) for om in oms], mem_budget=256 << 20)
    req = [(O.unit_columns(rng, om.N, b).astype(np.complex64), O.unit_columns(rng, om.N, b).astype(np.complex64)) for om in oms]
    srv.start()
    try:
        fs = [srv.submit(i, x, g) for i, (x, g) in enumerate(req)]
        for om, (x, g), f in zip(oms, req, fs):
            y, dp, gx = f.result(timeout=60)
            y_ref = O.propagate(om, x)
            G, _, gin = O.vjp_unitary(om, y_ref, g)
            assert O.rel_err(y, y_ref) < TOL
            assert O.rel_err(gx, gin) < TOL
            assert O.rel_err(dp, O.contract_dp(om, G)) < TOL
    finally:
        srv.stop()
