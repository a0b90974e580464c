"""Framed launches over the magnitudes of float32: a vector that comes in times a power of two leaves times that power, bit for
bit, and so do the gradients, however far the frames take the fields from their own size (cross states most of all).  There is
nothing to tolerate: such factors are exact as long as inputs and results are normal numbers."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O
from test_framed import SIZES, _backward, _forward, _mesh

pytestmark = pytest.mark.gpu
TILES = [(4, 4, 1, 16), (8, 4, 1, 8), (8, 3, 0, 8), (16, 2, 0, 8), (20, 1, 0, 4)]
KINDS = ["clements", "cross", "few_cross"]


def _cfg(t):
    return (t[0], t[1], t[3], 0, 0, 6 if t[2] else 5)


def _fields(rng, N, B):
    return O.unit_columns(rng, N, B).astype(np.complex64)


def _times(a, k):
    return (a * np.exp2(np.float64(k))[:, None]).astype(np.complex64)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("tile", TILES)
def test_forward(tile, kind):
    rng = np.random.default_rng(tile[0] + len(kind))
    N, B = SIZES[tile[0]][0], 45
    om = _mesh(rng, N, kind)
    x = _fields(rng, N, B)
    y = _forward(om, x, _cfg(tile))
    assert O.rel_err(y, O.propagate(om, x)) < 1e-5
    for k in (np.full(B, -100), np.full(B, 118), rng.integers(-100, 118, B)):
        assert np.array_equal(_forward(om, _times(x, k), _cfg(tile)), _times(y, k))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("tile", TILES)
def test_backward(tile, kind):
    """Fields times 2^k, gradients times 2^(c - k): dJ/dp times 2^c."""
    rng = np.random.default_rng(tile[0] + len(kind) + 50)
    N, B = SIZES[tile[0]][0], 45
    om = _mesh(rng, N, kind)
    y, g = _fields(rng, N, B), _fields(rng, N, B)
    x0, gx0, dp0 = _backward(om, y, g, _cfg(tile))
    assert O.rel_err(dp0, O.contract_dp(om, O.vjp_unitary(om, y, g)[0])) < 1e-5
    small = np.abs(dp0) < 2.0 ** -26                     # (their multiples may not be normal numbers)
    for c, k in ((-90, np.full(B, -45)), (-90, np.full(B, 5)), (-90, rng.integers(-100, 10, B)), (100, np.full(B, 110)),
                 (100, np.full(B, -10)), (0, rng.integers(-95, 95, B))):
        x, gx, dp = _backward(om, _times(y, k), _times(g, c - k), _cfg(tile))
        assert np.array_equal(x, _times(x0, k)) and np.array_equal(gx, _times(gx0, c - k)), c
        want = (dp0 * np.exp2(float(c))).astype(np.float32)
        assert np.array_equal(dp[~small], want[~small]), c
        assert np.all(np.abs(dp[small]) <= 2.0 ** (c - 26))


@pytest.mark.parametrize("spread", [4, 20, 120])
@pytest.mark.parametrize("tile", TILES)
def test_products_of_any_size_in_a_batch(tile, spread):
    """Warps and CTAs whose products need different scales add up (the library's 1e-5 relative Frobenius error)."""
    rng = np.random.default_rng(tile[0] + spread)
    N, B = SIZES[tile[0]][0], 301
    om = _mesh(rng, N, "few_cross", 20)
    y, g = _fields(rng, N, B), _fields(rng, N, B)
    y, g = _times(y, rng.integers(-spread // 2, spread // 2, B)), _times(g, rng.integers(-spread // 2, spread // 2, B))
    x, gx, dp = _backward(om, y, g, _cfg(tile))
    G, xin, gin = O.vjp_unitary(om, y, g)
    size = lambda a: np.linalg.norm(a, axis=1)
    assert np.all(size(x - xin) < 1e-5 * size(xin)) and np.all(size(gx - gin) < 1e-5 * size(gin))
    assert O.rel_err(dp, O.contract_dp(om, G)) < 1e-5


def test_vectors_without_a_scale():
    """Zero vectors and gradients, and ones with NaN or infinity, leave their neighbours' results what they were."""
    rng = np.random.default_rng(3)
    om = _mesh(rng, 130, "few_cross")
    cfg = (8, 4, 8, 0, 0, 6)
    y, g = _fields(rng, 130, 28), _fields(rng, 130, 28)
    x0, gx0, dp0 = _backward(om, y, g, cfg)
    k = np.where(np.arange(28) == 5, 60, -60)            # one vector beside which the others are nothing
    k[[2, 3]] = 0
    y1, g1 = _times(y, k), _times(g, 0 * k)
    y1[2], g1[3] = 0, 0
    x, gx, dp = _backward(om, y1, g1, cfg)
    keep = np.arange(28) != 3
    assert np.array_equal(gx[keep], gx0[keep]) and not gx[3].any() and not x[2].any()
    keep = np.arange(28) != 2
    assert np.array_equal(x[keep], _times(x0, k)[keep])
    _, _, only = _backward(om, np.where(np.arange(28)[:, None] == 5, y1, 0), g1, cfg)
    assert O.rel_err(dp, only) < 1e-6
    y1, g1 = y.copy(), g.copy()
    y1[7, 3], g1[8, 100] = np.nan, np.inf
    x, gx, _ = _backward(om, y1, g1, cfg)
    keep = (np.arange(28) != 7) & (np.arange(28) != 8)
    assert np.array_equal(x[keep], x0[keep]) and np.array_equal(gx[keep], gx0[keep])
    assert np.array_equal(x[8], x0[8]) and np.array_equal(gx[7], gx0[7])


def test_batched_and_served():
    """The persistent launches keep their items' scales as well: gradients 2^-100 of their size."""
    from meshes_gb300.batched import BatchedMeshes
    from meshes_gb300.serve import MeshServer
    from test_batched import gpu_mesh
    rng = np.random.default_rng(4)
    oms = [_mesh(rng, 130, "cross", 40), _mesh(rng, 256, "few_cross", 40)]
    xs, gs = [_fields(rng, om.N, 70) for om in oms], [_fields(rng, om.N, 70) for om in oms]
    k = np.full(70, -100)
    bm = BatchedMeshes([gpu_mesh(om) for om in oms], [70, 70])
    assert bm.n_framed == 2
    srv = MeshServer([gpu_mesh(om) for om in oms], mem_budget=256 << 20)
    srv.start()
    got = []
    try:
        for size in (0 * k, k):
            for st, x, g in zip(bm.states, xs, gs):
                st.x.copy_(torch.tensor(x))
                st.gy.copy_(torch.tensor(_times(g, size)))
            bm.forward()
            bm.backward()
            assert bm.check_status() == 0
            got.append([(st.dp.cpu().numpy(), st.gx.cpu().numpy()) for st in bm.states])
            fs = [srv.submit(i, x, _times(g, size)) for i, (x, g) in enumerate(zip(xs, gs))]
            got[-1] += [f.result(timeout=60)[1:] for f in fs]
    finally:
        srv.stop()
    for (dp0, gx0), (dp, gx) in zip(*got):
        small = np.abs(dp0) < 2.0 ** -20
        assert np.array_equal(gx, _times(gx0, k)) and np.array_equal(dp[~small], (dp0 * np.float32(2.0 ** -100))[~small])
        assert not small.all() and np.all(np.abs(dp[small]) <= 2.0 ** -120)
