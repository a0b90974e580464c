"""Measured cases of the mesh-propagation path: what a user's program calls, over the sizes that the package takes.

Each case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more of the same ranges;
``prepare`` makes the inputs and the objects a program keeps, ``run`` is one pass through the public entry points, and
``exact`` evaluates the same pass in 64 bits with plain tensor operations.

Common to all kinds: fields are iid complex Gaussian columns of unit norm, phases are uniform on [0, 2 pi) or those
of a mesh programmed to a Haar-random unitary ("programmed": sin^2(theta/2) ~ Beta(1, k), k the place along the
mesh's diagonal), splitting errors are N(0, 0.02).
"""
import math

import numpy as np
import torch

from meshes_gb300 import MeshNetworkGPU, geometry
from meshes_gb300.autograd import GraphedStep, mesh_apply, mesh_l2_loss
from meshes_gb300.batched import BatchedMeshes
from meshes_gb300.lossy import LossyMesh
from meshes_gb300.serve import MeshServer

SIGMA = 0.02
LARGEST = 7e10          # FLOP: about the largest listed case's; a drawn one stays below


def listed():
    return [
        # the smallest call: one programmed 10-mode mesh, a handful of vectors; launch latency is what a user sees
        dict(name="dot_N10_B7", kind="dot", N=10, B=7, geo="clements", X="mzi", split=True, programmed=False),
        # plain inference on a 64-mode chip with ideal splitters and a batch of 1024
        dict(name="dot_N64_B1024", kind="dot", N=64, B=1024, geo="clements", X="mzi", split=False, programmed=False),
        # inference with an imperfect 256-mode mesh and a full batch
        dict(name="dot_N256_B4096", kind="dot", N=256, B=4096, geo="clements", X="mzi", split=True, programmed=False),
        # forward-mode derivative (sensitivity along one phase direction), ragged sizes
        dict(name="diff_N130_B1000", kind="diff", N=130, B=1000, geo="clements", X="mzi", split=True, programmed=False),
        # the reference-style gradient call on a triangle programmed to a unitary, ragged sizes
        dict(name="grad_reck_N100_B777", kind="grad", N=100, B=777, geo="reck", X="mzi", split=True, programmed=True),
        # the training step of an imperfect mesh: loss to a target and its phase gradient
        dict(name="train_N256_B4096", kind="train", N=256, B=4096, geo="clements", X="mzi", split=True,
             programmed=False),
        # unitary fitting: identity batch, Haar target, the gradient step replayed as a CUDA graph
        dict(name="fit_N128", kind="fit", N=128, B=128, geo="clements", X="mzi", split=True, programmed=False),
        # the widest meshes, as a layer of a larger model: output, input gradient and phase gradient
        dict(name="layer_N600_B2048", kind="layer", N=600, B=2048, geo="clements", X="mzi", split=True,
             programmed=False),
        # a shallow FFT mesh over a large batch, as a layer: memory traffic counts more than arithmetic
        dict(name="layer_fft_N256_B20000", kind="layer", N=256, B=20000, geo="fft", X="mzi", split=True,
             programmed=False),
        # many independent meshes of uneven size in one persistent launch, forward and backward, graph replay, and
        # the results gathered into one tensor per kind
        dict(name="batched_96", kind="batched", count=96, Nmax=256, Bmax=2048),
        # a burst of mixed requests (1 in 5 with a gradient) on resident meshes, from host arrays to host arrays
        dict(name="serve_40", kind="serve", count=40, meshes=12, Nmax=256, Bmax=512),
        # a lossy mesh with its checkpointed adjoint: T from the phases, forward, backward to the phases
        dict(name="lossy_N128_B1024", kind="lossy", N=128, B=1024, geo="clements"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dot", "dot", "diff", "grad", "train", "fit", "layer", "layer", "batched", "serve", "lossy"])
    if kind == "batched":
        case = dict(kind=kind, count=_logint(rng, 16, 96), Nmax=rng.choice([64, 128, 256]), Bmax=_logint(rng, 256, 2048))
        while work(case)["flops"] > LARGEST:
            case["Bmax"] //= 2
        return case
    if kind == "serve":
        return dict(kind=kind, count=_logint(rng, 16, 44), meshes=rng.randint(4, 16), Nmax=rng.choice([64, 128, 256]),
                    Bmax=_logint(rng, 64, 512))
    if kind == "lossy":
        return dict(kind=kind, N=2 * _logint(rng, 8, 80), B=_logint(rng, 32, 1024), geo="clements")
    if kind == "fit":
        N = 2 * _logint(rng, 8, 128)
        return dict(kind=kind, N=N, B=N, geo="clements", X="mzi", split=rng.random() < 0.7, programmed=False)
    geo = rng.choice(["clements", "clements", "reck", "fft"])
    X = rng.choice(["mzi", "mzi", "mzi", "sym", "orth"])
    if geo == "fft":
        N, B = 2 ** rng.randint(4, 9), _logint(rng, 64, 20000)
    else:
        N, B = 2 * _logint(rng, 4, 300 if geo == "clements" else 150), _logint(rng, 1, 6000)
    case = dict(kind=kind, N=N, B=B, geo=geo, X=X, split=X != "orth" and rng.random() < 0.7,
                programmed=geo != "fft" and X == "mzi" and rng.random() < 0.4)
    while work(case)["flops"] > LARGEST:
        case["B"] = max(1, case["B"] // 2)
    return case


# ---------------------------------------------------------------------------------------------- inputs
def _geometry(geo, N):
    """(lens, shifts, strides) of one mesh; the unused ones None."""
    if geo == "fft":
        return None, None, geometry.fft(N)
    lens, shifts = geometry.clements(N) if geo == "clements" else geometry.reck(N)
    return lens, shifts, None


def _active(geo, N):
    lens, shifts, strides = _geometry(geo, N)
    return np.ones((len(strides), N // 2), bool) if strides is not None else geometry.active_mask_nn(N, lens, shifts)


def _params(rng, geo, N, X, split, programmed):
    """Phase grid (L, N/2, n_p) and splitter grid (L, N/2, n_s) or None, float32, zero on inactive slots."""
    mask = _active(geo, N)
    n_p, n_s = {"mzi": (2, 2), "sym": (2, 1), "orth": (1, 0)}[X]
    p = rng.uniform(0, 2 * np.pi, mask.shape + (n_p,))
    if programmed:
        k = rng.integers(1, N, mask.shape)
        p[..., 0] = 2 * np.arcsin(np.sqrt(rng.beta(1.0, k)))
    p = (p * mask[..., None]).astype(np.float32)
    s = (rng.normal(0, SIGMA, mask.shape + (n_s,)) * mask[..., None]).astype(np.float32) if split and n_s else None
    return p, s


def _fields(rng, B, N, real=False):
    """(B, N) rows of unit norm."""
    x = rng.standard_normal((B, N), dtype=np.float32)
    if not real:
        x = x + 1j * rng.standard_normal((B, N), dtype=np.float32)
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _haar(rng, N):
    q, r = np.linalg.qr(rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))
    return (q * (np.diagonal(r) / np.abs(np.diagonal(r)))).astype(np.complex64)


def _lossy_errors(rng, shape):
    """(alpha, beta, eight phase errors, four log-gains of about -0.02) per slot."""
    s = rng.normal(0, SIGMA, shape + (14,))
    s[..., 10:] = -np.abs(s[..., 10:])
    return s


def _composition(case, rng):
    """(geometry, crossing, N, B) of every mesh of a batched or served case."""
    sizes = [n for n in (8, 16, 32, 64, 128, 256) if n <= case["Nmax"]]
    out = []
    for i in range(case["count"] if case["kind"] == "batched" else case["meshes"]):
        N = int(rng.choice(sizes))
        if case["kind"] == "batched":
            geo, X = (("clements", "mzi"), ("reck", "mzi"), ("clements", "orth"))[i % 3]
            out.append((geo, X, N, int(rng.integers(1, case["Bmax"] + 1))))
        else:
            out.append(("fft" if i % 4 == 3 else "clements", "mzi", N, 0))
    return out


def _requests(case, rng):
    """(mesh, vectors, gradient wanted) of every request of a served case."""
    return [(int(rng.integers(case["meshes"])), max(1, int(round(case["Bmax"] ** rng.random()))), i % 5 == 4)
            for i in range(case["count"])]


def _inputs(case, seed):
    """Everything a case is made from, as numpy arrays."""
    # the composition of a batched or served case belongs to the case, its values to the seed
    shape_rng, rng = np.random.default_rng(case.get("count", 0)), np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("batched", "serve"):
        comp = _composition(case, shape_rng)
        meshes = [(geo, X, N, B) + _params(rng, geo, N, X, True, False) for geo, X, N, B in comp]
        if kind == "batched":
            return dict(meshes=meshes, x=[_fields(rng, B, N, X == "orth") for _, X, N, B in comp],
                        g=[_fields(rng, B, N, X == "orth") for _, X, N, B in comp])
        req = _requests(case, shape_rng)
        return dict(meshes=meshes, req=req, x=[_fields(rng, b, comp[m][2]) for m, b, _ in req],
                    g=[_fields(rng, b, comp[m][2]) if grad else None for m, b, grad in req])
    N, B = case["N"], case["B"]
    if kind == "lossy":
        mask = _active(case["geo"], N)
        p = rng.uniform(0, 2 * np.pi, mask.shape + (2,)) * mask[..., None]
        return dict(p=p, s=_lossy_errors(rng, mask.shape) * mask[..., None], x=_fields(rng, B, N), g=_fields(rng, B, N))
    p, s = _params(rng, case["geo"], N, case["X"], case["split"], case["programmed"])
    d = dict(p=p, s=s)
    if kind == "fit":
        d.update(x=np.eye(N, dtype=np.complex64), g=_haar(rng, N).T.copy())
    else:
        real = case["X"] == "orth"
        d.update(x=_fields(rng, B, N, real), g=_fields(rng, B, N, real))
    if kind == "diff":
        d["dp"] = (rng.standard_normal(p.shape) * _active(case["geo"], N)[..., None]).astype(np.float32)
    return d


# ---------------------------------------------------------------------------------------------- the measured passes
def _mesh(geo, X, N, p, s):
    lens, shifts, strides = _geometry(geo, N)
    return MeshNetworkGPU(N, p.shape[0], lens, shifts, p.reshape(-1), s, X, is_phase=False, strides=strides)


class _Serving:
    """A running server, stopped with the state that holds it."""

    def __init__(self, meshes):
        self.server = MeshServer(meshes, mem_budget=96 << 20)
        self.server.start()

    def __del__(self):
        self.server.stop(drain=False, timeout=5.0)


def _by_type(y, gx, dp):
    """The results of a batched pass in one list per quantity and type of field."""
    out = dict(dp=list(dp))
    for key, ts in (("y", y), ("gx", gx)):
        for t in ts:
            out.setdefault(key + ("_c" if "complex" in str(t.dtype) else "_r"), []).append(t)
    return out


def prepare(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    dev = (lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda())
    if kind == "batched":
        bm = BatchedMeshes([_mesh(geo, X, N, p, s) for geo, X, N, _, p, s in d["meshes"]],
                           [m[3] for m in d["meshes"]])
        bm.capture(backward=True)
        for buf, val in zip(bm.x + bm.gy, d["x"] + d["g"]):
            buf.copy_(dev(val))
        return dict(kind=kind, bm=bm, results=_by_type(bm.y, bm.gx, bm.dp))
    if kind == "serve":
        meshes = [_mesh(geo, X, N, p, s) for geo, X, N, _, p, s in d["meshes"]]
        return dict(kind=kind, serving=_Serving(meshes), req=d["req"], x=d["x"], g=d["g"])
    if kind == "lossy":
        lens, shifts, _ = _geometry(case["geo"], case["N"])
        return dict(kind=kind, mesh=LossyMesh(case["N"], lens, shifts), p=dev(d["p"]).requires_grad_(True),
                    s=dev(d["s"]), x=dev(d["x"]), g=dev(d["g"]))
    st = dict(kind=kind, mesh=_mesh(case["geo"], case["X"], case["N"], d["p"], d["s"]), x=dev(d["x"]), g=dev(d["g"]))
    if kind == "diff":
        st["dp"] = dev(d["dp"]).reshape(-1)
    if kind in ("train", "fit", "layer"):
        st["p"] = dev(d["p"]).requires_grad_(True)
    if kind == "layer":
        st["x"].requires_grad_(True)
    if kind == "fit":
        def step(mesh=st["mesh"], x=st["x"], t=st["g"], p=st["p"]):
            p.grad = None
            loss = mesh_l2_loss(mesh, x, t, p)
            loss.backward()
            return loss.detach()
        st["step"] = GraphedStep(step)
    return st


def run(state):
    kind = state["kind"]
    if kind == "batched":
        bm = state["bm"]
        bm.replay()
        return {key: torch.cat([t.reshape(-1) for t in ts]) for key, ts in state["results"].items()}
    if kind == "serve":
        server = state["serving"].server
        futures = [server.submit(m, x, g) for (m, _, _), x, g in zip(state["req"], state["x"], state["g"])]
        results = [f.result() for f in futures]
        return [list(r) if isinstance(r, tuple) else [r] for r in results]
    if kind == "fit":
        loss = state["step"]()
        return [loss, state["p"].grad]
    mesh = state["mesh"]
    if kind == "lossy":
        p = state["p"]
        p.grad = None
        y = mesh(state["x"], mesh.T(p, state["s"]))
        y.backward(state["g"])
        return [y.detach(), p.grad]
    if kind == "dot":
        return mesh.dot(state["x"].t())
    if kind == "diff":
        return list(mesh.dot(state["x"].t(), dp=state["dp"]))
    if kind == "grad":
        t = state["g"].t()
        return list(mesh.grad_phi(state["x"].t(), lambda y: 2 * (y - t)))
    p = state["p"]
    p.grad = None
    if kind == "train":
        loss = mesh_l2_loss(mesh, state["x"], state["g"], p)
        loss.backward()
        return [loss.detach(), p.grad]
    x = state["x"]
    x.grad = None
    y = mesh_apply(mesh, x, p)
    y.backward(state["g"])
    return [y.detach(), x.grad, p.grad]


# ---------------------------------------------------------------------------------------------- what a pass needs
def _mesh_work(geo, N, B, X, n_fields, flop):
    """Fields read and written once, phases and splitters read once, at the path's FLOP per MZI and vector."""
    mask = _active(geo, N)
    el, per, scale = (4, 1, 0.25) if X == "orth" else (8, 4 if X == "mzi" else 3, 1.0)
    return n_fields * B * N * el + 4 * per * int(mask.sum()), flop * scale * int(mask.sum()) * B


def work(case):
    """FLOP per MZI and vector: 32 forward, 96 forward-mode derivative, 96 back-propagation (a quarter for real)."""
    kind = case["kind"]
    if kind in ("batched", "serve"):
        rng = np.random.default_rng(case["count"])
        comp = _composition(case, rng)
        if kind == "batched":
            parts = [_mesh_work(geo, N, B, X, 4, 128) for geo, X, N, B in comp]
        else:
            parts = [_mesh_work(comp[m][0], comp[m][2], b, "mzi", 4 if g else 2, 128 if g else 32)
                     for m, b, g in _requests(case, rng)]
    elif kind == "lossy":
        parts = [_mesh_work(case["geo"], case["N"], case["B"], "mzi", 3, 128)]
    else:
        n_fields, flop = {"dot": (2, 32), "diff": (3, 96), "grad": (4, 128), "train": (2, 128), "fit": (2, 128),
                          "layer": (4, 128)}[kind]
        parts = [_mesh_work(case["geo"], case["N"], case["B"], case["X"], n_fields, flop)]
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _T64(X, p, s):
    """Transfer matrices (..., 2, 2) of the crossing in 64 bits, differentiable in p."""
    th = p[..., 0]
    C, S = torch.cos(th / 2), torch.sin(th / 2)
    if X == "orth":
        return torch.stack([torch.stack([S, -C], -1), torch.stack([C, S], -1)], -2)
    ph = p[..., 1]
    cis = (lambda a: torch.complex(torch.cos(a), torch.sin(a)))
    if X == "sym":
        a = torch.zeros_like(th) if s is None else s[..., 0]
        c2, s2 = torch.cos(2 * a), torch.sin(2 * a)
        off = torch.complex(torch.zeros_like(C), C * c2)
        return torch.stack([torch.stack([cis(ph) * torch.complex(S, C * s2), off], -1),
                            torch.stack([off, cis(-ph) * torch.complex(S, -C * s2)], -1)], -2)
    a, b = (torch.zeros_like(th), torch.zeros_like(th)) if s is None else (s[..., 0], s[..., 1])
    Cp, Cm, Sp, Sm = torch.cos(a + b), torch.cos(a - b), torch.sin(a + b), torch.sin(a - b)
    e0, e1 = cis(th / 2), cis(th / 2 + ph)
    return torch.stack([torch.stack([e1 * torch.complex(-C * Sp, S * Cm), e0 * torch.complex(-S * Sm, C * Cp)], -1),
                        torch.stack([e1 * torch.complex(S * Sm, C * Cp), e0 * torch.complex(-C * Sp, -S * Cm)], -1)],
                       -2)


def _T64_lossy(p, s):
    """S(beta) D2 S(alpha) D1 with phase errors and gains, differentiable in p."""
    def ep(phase, gain):
        return torch.exp(torch.complex(gain / 2, phase))

    def split(a):
        c, i_s = torch.cos(math.pi / 4 + a) + 0j, 1j * torch.sin(math.pi / 4 + a)
        return torch.stack([torch.stack([c, i_s], -1), torch.stack([i_s, c], -1)], -2)

    def diag(a, b):
        return torch.diag_embed(torch.stack([a, b], -1))

    d1 = diag(ep(p[..., 1] + s[..., 2] + s[..., 6], s[..., 10]), ep(s[..., 3] + s[..., 7], s[..., 11]))
    d2 = diag(ep(p[..., 0] + s[..., 4] + s[..., 8], s[..., 12]), ep(s[..., 5] + s[..., 9], s[..., 13]))
    return split(s[..., 1]) @ d2 @ split(s[..., 0]) @ d1


def _pairs(geo, N):
    """Per layer: the active slots and the two modes of each (index tensors on the GPU)."""
    lens, shifts, strides = _geometry(geo, N)
    out = []
    for l in range(len(strides if strides is not None else lens)):
        if strides is not None:
            q, w = np.arange(N // 2), 1 << strides[l]
            a = 2 * w * (q // w) + q % w
            b = a + w
        else:
            q = shifts[l] // 2 + np.arange(lens[l])
            a = shifts[l] + 2 * np.arange(lens[l])
            b = a + 1
        out.append(tuple(torch.as_tensor(v, device="cuda") for v in (q, a, b)))
    return out


def _pass64(pairs, T, x, g=None, dT=None):
    """y = U x for modes-major x (N, B); with dT also dy; with g (array or function of y) also (U^H g, dJ/dT)."""
    x = x.clone()
    dx = torch.zeros_like(x) if dT is not None else None
    inputs = []
    for l, (q, a, b) in enumerate(pairs):
        t = T[l, q][:, :, :, None]
        xa, xb = x[a], x[b]
        if g is not None:
            inputs.append((xa, xb))
        if dx is not None:
            d, da, db = dT[l, q][:, :, :, None], dx[a], dx[b]
            dx[a] = t[:, 0, 0] * da + t[:, 0, 1] * db + d[:, 0, 0] * xa + d[:, 0, 1] * xb
            dx[b] = t[:, 1, 0] * da + t[:, 1, 1] * db + d[:, 1, 0] * xa + d[:, 1, 1] * xb
        x[a], x[b] = t[:, 0, 0] * xa + t[:, 0, 1] * xb, t[:, 1, 0] * xa + t[:, 1, 1] * xb
    if dx is not None:
        return x, dx
    if g is None:
        return x
    g = g(x) if callable(g) else g.clone()
    gT = torch.zeros_like(T)
    for l in range(len(pairs) - 1, -1, -1):
        q, a, b = pairs[l]
        t, (xa, xb), ga, gb = T[l, q][:, :, :, None].conj(), inputs.pop(), g[a], g[b]
        gT[l, q] = torch.stack([torch.stack([(u * v.conj()).sum(1) for v in (xa, xb)], -1) for u in (ga, gb)], -2)
        g[a], g[b] = t[:, 0, 0] * ga + t[:, 1, 0] * gb, t[:, 0, 1] * ga + t[:, 1, 1] * gb
    return x, g, gT


def _wide(a):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _grad64(geo, N, T_of, p, x, g, chunk=512):
    """(y (B, N), U^H g (B, N), dJ/dp) with the batch taken in pieces; g (B, N) or a function (rows, y) of it."""
    p = _wide(p).requires_grad_(True)
    T, pairs = T_of(p), _pairs(geo, N)
    ys, gs, gT = [], [], torch.zeros_like(T.detach())
    for i in range(0, x.shape[0], chunk):
        rows = slice(i, i + chunk)
        y, gi, gt = _pass64(pairs, T.detach(), _wide(x[rows]).t(),
                            (lambda y, rows=rows: g(rows, y)) if callable(g) else _wide(g[rows]).t())
        ys.append(y.t())
        gs.append(gi.t())
        gT += gt
    T.backward(gT)
    return torch.cat(ys), torch.cat(gs), p.grad


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    host = (lambda t: t.detach().cpu().numpy())

    def crossing(X, s):
        s64 = None if s is None else _wide(s)
        return lambda p: _T64(X, p, s64)

    if kind == "batched":
        per_mesh = [[host(v) for v in _grad64(geo, N, crossing(X, s), p, x, g)]
                    for (geo, X, N, _, p, s), x, g in zip(d["meshes"], d["x"], d["g"])]
        return {key: np.concatenate([t.reshape(-1) for t in ts]) for key, ts in _by_type(*zip(*per_mesh)).items()}
    if kind == "serve":
        out, meshes = [], [(geo, N, p, crossing(X, s)) for geo, X, N, _, p, s in d["meshes"]]
        for (m, _, grad), x, g in zip(d["req"], d["x"], d["g"]):
            geo, N, p, T_of = meshes[m]
            if grad:
                y, gx, dp = _grad64(geo, N, T_of, p, x, g)
                out.append([host(y), host(dp), host(gx)])
            else:
                out.append([host(_pass64(_pairs(geo, N), T_of(_wide(p)), _wide(x).t()).t())])
        return out
    geo, N, p, x, g = case["geo"], case["N"], d["p"], d["x"], d["g"]
    if kind == "lossy":
        s = _wide(d["s"])
        y, _, dp = _grad64(geo, N, lambda q: _T64_lossy(q, s), p, x, g)
        return [host(y), host(dp)]
    T_of = crossing(case["X"], d["s"])
    if kind == "dot":
        return host(_pass64(_pairs(geo, N), T_of(_wide(p)), _wide(x).t()))
    if kind == "diff":
        p64, dp64 = _wide(p), _wide(d["dp"])
        _, dT = torch.autograd.functional.jvp(T_of, p64, dp64)
        return [host(v) for v in _pass64(_pairs(geo, N), T_of(p64), _wide(x).t(), dT=dT)]
    if kind == "layer":
        return [host(v) for v in _grad64(geo, N, T_of, p, x, g)]
    losses = []

    def residual(rows, y):
        r = y - _wide(g[rows]).t()
        losses.append(float((r.abs() ** 2).sum()))
        return 2 * r

    y, gx, dp = _grad64(geo, N, T_of, p, x, residual)
    if kind == "grad":
        return [host(dp).reshape(-1), host(gx.t())]
    return [np.float64(sum(losses)), host(dp)]
