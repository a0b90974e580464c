"""Checkpoint spacings of the lossy adjoint, against the complex128 oracle.  Tolerance: the library's 1e-5 relative Frobenius
error."""
import numpy as np
import pytest
import torch

from oracle import meshes_oracle as O

TOL = 1e-5


def _case(N, L, B):
    rng = np.random.default_rng(N + L)
    lens, shifts = O.clements_geometry(N)
    lens, shifts = lens[:L], shifts[:L]
    om = O.OracleMesh(N=N, L=L, crossing="mzi", lens=list(lens), shifts=list(shifts),
                      p=rng.uniform(0, 2 * np.pi, (L, N // 2, 2)).astype(np.float32))
    om.p[~om.active_mask()] = 0
    T = np.ascontiguousarray(om.T_grid(), dtype=np.complex64)
    T[om.active_mask()] *= np.float32(0.95)              # 5% loss per crossing
    om.T_override = T
    return om, T, O.unit_columns(rng, N, B), O.unit_columns(rng, N, B)


def _check(om, T, x, g, mesh):
    xd = torch.tensor(x, dtype=torch.complex64, device="cuda", requires_grad=True)
    Td = torch.tensor(T, device="cuda", requires_grad=True)
    y = mesh(xd, Td)
    assert O.rel_err(y.detach().cpu().numpy(), O.propagate(om, x)) < TOL
    y.backward(torch.tensor(g, dtype=torch.complex64, device="cuda"))
    G, gin = O.vjp_stored(om, x, g)
    assert O.rel_err(xd.grad.cpu().numpy(), gin) < TOL and O.rel_err(Td.grad.cpu().numpy(), np.conj(G)) < TOL
    assert mesh.status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("N,L,segment", [(258, 17, 16), (512, 18, 16), (512, 19, 9), (256, 36, 32), (128, 70, 64), (64, 60, 48)])
def test_shallow_meshes_with_long_segments(N, L, segment):
    """Meshes whose tiles all fit one pipeline stage, cut by checkpoints: two stages of a segment each need not fit."""
    from meshes_gb300.lossy import LossyMesh
    om, T, x, g = _case(N, L, 5)
    _check(om, T, x, g, LossyMesh(N, om.lens, om.shifts, segment=segment))


@pytest.mark.gpu
@pytest.mark.parametrize("B,segment", [(5, None), (300, 24)])
def test_without_memory_for_the_stored_inputs(B, segment, monkeypatch):
    """Back-propagation then runs by the shortest spacing; a spacing that the caller fixed stays (and the error with it)."""
    from meshes_gb300 import lossy
    om, T, x, g = _case(64, 40, B)
    mesh = lossy.LossyMesh(64, om.lens, om.shifts, segment=segment)
    stored, asked = lossy._stored_inputs, []

    def scarce(layers, *args):
        asked.append(layers)
        if layers > 7:
            raise torch.OutOfMemoryError("scarce")
        return stored(layers, *args)
    monkeypatch.setattr(lossy, "_stored_inputs", scarce)
    if segment:
        with pytest.raises(torch.OutOfMemoryError):
            _check(om, T, x, g, mesh)
        assert asked == [24]
    else:
        _check(om, T, x, g, mesh)
        assert asked == [40, 7] and mesh.segment == 7 and mesh.segment_for(B) == 40
