"""What the host refuses, or plans otherwise, before anything is launched; runs without a GPU."""
import ctypes

import pytest
import torch


def _plan(op, N, L, B, crossing=0, geo=0, cfg=None):
    from meshes_gb300 import _lib
    i = _lib.mg_plan_info()
    c = None if cfg is None else _lib.cfg_ptr(_lib.config(*cfg))
    return i if _lib.load().mg_plan(op, N, L, B, crossing, geo, c, ctypes.byref(i)) == 0 else None


def test_l2_target_on_another_device_is_refused():
    from meshes_gb300.autograd import MeshL2Function
    x = torch.zeros(3, 8, dtype=torch.complex64)
    with pytest.raises(RuntimeError, match="target is on meta"):
        MeshL2Function.apply(x, torch.zeros(8, 4, 2), torch.zeros(3, 8, dtype=torch.complex64, device="meta"), None)


@pytest.mark.parametrize("op", [0, 2])
def test_framed_warps_come_in_fours(op):
    for M, V, N in ((4, 1, 100), (8, 4, 256), (16, 1, 400), (20, 2, 600)):
        for W in range(1, 9):
            assert (_plan(op, N, 64, 300, cfg=(M, V, W, 0, 0, 5)) is not None) == (W % 4 == 0), (M, W)


def test_tuned_framed_entry_at_other_depths():
    """A recorded framed launch holds for depths that may be framed and gain by it; the others keep the launch they had."""
    from meshes_gb300 import _lib
    lib = _lib.load()
    shapes = [(op, L) for op in (0, 2) for L in (0, 1, 8, 300, 4096, 4097, 5000)]
    before = [_plan(op, 300, L, 50) for op, L in shapes]
    try:
        for op in (0, 2):
            _lib.check(lib.mg_set_tuned(op, 0, 0, 300, 1, 100, ctypes.byref(_lib.config(16, 2, 4, 0, 0, 5))), "mg_set_tuned")
        after = [_plan(op, 300, L, 50) for op, L in shapes]
    finally:
        for op in (0, 2):
            lib.mg_set_tuned(op, 0, 0, 300, 0, 0, None)
    for (op, L), a, b in zip(shapes, before, after):
        assert b is not None, (op, L)
        if L in (300, 4096):
            assert (b.V, b.W) == (2, 4)
        else:
            assert all(getattr(a, f) == getattr(b, f) for f, _ in a._fields_), (op, L)
