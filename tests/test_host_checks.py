"""What the host refuses, or plans otherwise, before anything is launched; runs without a GPU."""
import pytest
import torch


def test_l2_target_on_another_device_is_refused():
    from meshes_gb300.autograd import MeshL2Function
    x = torch.zeros(3, 8, dtype=torch.complex64)
    with pytest.raises(RuntimeError, match="target is on meta"):
        MeshL2Function.apply(x, torch.zeros(8, 4, 2), torch.zeros(3, 8, dtype=torch.complex64, device="meta"), None)
