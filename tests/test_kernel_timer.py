"""What the timer of single kernels does to the functions it stands in front of, on the CPU."""
import torch

from citlali_b200 import ops
from citlali_b200.measure import KernelTimer


def test_layers_are_timed_kernel_by_kernel(monkeypatch):
    """One call for a layer's six kernels would give one time for all of them: while the timer is on, no layer comes from one call."""
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    before = dict(vars(ops))
    with KernelTimer():
        assert ops.dense_layer_supports(8, 2, 128, 64, 23) is False and ops.gemm_tc is not before["gemm_tc"]
    assert all(vars(ops)[name] is value for name, value in before.items())
