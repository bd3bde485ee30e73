"""The tensor-core product with a bias and an activation in its epilogue against float64, in every form of the product: few rows (the
weights on the wide side, with and without a split of K), one block a tile, pairs of SMs, sizes at and around the tiles' edges."""
import pytest
import torch

import citlali_b200 as cb
from citlali_b200 import ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("M, N, K", [(1, 64, 128), (5, 200, 520), (16, 4096, 1024), (33, 160, 64), (100, 608, 256), (129, 416, 72),
                                     (250, 2080, 320), (300, 24, 136), (513, 3104, 256), (2000, 4128, 128)])
@pytest.mark.parametrize("biased", [False, True])
def test_epilogues_against_float64(M, N, K, biased):
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    bias = torch.randn(N, generator=g) if biased else None
    v = x.double() @ w.double().T + (bias.double() if biased else 0.0)
    dev = lambda t: None if t is None else t.to(DEV)
    flag = torch.zeros(4, dtype=torch.int32, device=DEV)
    run = lambda y, **kw: ops.gemm_tc_act(dev(x), dev(w), y, bias=dev(bias), error_flag=flag, **kw)
    bf16 = lambda y, ref: float((y.double().cpu() - ref).abs().max()) <= 2 ** -8 * float(ref.abs().max())     # one rounding, and sums of 1e-6

    squared = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    run(squared, act="relu_squared")
    assert bf16(squared, v.clamp(min=0.0) ** 2)
    stored = torch.full((M, N), float("nan"), device=DEV)
    run(stored)
    assert float((stored.cpu().double() - v).abs().max()) <= 2e-5 * float(v.abs().max())
    base = torch.randn(M, N, generator=g)
    added = base.to(DEV)
    run(added, accumulate=True)
    assert float((added.cpu().double() - base.double() - v).abs().max()) <= 2e-5 * float(v.abs().max())
    if N % 32 == 0:
        gate, up = v.view(M, N // 32, 2, 16).unbind(2)
        gated = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
        run(gated, act="gelu_gate")
        assert bf16(gated, (torch.nn.functional.gelu(gate, approximate="tanh") * up).reshape(M, N // 2))
    assert not any(flag.tolist())


def test_epilogues_refuse_what_is_none():
    x, w = torch.zeros(4, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(48, 64, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(cb.CitlaliError):
        ops.gemm_tc_act(x, w, torch.zeros(4, 24, dtype=torch.bfloat16, device=DEV), act="gelu_gate")        # 48 is no multiple of 32
    with pytest.raises(cb.CitlaliError):
        ops.gemm_tc_act(x, w, torch.zeros(4, 48, device=DEV), act="relu_squared")                          # a float32 result
    with pytest.raises(cb.CitlaliError):
        ops.gemm_tc_act(x, w, torch.zeros(4, 48, device=DEV), bias=torch.zeros(49, device=DEV)[1:])         # off a 16-byte boundary
