"""Kernels that take several rows, heads or streams at once against plain float64, and against the forms they stand beside."""
import math

import pytest
import torch

from citlali_b200 import ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("nq, nkv, d, window, dtype", [
    (8, 2, 128, 0, torch.float32), (8, 1, 64, 33, torch.float32), (6, 3, 20, 0, torch.float32), (3, 1, 256, 70, torch.float32),
    (4, 1, 7, 0, torch.float32), (5, 5, 200, 0, torch.bfloat16), (8, 2, 40, 5, torch.bfloat16)])
def test_attention_rows_of_a_group_have_the_bits_of_single_heads(nq, nkv, d, window, dtype):
    """Room for more keys than there are picks the form that takes one head at a time."""
    g = torch.Generator().manual_seed(nq * d)
    lengths, page = [1, 2, 130, 301], 16
    pages = [(n + page - 1) // page for n in lengths]
    order = torch.randperm(sum(pages), generator=g).tolist()
    table = torch.zeros(len(lengths), max(pages), dtype=torch.int32)
    for b, n in enumerate(pages):
        table[b, :n] = torch.tensor([order.pop() for _ in range(n)], dtype=torch.int32)
    k, v = (torch.randn(sum(pages), nkv, page, d, generator=g).to(dtype).to(DEV) for _ in range(2))
    slot = torch.cat([torch.full((n,), b) for b, n in enumerate(lengths)]).to(torch.int32).to(DEV)
    pos = torch.cat([torch.arange(n) for n in lengths]).to(torch.int32).to(DEV)
    q = (3.0 * torch.randn(sum(lengths), nq * d + 5, generator=g)).to(dtype).to(DEV)
    outs = []
    for max_keys in (301, 40000):
        out = torch.full((sum(lengths), nq * d), float("nan"), dtype=dtype, device=DEV)
        ops.attention_rows(q, q.shape[1], k, v, table.to(DEV), slot, pos, out, nq, nkv, d, page, window, max_keys, d ** -0.5)
        outs.append(out.cpu())
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1])
    at = 0
    for b, n in enumerate(lengths):
        rows = lambda t: torch.cat([t[table[b, i]] for i in range(pages[b])], 1)[:, :n].double().cpu()      # [nkv, n, d]
        kk, vv = (rows(t).repeat_interleave(nq // nkv, 0) for t in (k, v))
        qq = q[at:at + n, :nq * d].double().cpu().view(n, nq, d).transpose(0, 1)
        far = torch.arange(n)[:, None] - torch.arange(n)[None, :]
        s = (qq @ kk.transpose(1, 2) * d ** -0.5).masked_fill((far < 0) | (far >= (window or n)), -math.inf)
        want = (torch.softmax(s, -1) @ vv).transpose(0, 1).reshape(n, nq * d)
        assert float((outs[0][at:at + n].double() - want).abs().max()) <= (2e-5 if dtype == torch.float32 else 1e-2) * float(want.abs().max())
        at += n
