"""The per-head products of latent attention over few rows against float64 and against the form for many rows: row counts up to a tile,
sizes that do not fill the tiles, both gates, both rotation layouts, outputs in both dtypes."""
import pytest
import torch

from citlali_b200 import ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("rows", [1, 7, 8, 16])
@pytest.mark.parametrize("H, K, N, tail, rot_dims, halves, gate, out", [
    (3, 128, 512, 64, 64, False, None, torch.float32), (16, 512, 128, 0, 0, False, "elements", torch.bfloat16),
    (5, 16, 40, 6, 4, True, None, torch.float32), (2, 80, 24, 9, 8, False, "heads", torch.bfloat16), (1, 1040, 7, 0, 0, True, "heads", torch.float32)])
def test_heads_product_of_few_rows(rows, H, K, N, tail, rot_dims, halves, gate, out):
    g = torch.Generator().manual_seed(rows * K + N)
    many = 70                                                   # the same rows among others take the other kernel
    x = torch.randn(many, H, K + tail + (tail & 1), generator=g).to(torch.bfloat16).float()      # exact in both kernels' operands
    M = (torch.randn(H, N, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    z = torch.randn(many, H * N if gate == "elements" else H, generator=g)
    pos = torch.randint(0, 3000, (many,), generator=g).to(torch.int32)
    freq = 1e4 ** (-torch.arange(rot_dims // 2).double() / max(rot_dims // 2, 1))
    got = {}
    for n in (rows, many):
        y = torch.full((n, H, N + tail), float("nan"), dtype=out, device=DEV)
        ops.heads_product(x[:n].contiguous().to(DEV), x.stride(0), x.stride(1), M.to(DEV), N * K, 1, K, y, H * (N + tail), N + tail, n, H, K, N,
                          tail=tail, inv_freq=freq.float().to(DEV), rot_dims=rot_dims, row_pos=pos[:n].to(DEV),
                          gate=None if gate is None else z[:n].contiguous().to(DEV), gate_stride=z.shape[1], rot_halves=halves,
                          gate_per_head=gate == "heads")
        got[n] = y[:rows].double().cpu()
    want = torch.einsum("rhk,hnk->rhn", x[:rows, :, :K].double(), M.double())
    if gate is not None:
        want = want * torch.sigmoid(z[:rows].double().view(rows, H, -1))
    scale = float(want.abs().max())
    tol = 2e-6 * K ** 0.5 if out == torch.float32 else 2 ** -8            # sums of K products in float32; one rounding
    assert float((got[rows][..., :N] - want).abs().max()) <= tol * scale
    assert float((got[rows] - got[many]).abs().max()) <= tol * scale and torch.equal(got[rows][..., N:], got[many][..., N:])
