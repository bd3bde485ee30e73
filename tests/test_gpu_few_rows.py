"""The per-head products of latent attention over few rows against float64 and against the form for many rows: row counts up to a tile,
sizes that do not fill the tiles, both gates, both rotation layouts, outputs in both dtypes."""
import pytest
import torch

import citlali_b200 as cb
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


@pytest.mark.parametrize("D, V, H, KH, mode", [(128, 128, 4, 2, 0), (40, 36, 6, 2, 0), (20, 8, 2, 1, 1), (128, 100, 3, 3, 1), (200, 64, 2, 2, 0)])
@pytest.mark.parametrize("taps", [1, 2, 4])
def test_delta_step_against_the_kernels_it_stands_for(D, V, H, KH, mode, taps):
    """One token a sequence, several steps: the kept inputs, the state and the output of the two launches against those of the four."""
    B, GD, C = 5, D if mode else 1, 2 * KH * D + H * V
    g = torch.Generator().manual_seed(D * V + taps)
    dev = lambda *shape: torch.randn(*shape, generator=g).to(DEV)
    taps_w, a_log, bias, weight = dev(C, taps), 0.3 * dev(H), dev(H * GD), dev(V)
    i32 = lambda v: torch.as_tensor(v, dtype=torch.int32, device=DEV)
    slots, starts = i32([6, 1, 0, 3, 5]), i32(list(range(B + 1)))
    first = 0.5 * dev(8, H * D * V + (taps - 1) * C)
    states = [first.clone(), first.clone()]
    for step in range(3):
        proj, decay = dev(B, C + H * V + 2 * H), dev(B, H * GD) if mode else None
        gate = proj[:, C:]
        outs = []
        for kind, state in enumerate(states):
            prep = torch.empty(B, C + H + H * GD, device=DEV)
            ops.delta_prepare(proj, taps_w, state, H * D * V, slots, starts, slots, B, a_log, bias, prep, H, KH, D, V, 1e-6,
                              block_a_segment=True, one_row_each=kind == 1, decay_in=decay, channel_decay=bool(mode))
            y = torch.full((B, H * V), float("nan"), device=DEV)
            if kind == 0:
                o = torch.empty(B, H * V, device=DEV)
                ops.delta_rule(prep, state, starts, slots, B, H, KH, D, V, o, mode=mode)
                ops.delta_output(o, gate, proj.shape[1], weight, y, H, V, 1e-5)
            else:
                ops.delta_step(prep, state, starts, slots, B, H, KH, D, V, gate, proj.shape[1], weight, y, 1e-5, mode=mode)
            outs.append((prep.cpu(), y.cpu(), state.cpu()))
        assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][2][:, H * D * V:], outs[1][2][:, H * D * V:])
        for a, b in zip(outs[0][1:], outs[1][1:]):         # the same sums in the same order, up to what the compiler fuses
            assert float((a - b).abs().max()) <= 2e-6 * float(a.abs().max())
    with pytest.raises(Exception, match="one each"):
        ops.delta_prepare(proj, taps_w, states[0], H * D * V, slots, i32([0, 2, 2, 3, 4]), slots, B - 1, a_log, bias, prep, H, KH, D, V, 1e-6,
                          block_a_segment=True, one_row_each=True, decay_in=decay, channel_decay=bool(mode))


@pytest.mark.parametrize("d, heads, kv", [(128, 4, 2), (64, 6, 3), (80, 4, 4)])
@pytest.mark.parametrize("lengths", [(2,), (47,), (48,), (128,), (5, 1, 60, 3), (1, 31, 32, 33, 31)])
def test_a_layer_from_one_call_gives_the_bits_of_its_launches_one_by_one(d, heads, kv, lengths, monkeypatch):
    """Few new rows of one or several sequences, at their start and behind cached tokens, either side of the tcgen05 attention's 48 rows."""
    from citlali_b200.engine.step import StepEntry
    from citlali_b200.parts.block import PreNormResidualBlock
    config = cb.config_from_dict(dict(
        architectures=["Qwen3ForCausalLM"], num_hidden_layers=3, hidden_size=256, num_attention_heads=heads, num_key_value_heads=kv,
        head_dim=d, intermediate_size=352, vocab_size=500, rope_theta=1e4, rms_norm_eps=1e-6, tie_word_embeddings=True,
        max_position_embeddings=512))
    session = cb.InferenceSession().load_random(config, seed=3, max_context=400, dtype="bfloat16", device=DEV, max_batch=len(lengths),
                                                gain_spread=0.1)
    calls = []
    whole = ops.dense_layer
    monkeypatch.setattr(ops, "dense_layer", lambda *a: (calls.append(1), whole(*a)))

    def steps():
        g = torch.Generator().manual_seed(7)
        slots = [session.acquire() for _ in lengths]
        out = []
        for _ in range(2):
            tokens = [torch.randint(0, 500, (n,), generator=g).tolist() for n in lengths]
            out.append(session.step([StepEntry(s, t, list(range(len(t)))) for s, t in zip(slots, tokens)]))
        for s in slots:
            session.release(s)
        return out

    got = steps()
    assert len(calls) == 6
    monkeypatch.setattr(PreNormResidualBlock, "_from_one_call", lambda *a: False)
    want = steps()
    session.check_device_errors()
    assert len(calls) == 6 and all(torch.equal(a, b) for a, b in zip(got, want))
