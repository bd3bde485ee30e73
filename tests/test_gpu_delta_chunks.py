"""The gated delta rule 32 tokens at a time against the recurrence in float64, and no further off than the walk: lengths around a chunk,
sequences side by side, states carried over, key and value sizes that do not fill the tiles, decays of nothing and of everything."""
import math

import pytest
import torch

from citlali_b200 import ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def recurrence(prep, lengths, H, KH, D, V, S):
    """Float64; ``S`` [sequences, H, D, V] is left as the state."""
    C, out, at = 2 * KH * D + H * V, [], 0
    p = prep.double()
    for s, n in enumerate(lengths):
        for t in range(at, at + n):
            q = p[t, :KH * D].view(KH, D).repeat_interleave(H // KH, 0)
            k = p[t, KH * D:2 * KH * D].view(KH, D).repeat_interleave(H // KH, 0)
            v, beta, g = p[t, 2 * KH * D:C].view(H, V), p[t, C:C + H, None], p[t, C + H:, None]
            S[s] *= g[..., None]
            u = beta * (v - torch.einsum("hdv,hd->hv", S[s], k))
            S[s] += k[..., None] * u[:, None]
            out.append(torch.einsum("hdv,hd->hv", S[s], q).flatten())
        at += n
    return torch.stack(out)


@pytest.mark.parametrize("D, V, H, KH, lengths, decays", [
    (128, 128, 4, 2, [200, 1, 64], "mixed"), (128, 128, 2, 2, [31, 32, 33, 65], "slow"), (64, 40, 6, 2, [96, 7], "none"),
    (20, 4, 2, 1, [70], "fast"), (128, 128, 32, 16, [100], "mixed"), (96, 36, 8, 8, [40, 129, 32, 5, 1], "mixed")])
def test_chunks_against_float64_and_the_walk(D, V, H, KH, lengths, decays):
    T, C = sum(lengths), 2 * KH * D + H * V
    g = torch.Generator().manual_seed(D + T)
    prep = torch.zeros(T, C + 2 * H)
    unit = torch.nn.functional.normalize(torch.randn(T, 2 * KH, D, generator=g) + 0.3, dim=-1)      # keys that lean one way
    prep[:, :2 * KH * D] = unit.view(T, -1)
    prep[:, :KH * D] *= D ** -0.5
    prep[:, 2 * KH * D:C] = torch.randn(T, H * V, generator=g)
    prep[:, C:C + H] = torch.rand(T, H, generator=g)
    r = torch.rand(T, H, generator=g)
    prep[:, C + H:] = {"mixed": torch.where(r < 0.05, torch.zeros(()), r ** 0.1), "slow": 1 - 1e-3 * r, "none": torch.ones(T, H),
                       "fast": 1e-6 * r}[decays]
    bounds = [0]
    for n in lengths:
        bounds.append(bounds[-1] + n)
    seq_start = torch.tensor(bounds, dtype=torch.int32, device=DEV)
    slots = list(range(len(lengths)))[::-1]
    seq_slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
    extra = 24                                                 # a state region holds more than S
    start = torch.randn(len(lengths), H * D * V + extra, generator=g)
    want_state = torch.stack([start[s, :H * D * V].view(H, D, V) for s in slots]).double()
    want = [recurrence(prep, lengths, H, KH, D, V, want_state), recurrence(prep, lengths, H, KH, D, V, want_state)]
    off = {}
    for name in ("chunks", "walk"):
        state, got = start.to(DEV), []
        for _ in range(2):                                     # the same rows once more, from the states just left
            out = torch.full((T, H * V), float("nan"), device=DEV)
            if name == "chunks":
                ops.delta_chunks(prep.to(DEV), state, seq_start, seq_slot, len(lengths), max(lengths), H, KH, D, V, out)
            else:
                ops.delta_rule(prep.to(DEV), state, seq_start, seq_slot, len(lengths), H, KH, D, V, out, pairs=True)
            got.append(out.cpu())
        assert torch.equal(state[:, H * D * V:].cpu(), start[:, H * D * V:])
        left = torch.stack([state[s, :H * D * V].view(H, D, V) for s in slots]).cpu().double()
        off[name] = [float((a.double() - b).norm() / b.norm()) for a, b in [(got[0], want[0]), (got[1], want[1]), (left, want_state)]]
    # 32-bit sums: a few 2^-24 each, along chains of a chunk's 32 tokens instead of the walk's pairs
    for a, b in zip(off["chunks"], off["walk"]):
        assert a <= 2e-6 and a <= 2.0 * b + 1e-7, off


@pytest.mark.parametrize("D, V, H, KH, lengths, decays", [
    (128, 128, 16, 8, [33, 5, 70, 150, 64], "mixed"), (96, 36, 16, 8, [40, 129, 32, 5, 1], "mixed"), (20, 40, 16, 16, [31, 64, 1, 200], "slow"),
    (64, 4, 2, 1, [1, 2, 33, 3, 7, 64] * 50, "mixed")], ids=["five", "columns left over", "small", "300"])
def test_blocks_of_32_columns_and_many_sequences(D, V, H, KH, lengths, decays):
    """Above: blocks of 16 columns mostly.  Several sequences, the longest first, and so many that they are not sorted."""
    assert len(lengths) * H * ((V + 31) // 32) >= torch.cuda.get_device_properties(0).multi_processor_count * 3 // 4
    test_chunks_against_float64_and_the_walk(D, V, H, KH, lengths, decays)


@pytest.mark.parametrize("kind", ["random", "leaning", "repeated", "silu", "fast"])
def test_chunks_are_as_near_float64_as_the_walk(kind):
    """Means over four seeds of 640 rows; the sums' orders differ, so the two distances do by some tenths."""
    H, KH, D, V, T = 4, 2, 128, 128, 640
    C, off = 2 * KH * D + H * V, {"chunks": 0.0, "walk": 0.0}
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    for seed in range(4):
        g = torch.Generator().manual_seed(seed)
        keys, beta, decay = torch.randn(T, KH, D, generator=g), torch.rand(T, H, generator=g), torch.rand(T, H, generator=g)
        if kind == "repeated":
            keys, beta = keys[:1].expand(T, -1, -1), torch.ones(T, H)
        keys = {"leaning": keys + 0.3, "silu": torch.nn.functional.silu(keys)}.get(kind, keys)
        decay = {"random": decay ** 0.1, "silu": 1 - 1e-3 * decay, "fast": 0.1 * decay}.get(kind, torch.ones(T, H))
        prep = torch.zeros(T, C + 2 * H)
        prep[:, :KH * D] = torch.nn.functional.normalize(torch.randn(T, KH, D, generator=g), dim=-1).view(T, -1) * D ** -0.5
        prep[:, KH * D:2 * KH * D] = torch.nn.functional.normalize(keys, dim=-1).reshape(T, -1)
        prep[:, 2 * KH * D:C] = torch.randn(T, H * V, generator=g)
        prep[:, C:C + H], prep[:, C + H:] = beta, decay
        want = recurrence(prep, [T], H, KH, D, V, torch.zeros(1, H, D, V, dtype=torch.float64))
        for name in off:
            state, out = torch.zeros(1, H * D * V, device=DEV), torch.empty(T, H * V, device=DEV)
            if name == "chunks":
                ops.delta_chunks(prep.to(DEV), state, i32([0, T]), i32([0]), 1, T, H, KH, D, V, out)
            else:
                ops.delta_rule(prep.to(DEV), state, i32([0, T]), i32([0]), 1, H, KH, D, V, out, pairs=True)
            off[name] += float((out.cpu().double() - want).norm() / want.norm()) / 4
    print(f"[{kind}] chunks {off['chunks']:.2e}, walk {off['walk']:.2e} off float64")
    assert off["chunks"] <= 1.3 * off["walk"], off


@pytest.mark.parametrize("heads", [4, 64])                    # columns of the values a block: 16, 32
@pytest.mark.parametrize("part", ["query", "key", "value", "strength", "decay"])
@pytest.mark.parametrize("bad", [math.nan, math.inf])
def test_a_token_that_is_not_finite_reaches_no_earlier_one(heads, part, bad):
    """Not even times zero: the rows before it keep their bits, whatever their places in its chunk."""
    D = V = 128
    H, KH, T, C = heads, heads // 2, 75, heads * 2 * D
    assert (2 * H * 4 >= torch.cuda.get_device_properties(0).multi_processor_count * 3 // 4) == (heads == 64)
    g = torch.Generator().manual_seed(heads)
    prep = torch.zeros(T, C + 2 * H)
    prep[:, :2 * KH * D] = torch.nn.functional.normalize(torch.randn(T, 2 * KH, D, generator=g), dim=-1).view(T, -1)
    prep[:, 2 * KH * D:C] = torch.randn(T, H * V, generator=g)
    prep[:, C:] = 0.5 + 0.5 * torch.rand(T, 2 * H, generator=g)
    span = {"query": (0, KH * D), "key": (KH * D, 2 * KH * D), "value": (2 * KH * D, C), "strength": (C, C + H), "decay": (C + H, C + 2 * H)}[part]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)

    def run(rows):
        out = torch.full((2 * T, H * V), float("nan"), device=DEV)
        ops.delta_chunks(torch.cat([rows, prep]).to(DEV), torch.zeros(2, H * D * V, device=DEV), i32([0, T, 2 * T]), i32([1, 0]), 2, T, H, KH, D, V, out)
        return out[:T].cpu(), out[T:].cpu()

    clean, beside = run(prep)
    for at in (0, 1, 2, 3, 6, 17, 30, 31, 32, 45, 63, 64, 74):
        rows = prep.clone()
        rows[at, span[0]:span[1]] = bad
        got, other = run(rows)
        assert torch.equal(got[:at], clean[:at]) and torch.equal(other, beside), (at, int(torch.isfinite(got).all(1).long().argmin()))
        assert not torch.isfinite(got[at]).all()
