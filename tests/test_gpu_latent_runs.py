"""Latent attention of runs of new tokens with the heads' keys and values written out, against float64 and against the walk over the
latents that the same mixer takes otherwise: lengths around the tiles of 128 keys and 256 query rows, several sequences a step,
steps behind cached tokens, windows, sinks, both gates and both rotation layouts, narrow rotated parts, odd head counts."""
import math

import pytest
import torch

from citlali_b200 import ops
from citlali_b200.cache import SequenceCache
from citlali_b200.parts import part_class
from test_gpu_lanizen_parts import DEV, ctx_for, handles, run_steps, weights_for

pytestmark = pytest.mark.gpu
HIDDEN = 64


def mixer_for(heads=3, rot_dim=64, kv_rank=512, window=None, rot_dims=None, layout="pairs", gate="elements", sink=True):
    params = dict(heads=heads, dim=128, rot_dim=rot_dim, vdim=128, q_rank=48, kv_rank=kv_rank, scale=0.1, window=window,
                  rot_dims=rot_dim if rot_dims is None else rot_dims, rot_base=1e4, rot_layout=layout, gate=gate, hidden_size=HIDDEN,
                  norm_eps=1e-5)
    if not sink:
        params["names"] = {"sink": None}
    return part_class("mixer", "latent_attention")(params, "m"), params


def exact(h, w, p):
    """The mixer in float64."""
    w = {k: v.double() for k, v in w.items()}
    h = h.double()
    T, H, P, R = h.shape[0], p["heads"], p["rot_dim"], p["kv_rank"]
    rms = lambda x, g: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * g
    half = p["rot_dims"] // 2
    angle = torch.arange(T).double()[:, None] * (1e4 ** (-torch.arange(half).double() / max(half, 1)))
    a, b = (slice(0, half), slice(half, 2 * half)) if p["rot_layout"] == "halves" else (slice(0, 2 * half, 2), slice(1, 2 * half, 2))

    def turn(x):                                   # [T, heads, P]
        out = x.clone()
        c, s = angle.cos()[:, None], angle.sin()[:, None]
        out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
        return out

    q = (rms(h @ w["m.dq"].T, w["m.dq_norm"]) @ w["m.uq"].T).view(T, H, 128 + P)
    q = torch.cat([q[..., :128], turn(q[..., 128:])], -1)
    down = h @ w["m.dkv"].T
    c = rms(down[:, :R], w["m.dkv_norm"])
    k = torch.cat([(c @ w["m.uk"].T).view(T, H, 128), turn(down[:, None, R:]).expand(-1, H, -1)], -1)
    s = torch.einsum("ihd,jhd->hij", q, k) * p["scale"]
    far = torch.arange(T)[:, None] - torch.arange(T)[None, :]
    s = s.masked_fill((far < 0) | (far >= (p["window"] or T + 1)), -math.inf)
    if "m.sink" in w:
        s = torch.cat([s, w["m.sink"][:, None, None].expand(-1, T, 1)], -1)
    o = torch.einsum("hij,jhd->ihd", torch.softmax(s, -1)[..., :T], (c @ w["m.uv"].T).view(T, H, 128))
    g = torch.sigmoid(h @ w["m.gate"].T)
    o = o * (g[..., None] if p["gate"] == "heads" else g.view(T, H, 128))
    return o.flatten(1) @ w["m.o"].T


CASES = [dict(), dict(window=100, heads=2), dict(window=300, layout="halves"), dict(gate="heads", sink=False, layout="halves", kv_rank=64),
         dict(rot_dim=16, rot_dims=8, window=64), dict(rot_dim=40, rot_dims=24, layout="halves", heads=1, window=128),
         dict(rot_dim=8, rot_dims=0, gate="heads", kv_rank=72)]


@pytest.mark.parametrize("case", CASES, ids=str)
def test_runs_against_float64_and_the_walk(case, monkeypatch):
    mixer, p = mixer_for(**case)
    w = weights_for(mixer, 5, {"_norm": lambda r: 1 + 0.3 * r, "sink": lambda r: 2 * r})
    mixer.bind(handles(w, torch.bfloat16), ctx_for(torch.bfloat16))
    x = torch.randn(700, HIDDEN, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).float()
    want = exact(x, w, p)
    ran = []
    plain_call = ops.latent_run_attention
    monkeypatch.setattr(ops, "latent_run_attention", lambda *a, **k: (ran.append(a[0].shape[0]), plain_call(*a, **k)))

    def steps(walk):
        kept, mixer.kv_up = mixer.kv_up, None if walk else mixer.kv_up
        cache = SequenceCache([mixer.cache_requirement()], 6, 8192, 1024, torch.bfloat16, DEV)
        s = [cache.acquire() for _ in range(6)]
        cut = lambda slot, lo, hi: (slot, x[lo:hi])
        got = run_steps(mixer, cache, HIDDEN, [
            [cut(s[0], 0, 700)],                                                          # a long run alone
            [cut(s[1], 0, 127), cut(s[2], 0, 128), cut(s[3], 0, 129), cut(s[4], 0, 32)],  # around the tiles, and the shortest
            [cut(s[1], 127, 383), cut(s[2], 128, 257), cut(s[3], 129, 699)],              # behind cached tokens
            [cut(s[5], 0, 64)], [cut(s[5], 64, 200)], [cut(s[5], 200, 520)]], torch.bfloat16)
        mixer.kv_up = kept
        return got

    runs = steps(False)
    assert ran == [700, 416, 955, 64, 136, 320]
    walk = steps(True)
    assert len(ran) == 6
    for slot, rows in runs.items():
        ref = want[:rows.shape[0]]
        off = lambda y: float((y.double().cpu() - ref).norm() / ref.norm())
        # bfloat16 operands and results: 2^-9 a rounding, a handful of them; and no further off than the walk, whose rounding of
        # queries and weighted latents takes the place of that of keys and values
        assert off(rows) <= 2e-2 and off(rows) <= 1.15 * off(walk[slot]) + 2e-4, (slot, off(rows), off(walk[slot]))
        one = (rows.double().cpu() - ref).norm(dim=1) / ref.norm(dim=1).median()
        assert float(one.max()) <= 6e-2, (slot, int(one.argmax()), float(one.max()))


def test_a_sequence_beside_one_of_infinities():
    """Nothing of another sequence's keys or values reaches a row, not even times zero."""
    mixer, _ = mixer_for(heads=2)
    w = weights_for(mixer, 6, {"_norm": lambda r: 1 + 0.3 * r, "sink": lambda r: r})
    mixer.bind(handles(w, torch.bfloat16), ctx_for(torch.bfloat16))
    x = torch.randn(330, HIDDEN, generator=torch.Generator().manual_seed(4)).to(torch.bfloat16).float()
    bad = x.clone()
    bad[5] = math.inf
    out = []
    for other in (x, bad):
        cache = SequenceCache([mixer.cache_requirement()], 3, 2048, 512, torch.bfloat16, DEV)
        a, b, c = cache.acquire(), cache.acquire(), cache.acquire()
        out.append(run_steps(mixer, cache, HIDDEN, [[(a, other[:200]), (b, x[:130]), (c, other)]], torch.bfloat16)[b])
    assert torch.isfinite(out[1]).all() and torch.equal(out[0], out[1])


@pytest.mark.parametrize("window, sink", [(None, True), (100, True), (None, False)])
@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("walk", [False, True])
def test_a_token_that_is_not_finite_reaches_the_rows_that_see_it_and_no_others(window, sink, bad, walk):
    """Rows before it, and rows whose window has left it behind, stay what they are (up to the order of a sum, which the prompt kernel
    chooses for 32 rows together); no row that sees it has a finite result."""
    mixer, _ = mixer_for(heads=2, window=window, sink=sink)
    w = weights_for(mixer, 8, {"_norm": lambda r: 1 + 0.3 * r, "sink": lambda r: r})
    mixer.bind(handles(w, torch.bfloat16), ctx_for(torch.bfloat16))
    if walk:
        mixer.kv_up = None
    x = torch.randn(420, HIDDEN, generator=torch.Generator().manual_seed(9)).to(torch.bfloat16).float()

    def run(rows):
        cache = SequenceCache([mixer.cache_requirement()], 2, 2048, 512, torch.bfloat16, DEV)
        a = cache.acquire()
        return run_steps(mixer, cache, HIDDEN, [[(a, rows[:260])], [(a, rows[260:])]], torch.bfloat16)[a]

    clean = run(x)
    for at in (1, 77, 127, 128, 250, 300):
        rows = x.clone()
        rows[at] = bad
        got = run(rows)
        sees = torch.zeros(420, dtype=torch.bool)
        sees[at:at + (window or 420)] = True
        assert float((got - clean)[~sees].abs().max()) <= 2 ** -8 * float(clean.abs().max()), at
        assert not torch.isfinite(got[sees]).any(), at
