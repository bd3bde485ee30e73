"""What the library is timed on: steps of whole models through ``InferenceSession``, as a serving or replaying program calls it.

A case names a model (``design`` and its sizes), the compute dtype and one step:

* ``prompt``: new sequences in one step, logits of every sequence's last token (``want: "all"``: of every token, what a
  replay of a trace asks for).  The slots are taken and given back inside the pass.
* ``extend``: sequences that hold ``context`` tokens go on by several (a chat's next turn, a long prompt in portions).
* ``decode``: every sequence gets one token through ``InferenceSession.decode`` (the replayed graph where the model has
  one, else ``step`` and the sampler), greedy.  What comes back are the step's logits, not the tokens: among 152,000 nearly
  level logits of a random model the largest one changes with the last bit.

Lengths are ``tokens`` for every sequence, or drawn between ``shortest`` and ``tokens`` from ``lengths`` (a seed of the
case, so that every pass and every seed of the inputs does the same work).  Token ids come from ``seed``; the model is one
model, as a program loads one (``WEIGHTS``).

Three designs stand for the seven: Qwen3 (the dense decoder that the library serves first, and its benchmark's model),
Lanizen (a matrix of state a head, latent attention, several residual streams) and Pivavik (latent and soft-capped window
attention beside biased feed-forwards, a repeated run of layers).  Layers that route tokens to experts are not held here:
where two experts' scores nearly tie, a last bit of rounding changes the expert, and with it the logits by tens of per
cent, so no tolerance tells a fault from a tie.
"""
from __future__ import annotations

import math
import random

import torch

import citlali_b200 as cb
from citlali_b200.engine.step import StepEntry

DEVICE = "cuda:0"
WEIGHTS = 1                # the seed of every model's random weights
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# ---- the cases --------------------------------------------------------------------------------------------------------------

# the shapes the benchmark runs, Qwen3-8B and Qwen3-1.7B, at a third and at half of their depth: all layers are alike, and through
# all 36 of them the rounding noise of bfloat16 on random weights adds up to more than a tolerance can tell from a fault
QWEN3_8B = dict(design="qwen3", layers=12, width=4096, heads=32, kv_heads=8, head_dim=128, ff=12288, vocab=151936, tied=False)
QWEN3_1_7B = dict(design="qwen3", layers=14, width=2048, heads=16, kv_heads=8, head_dim=128, ff=6144, vocab=151936, tied=True)


def _four_layers(design, width, **more):
    """The sizes ``bench.py --design`` compares designs at: four layers, heads of 128, a vocabulary of 32,768."""
    heads = max(1, width // 128)
    sizes = dict(design=design, layers=4, width=width, heads=heads, head_dim=128, vocab=32768)
    if design == "qwen3":
        sizes.update(kv_heads=max(1, heads // 4), ff=(8 * width // 3 + 255) // 256 * 256, tied=False)
    elif design == "lanizen":
        sizes.update(kv_heads=max(1, heads // 2), ff=4 * width, streams=4, window=1024, kv_rank=512, rot_dim=64)
    else:
        sizes.update(kv_heads=max(1, heads // 4), ff=(8 * width // 3 + 255) // 256 * 256, window=1024, kv_rank=512, rot_dim=64)
    sizes.update(more)
    return sizes


def _case(name, model, dtype, step, batch, tokens, shortest=0, context=0, want="last", lengths=0):
    c = dict(model, dtype=dtype, step=step, batch=batch, tokens=tokens, shortest=shortest or tokens, context=context, want=want,
             lengths=lengths)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the benchmark's prompt: one long prompt, the time to a first token
        _case("qwen3-8b prompt 2048", QWEN3_8B, "bfloat16", "prompt", 1, 2048),
        # the benchmark's headline: eight sequences decoding near the context limit, bound by the bytes of weights and keys
        _case("qwen3-8b decode 8 at 4000", QWEN3_8B, "bfloat16", "decode", 8, 1, context=4000),
        # chat turns: conversations of unequal length go on by some hundred tokens each
        _case("qwen3-8b extend 4 at 1500", QWEN3_8B, "bfloat16", "extend", 4, 333, shortest=40, context=1500, lengths=3),
        # the batch workload of unequal prompts, in one step
        _case("qwen3-1.7b 16 prompts", QWEN3_1_7B, "bfloat16", "prompt", 16, 1024, shortest=64, lengths=1),
        # a single short question: the step's launches are all there is
        _case("qwen3-1.7b prompt 23", QWEN3_1_7B, "bfloat16", "prompt", 1, 23),
        # one user's reply, token by token
        _case("qwen3-1.7b decode 1 at 700", QWEN3_1_7B, "bfloat16", "decode", 1, 1, context=700),
        # the true 32-bit path, as a trace replay uses it: unequal prompts, logits of every token
        _case("qwen3 float32 replay", _four_layers("qwen3", 1024), "float32", "prompt", 3, 301, shortest=77, want="all", lengths=2),
        # the recurrent design: a long prompt and a batch of unequal ones at another width, then decoding
        _case("lanizen prompt 2048", _four_layers("lanizen", 4096), "bfloat16", "prompt", 1, 2048),
        _case("lanizen 5 prompts", _four_layers("lanizen", 2048), "bfloat16", "prompt", 5, 700, shortest=50, lengths=4),
        _case("lanizen decode 8 at 2048", _four_layers("lanizen", 4096), "bfloat16", "decode", 8, 1, context=2048),
        # the latent and windowed attention design: a long prompt, then decoding over every earlier token
        _case("pivavik prompt 2048", _four_layers("pivavik", 4096), "bfloat16", "prompt", 1, 2048),
        _case("pivavik decode 8 at 2048", _four_layers("pivavik", 2048, window=0), "bfloat16", "decode", 8, 1, context=2048),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))) - 0.5))))


def draw(rng):
    """Another case of the ranges the listed ones stand for: any of the three designs and of the steps it is held in, 1 to 16
    sequences, 1 to 3,000 tokens each, contexts up to 4,000, widths 1,024 to 4,096, both dtypes."""
    while True:
        design = rng.choice(["qwen3", "qwen3", "qwen3", "lanizen", "lanizen", "pivavik", "pivavik"])
        dtype = "float32" if rng.random() < 0.15 else "bfloat16"
        if design == "qwen3" and dtype == "bfloat16" and rng.random() < 0.5:
            model = dict(rng.choice([QWEN3_8B, QWEN3_1_7B]))
        else:
            model = _four_layers(design, rng.choice([1024, 2048, 4096]) if dtype == "bfloat16" else 1024)
        step = rng.choice(["prompt", "decode", "extend"] if design == "qwen3" else ["prompt", "prompt", "decode"])
        batch = _log_uniform(rng, 1, 16)
        context = 0 if step == "prompt" else _log_uniform(rng, 16, 4000 if dtype == "bfloat16" else 500)
        tokens = 1 if step == "decode" else _log_uniform(rng, 2, 3000 if dtype == "bfloat16" else 400)
        shortest = rng.randint(max(1, tokens // 8), tokens)
        if design == "pivavik":
            model["window"] = 0 if step == "decode" else rng.choice([0, 100, 1024])
        want = "all" if dtype == "float32" and step == "prompt" else "last"
        c = _case(None, model, dtype, step, batch, tokens, shortest=shortest, context=context, want=want, lengths=rng.randint(0, 10**6))
        # no more than the listed cases' largest; the two smaller designs take more time an operation
        top = 1.1e11 if dtype == "float32" else 1.0e13 if design == "qwen3" else 4.0e12
        if work(c)["flops"] <= top and batch * (context + tokens) <= 33000:
            return c


# ---- what a case's sizes mean -------------------------------------------------------------------------------------------------

def _lengths(case):
    """The tokens each sequence brings."""
    rng = random.Random(case["lengths"])
    return [rng.randint(case["shortest"], case["tokens"]) for _ in range(case["batch"])]


def _past(case):
    """The tokens each sequence holds before the pass: unequal, up to ``context``."""
    rng = random.Random(case["lengths"] + 1)
    return [rng.randint(case["context"] * 3 // 4, case["context"]) if case["step"] == "extend" else case["context"]
            for _ in range(case["batch"])]


def _tokens(case, seed):
    """Per sequence: the tokens it holds and the tokens it brings."""
    gen = torch.Generator().manual_seed(seed * 7919 + 17)
    ids = lambda n: torch.randint(0, case["vocab"], (n,), generator=gen).tolist()
    return [(ids(p), ids(n)) for p, n in zip(_past(case), _lengths(case))]


def _layer_kinds(case):
    kinds = {"qwen3": ["attention"], "lanizen": ["delta", "delta", "delta", "latent"], "pivavik": ["latent", "window"]}[case["design"]]
    return [kinds[i % len(kinds)] for i in range(case["layers"])]


def _q_rank(case):
    return max(256, case["width"] * 3 // 8)


def _scale(case, kind):
    return (case["head_dim"] + (case["rot_dim"] if kind == "latent" else 0)) ** -0.5


def _mask(case):
    return {"mask": {"size": case["window"]}} if case["window"] else {}


def _config(case):
    """The configuration as config.json would hold it."""
    W, H, G, D = case["width"], case["heads"], case["kv_heads"], case["head_dim"]
    if case["design"] == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=case["layers"], hidden_size=W, num_attention_heads=H,
                    num_key_value_heads=G, head_dim=D, intermediate_size=case["ff"], vocab_size=case["vocab"], rope_theta=1e6,
                    rms_norm_eps=1e-6, tie_word_embeddings=case["tied"], max_position_embeddings=40960)
    latent = {"heads": H, "dim": D, "rot_dim": case["rot_dim"], "vdim": D, "q_rank": _q_rank(case), "kv_rank": case["kv_rank"],
              "scale": _scale(case, "latent"), "rot": {"base": 10000.0, "dims": case["rot_dim"]}}
    mlp = {"kind": "dense", "ff": case["ff"]}
    if case["design"] == "lanizen":
        delta = {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "conv": 4}
        mixer = {"delta": ("delta", delta), "latent": ("latent_attention", dict(latent, **_mask(case)))}
        top = {"architecture": "Lanizen", "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "streams": case["streams"]}
    else:
        window = {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": _scale(case, "window"), "softcap": 30.0, **_mask(case)}
        mixer = {"latent": ("latent_attention", latent), "window": ("attention", window)}
        top = {"architecture": "Pivavik", "norm": {"eps": 1e-5}, "logit_softcap": 30.0,
               "loop": {"start": 1, "stop": case["layers"] - 1, "times": 1}}
    return dict(top, vocab=case["vocab"], width=W, layers=[{"type": mixer[k][0], "mixer": dict(mixer[k][1]), "mlp": dict(mlp)}
                                                           for k in _layer_kinds(case)])


def work(case):
    """Every matrix and every visible cached key once, the new keys and the logits once; two operations a multiply-add."""
    W, H, G, D, F = case["width"], case["heads"], case["kv_heads"], case["head_dim"], case["ff"]
    size = 4 if case["dtype"] == "float32" else 2
    past, new = _past(case), _lengths(case)
    rows = sum(new)
    wanted = rows if case["want"] == "all" else case["batch"]
    weights, flops, moved = 0, 0.0, 0.0

    def keys_seen(window):
        """(row, visible key) pairs, and the cached keys that any new row sees."""
        pairs = seen = 0
        for p, n in zip(past, new):
            pairs += sum(min(i + 1, window) if window else i + 1 for i in range(p, p + n))
            seen += min(p, window - 1) if window else p
        return pairs, seen

    for kind in _layer_kinds(case):
        if kind in ("attention", "window"):
            qkv = (H + 2 * G) * D * W + H * D * W + (H * D * W if kind == "window" else 0)
            pairs, seen = keys_seen(case.get("window", 0) if kind == "window" else 0)
            flops += 4.0 * pairs * H * D
            moved += (seen + rows) * 2 * G * D * size
        elif kind == "delta":
            qkv = 2 * G * D * W + H * D * W * 3 + 2 * H * W
            flops += 6.0 * rows * H * D * D
            moved += 2.0 * case["batch"] * H * D * D * 4
        else:
            R, P, Q = case["kv_rank"], case["rot_dim"], _q_rank(case)
            gate = H * D * W if case["design"] == "lanizen" else H * W
            qkv = Q * W + Q * H * (D + P) + (R + P) * W + 2 * R * H * D + gate + H * D * W
            pairs, seen = keys_seen(case["window"] if case["design"] == "lanizen" else 0)
            flops += 2.0 * pairs * H * (2 * D + P)
            moved += (seen + rows) * (R + P) * size
        weights += qkv + (2 if case["design"] == "lanizen" else 3) * W * F
    if case["design"] == "pivavik":
        weights += 2 * W * W
    flops += 2.0 * rows * weights + 2.0 * wanted * W * case["vocab"]
    return {"bytes": (weights + W * case["vocab"] + rows * W) * size + moved + 4.0 * wanted * case["vocab"], "flops": flops}


def tolerance(case):
    """About four times the distance from ``exact`` as measured: 3e-6 in float32; in bfloat16 0.003 (lanizen), 0.006 (pivavik) and
    0.02 to 0.026 for the deeper Qwen3 models, where it is held tighter than that."""
    if case["dtype"] == "float32":
        return {"rel": 1.2e-5}
    return {"rel": {"qwen3": 0.03, "lanizen": 0.012, "pivavik": 0.024}[case["design"]]}


# ---- preparing and running -----------------------------------------------------------------------------------------------------

class State:
    """A loaded session, the sequences it holds and the step's tokens."""

    def __init__(self, case, seed):
        self.step = case["step"]
        held = _tokens(case, seed)
        self.new = [n for _, n in held]
        self.past = [len(p) for p, _ in held]
        longest = max(p + len(n) for p, n in zip(self.past, self.new))
        # a model that cannot be rewound goes on from where the last pass left it
        self.rewinds = case["design"] == "qwen3" or (case["design"] == "pivavik" and not case["window"])
        room = 0 if case["step"] == "prompt" or self.rewinds else 20000
        self.session = cb.InferenceSession().load_random(cb.config_from_dict(_config(case)), seed=WEIGHTS, max_context=longest + 8 + room,
                                                         dtype=case["dtype"], device=DEVICE, max_batch=case["batch"], gain_spread=0.1)
        self.slots = []
        self.entry_want = (lambda n: list(range(n))) if case["want"] == "all" else (lambda n: [n - 1])
        if self.step != "prompt":
            self.slots = [self.session.acquire() for _ in held]
            decodes = self.step == "decode"
            for slot, (p, _) in zip(self.slots, held):
                self.session.step([StepEntry(slot, p[:-1] if decodes else p, [])])
            if decodes:                       # a program that decodes has decoded before: the step's graph is there
                self.decode([p[-1] for p, _ in held])

    def entries(self, slots):
        return [StepEntry(s, n, self.entry_want(len(n))) for s, n in zip(slots, self.new)]

    def decode(self, fed):
        session = self.session
        if session.runner is not None:
            session.decode(self.slots, fed, 0.0, [])
            return session.runner.logits[(len(fed), True)]
        logits = session.step([StepEntry(s, [t], [0]) for s, t in zip(self.slots, fed)])
        session.sampler.sample(logits, 0.0, [])
        return logits


def prepare(case, seed):
    return State(case, seed)


def run(state):
    session = state.session
    if state.step != "prompt" and state.rewinds:
        for slot, p in zip(state.slots, state.past):
            session.cache.rewind(slot, p)
    if state.step == "decode":
        return state.decode([n[0] for n in state.new])
    if state.step == "extend":
        return session.step(state.entries(state.slots))
    slots = [session.acquire() for _ in state.new]
    logits = session.step(state.entries(slots))
    for slot in slots:
        session.release(slot)
    return logits


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------------

def _rms(x, eps, gain=1.0):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _rotate(x, positions, dims, base, halves):
    """x [T, heads, n]: pairs among the first ``dims`` elements turn by position * base^(-2i/dims); a pair is (i, i + dims/2) or
    (2i, 2i + 1)."""
    half = dims // 2
    freq = base ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / dims)
    angle = positions.double()[:, None, None] * freq
    c, s = angle.cos(), angle.sin()
    out = x.clone()
    a, b = (slice(0, half), slice(half, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


class _Exact:
    """The model in float64 on rows of all sequences side by side; logits of the wanted rows."""

    def __init__(self, case, seed):
        self.case = case
        self.seqs = [p + n for p, n in _tokens(case, seed)]
        self.bounds, at = [], 0
        for s in self.seqs:
            self.bounds.append((at, at + len(s)))
            at += len(s)
        self.positions = torch.cat([torch.arange(len(s), device=DEVICE) for s in self.seqs])

    def w(self, name, *shape, gain=False):
        """The tensor that ``load_random`` makes of this name: N(0, 0.02), or a gain 1 + N(0, 0.1), from a seed made of the name
        (64-bit FNV-1a), rounded to the compute dtype."""
        h = 0xCBF29CE484222325 ^ WEIGHTS
        for b in name.encode():
            h = ((h ^ b) * 0x100000001B3) & 0xFFFFFFFFFFFFFFFF
        gen = torch.Generator(device=DEVICE).manual_seed(h & 0x7FFFFFFFFFFFFFFF)
        t = torch.randn(shape, generator=gen, dtype=torch.float32, device=DEVICE)
        t = t * 0.1 + 1.0 if gain else t * 0.02
        return t.to(DTYPES[self.case["dtype"]]).double()

    def linear(self, x, name, out, bias=False):
        y = x @ self.w(name, out, x.shape[1]).T
        return y + self.w(name + ".b", out) if bias else y

    def causal(self, q, k, v, scale, window=0, cap=0.0, sink=None):
        """q [rows, H, d], k [rows, G, d], v [rows, G, e] of all sequences; softmax over a row's visible keys, and over a head's
        ``sink`` beside them, which has no value."""
        H, G = q.shape[1], k.shape[1]
        out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device=q.device)
        for lo, hi in self.bounds:
            n = hi - lo
            far = torch.arange(n, device=q.device)[:, None] - torch.arange(n, device=q.device)[None, :]
            hidden = (far < 0) | (far >= window) if window else far < 0
            for g in range(G):
                heads = slice(g * (H // G), (g + 1) * (H // G))
                s = torch.einsum("ihd,jd->hij", q[lo:hi, heads], k[lo:hi, g]) * scale
                s = (cap * torch.tanh(s / cap) if cap else s).masked_fill_(hidden, -math.inf)
                if sink is not None:
                    s = torch.cat([s, sink[heads, None, None].expand(-1, n, 1)], -1)
                out[lo:hi, heads] = torch.einsum("hij,je->ihe", torch.softmax(s, -1)[..., :n], v[lo:hi, g])
        return out

    def latent(self, h, p, eps, window, halves):
        c = self.case
        H, D, P, R, Q = c["heads"], c["head_dim"], c["rot_dim"], c["kv_rank"], _q_rank(c)
        down = self.linear(h, p + ".dkv", R + P)
        lat = _rms(down[:, :R], eps, self.w(p + ".dkv.norm", R, gain=True))
        shared = _rotate(down[:, None, R:], self.positions, P, 10000.0, halves)
        q = self.linear(_rms(self.linear(h, p + ".dq", Q), eps, self.w(p + ".dq.norm", Q, gain=True)), p + ".uq", H * (D + P)).view(-1, H, D + P)
        q = torch.cat([q[..., :D], _rotate(q[..., D:], self.positions, P, 10000.0, halves)], -1)
        k = torch.cat([self.linear(lat, p + ".uk", H * D).view(-1, H, D), shared.expand(-1, H, -1)], -1)
        o = self.causal(q, k, self.linear(lat, p + ".uv", H * D).view(-1, H, D), _scale(c, "latent"), window,
                        sink=self.w(p + ".sink", H) if c["design"] == "lanizen" else None)
        if c["design"] == "lanizen":
            o = o.flatten(1) * torch.sigmoid(self.linear(h, p + ".g", H * D))
        else:
            o = (o * torch.sigmoid(self.linear(h, p + ".g", H))[..., None]).flatten(1)
        return self.linear(o, p + ".o", c["width"])

    def delta(self, h, p, eps):
        c = self.case
        H, G, D = c["heads"], c["kv_heads"], c["head_dim"]

        def channels(name, n):
            x, taps = self.linear(h, f"{p}.{name}", n), self.w(f"{p}.{name}.conv", n, 4)
            y = x * taps[:, 3]
            for lo, hi in self.bounds:
                for back in range(1, min(4, hi - lo)):
                    y[lo + back:hi] += x[lo:hi - back] * taps[:, 3 - back]
            return torch.nn.functional.silu(y)

        unit = lambda x: x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        q = unit(channels("q", G * D).view(-1, G, D)).repeat_interleave(H // G, 1) * D ** -0.5
        k = unit(channels("k", G * D).view(-1, G, D)).repeat_interleave(H // G, 1)
        v = channels("v", H * D).view(-1, H, D)
        beta = torch.sigmoid(self.linear(h, p + ".b", H))
        step = torch.nn.functional.softplus(self.linear(h, p + ".a", H) + self.w(p + ".dt_bias", H))
        g = torch.exp(-torch.exp(self.w(p + ".A_log", H)) * step)
        o = torch.empty_like(v)
        # all sequences walk together; one that has ended is fed zeros, which its state no longer matters for
        longest = max(hi - lo for lo, hi in self.bounds)
        pad = lambda x: torch.stack([torch.nn.functional.pad(x[lo:hi], [0, 0] * (x.dim() - 1) + [0, longest - (hi - lo)])
                                     for lo, hi in self.bounds], 1)
        Q, K, V, B, E = pad(q), pad(k), pad(v), pad(beta), pad(g)
        S = torch.zeros(len(self.bounds), H, D, D, dtype=torch.float64, device=h.device)
        walked = torch.empty_like(V)
        for t in range(longest):
            S = S * E[t][..., None, None]
            u = (V[t] - torch.einsum("bhdv,bhd->bhv", S, K[t])) * B[t][..., None]
            S.addcmul_(K[t][..., :, None], u[..., None, :])
            walked[t] = torch.einsum("bhdv,bhd->bhv", S, Q[t])
        for i, (lo, hi) in enumerate(self.bounds):
            o[lo:hi] = walked[:hi - lo, i]
        o = _rms(o, eps, self.w(p + ".norm", D, gain=True)).flatten(1) * torch.nn.functional.silu(self.linear(h, p + ".g", H * D))
        return self.linear(o, p + ".o", c["width"])

    def embedded(self, name):
        table = self.w(name, self.case["vocab"], self.case["width"])
        return table[torch.tensor([t for s in self.seqs for t in s], device=DEVICE)]

    def wanted(self):
        places = []
        for (lo, hi), n in zip(self.bounds, _lengths(self.case)):
            places += list(range(lo, hi)) if self.case["want"] == "all" else [hi - 1]
        return torch.tensor(places, device=DEVICE)

    def qwen3(self):
        c, eps = self.case, 1e-6
        W, H, G, D, F = c["width"], c["heads"], c["kv_heads"], c["head_dim"], c["ff"]
        x = self.embedded("model.embed_tokens.weight")
        for i in range(c["layers"]):
            p = f"model.layers.{i}"
            norm = lambda y, name, n: _rms(y, eps, self.w(f"{p}.{name}.weight", n, gain=True))
            lin = lambda y, name, out: self.linear(y, f"{p}.{name}.weight", out)
            h = norm(x, "input_layernorm", W)
            q = norm(lin(h, "self_attn.q_proj", H * D).view(-1, H, D), "self_attn.q_norm", D)
            k = norm(lin(h, "self_attn.k_proj", G * D).view(-1, G, D), "self_attn.k_norm", D)
            q, k = (_rotate(t, self.positions, D, 1e6, True) for t in (q, k))
            o = self.causal(q, k, lin(h, "self_attn.v_proj", G * D).view(-1, G, D), D ** -0.5)
            x = x + lin(o.flatten(1), "self_attn.o_proj", W)
            h = norm(x, "post_attention_layernorm", W)
            x = x + lin(torch.nn.functional.silu(lin(h, "mlp.gate_proj", F)) * lin(h, "mlp.up_proj", F), "mlp.down_proj", W)
        h = _rms(x[self.wanted()], eps, self.w("model.norm.weight", W, gain=True))
        return self.linear(h, "model.embed_tokens.weight" if c["tied"] else "lm_head.weight", c["vocab"])

    def lanizen(self):
        c, eps, S = self.case, 1e-6, self.case["streams"]
        W = c["width"]
        X = self.embedded("embed").expand(S, -1, -1)
        for i, kind in enumerate(_layer_kinds(c)):
            p = f"l{i}"
            for sub in (1, 2):
                read = torch.einsum("s,stw->tw", self.w(f"{p}.hc{sub}.in", S), X)
                h = _rms(read, eps, 1.0 + self.w(f"{p}.norm{sub}", W, gain=True))
                if sub == 2:
                    y = self.linear(torch.relu(self.linear(h, p + ".mlp.up", c["ff"])) ** 2, p + ".mlp.down", W)
                else:
                    y = self.delta(h, p + ".mix", eps) if kind == "delta" else self.latent(h, p + ".mix", eps, c["window"], False)
                X = torch.einsum("st,srw->trw", self.w(f"{p}.hc{sub}.mix", S, S), X) + self.w(f"{p}.hc{sub}.out", S)[:, None, None] * y
        h = _rms(X.sum(0)[self.wanted()], eps, 1.0 + self.w("final.norm", W, gain=True))
        return self.linear(h, "head", c["vocab"])

    def pivavik(self):
        c, eps = self.case, 1e-5
        W, H, G, D, F = c["width"], c["heads"], c["kv_heads"], c["head_dim"], c["ff"]
        x0 = _rms(self.embedded("embed"), eps, 1.0 + self.w("embed.norm", W, gain=True))
        x = x0
        for i, kind in enumerate(_layer_kinds(c)):
            p = f"l{i}"
            if i == 1:                                 # ahead of the repeated run's only pass
                x = self.linear(torch.cat([x, x0], -1), "loop.in", W) + self.w("loop.step", 1, W)[0]
            h = _rms(x, eps, 1.0 + self.w(p + ".norm1", W, gain=True))
            if kind == "latent":
                y = self.latent(h, p + ".mix", eps, 0, True)
            else:
                q, k, v = (self.linear(h, f"{p}.mix.{n}", heads * D, bias=True).view(-1, heads, D) for n, heads in (("q", H), ("k", G), ("v", G)))
                o = self.causal(q, k, v, _scale(c, kind), c["window"], 30.0).flatten(1)
                y = self.linear(o * torch.sigmoid(self.linear(h, p + ".mix.g", H * D)), p + ".mix.o", W)
            gate, up = (self.linear(h, f"{p}.mlp.{n}", F, bias=True) for n in ("gate", "up"))
            x = x + y + self.linear(torch.nn.functional.gelu(gate, approximate="tanh") * up, p + ".mlp.down", W, bias=True)
        h = _rms(x[self.wanted()], eps, 1.0 + self.w("final.norm", W, gain=True))
        return 30.0 * torch.tanh(self.linear(h, "embed", c["vocab"]) / 30.0)


def exact(case, seed):
    """The logits in 64 bits, on the GPU by plain torch."""
    whole = dict(case, batch=case["batch"], step="prompt")
    rows = sum(p + n for p, n in zip(_past(case), _lengths(case)))
    if rows * work(whole)["flops"] / max(1, sum(_lengths(case))) > 2.5e14:        # beyond about 20 seconds
        return None
    return getattr(_Exact(case, seed), case["design"])()
