"""Kernels that take several rows, heads or streams at once against plain float64, and against the forms they stand beside."""
import math
import os
import subprocess
import sys

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


@pytest.mark.parametrize("nq, nkv, d", [(8, 8, 128), (6, 2, 20), (8, 2, 128), (16, 8, 64), (3, 3, 256)])
def test_attention_over_a_few_keys_has_the_bits_of_single_heads(nq, nkv, d):
    g = torch.Generator().manual_seed(nq + d)
    k, v = (torch.randn(1, nkv, 64, d, generator=g).to(DEV) for _ in range(2))
    table = torch.zeros(1, 1, dtype=torch.int32, device=DEV)
    for keys in (1, 2, 7, 8, 9, 17):
        slot, pos = torch.zeros(keys, dtype=torch.int32, device=DEV), torch.arange(keys, dtype=torch.int32, device=DEV)
        q, outs = torch.randn(keys, nq * d, generator=g).to(DEV), []
        for room in (keys, 8, 40000):
            if room < keys:
                continue
            outs.append(torch.full((keys, nq * d), float("nan"), device=DEV))
            ops.attention_rows(q, nq * d, k, v, table, slot, pos, outs[-1], nq, nkv, d, 64, 0, room, d ** -0.5)
        assert all(torch.equal(o, outs[-1]) for o in outs)
        s = torch.einsum("ihd,hjd->hij", q.double().view(keys, nq, d), k[0, :, :keys].double().repeat_interleave(nq // nkv, 0)) * d ** -0.5
        s = s.masked_fill(torch.ones(keys, keys, device=DEV).triu(1).bool(), -math.inf)
        want = torch.einsum("hij,hjd->ihd", torch.softmax(s, -1), v[0, :, :keys].double().repeat_interleave(nq // nkv, 0)).flatten(1)
        assert float((outs[0].double() - want).abs().max()) <= 2e-6 * float(want.abs().max())


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("D, V, channel", [(128, 128, False), (20, 40, False), (160, 72, False), (48, 256, True)])
def test_delta_prepare_against_float64(taps, D, V, channel):
    H, KH, lengths, past = 4, 2, [5, 1, 17, 2, 8, 30], 3        # runs of eight rows begin in, at and between sequences
    T, C, GD = sum(lengths), 2 * KH * D + H * V, D if channel else 1
    g = torch.Generator().manual_seed(taps * D)
    proj = torch.randn(T, C + H * V + 2 * H, generator=g)
    decay = torch.randn(T, H * GD, generator=g) if channel else None
    w, a_log, bias = torch.randn(C, taps, generator=g), torch.randn(H, generator=g) * 0.3, torch.randn(H * GD, generator=g)
    state = torch.randn(8, H * D * V + (taps - 1) * C, generator=g)
    slots = [3, 0, 7, 5, 1, 2]
    bounds = torch.tensor([0] + lengths).cumsum(0)
    slot_of = torch.cat([torch.full((n,), s) for n, s in zip(lengths, slots)]).to(torch.int32)
    got, kept = {}, state.to(DEV)
    prep = torch.full((T, C + H + H * GD), float("nan"), device=DEV)
    i32 = lambda t: torch.as_tensor(t, dtype=torch.int32, device=DEV)
    ops.delta_prepare(proj.to(DEV), w.to(DEV), kept, H * D * V, i32(slot_of), i32(bounds), i32(slots), len(slots), a_log.to(DEV), bias.to(DEV),
                      prep, H, KH, D, V, 1e-6, decay_in=None if decay is None else decay.to(DEV), channel_decay=channel)
    prep = prep.cpu().double()
    for b, (n, s) in enumerate(zip(lengths, slots)):
        lo, hi = int(bounds[b]), int(bounds[b + 1])
        before = state[s, H * D * V:].view(taps - 1, C)
        x = torch.cat([before, proj[lo:hi, :C]]).double()
        y = sum(x[t:t + n] * w[:, t].double() for t in range(taps))
        y = y * torch.sigmoid(y)
        q, k = (z.reshape(n, KH, D) / torch.sqrt((z.reshape(n, KH, D) ** 2).sum(-1, keepdim=True) + 1e-6) for z in (y[:, :KH * D], y[:, KH * D:2 * KH * D]))
        want = torch.cat([q.flatten(1) * D ** -0.5, k.flatten(1), y[:, 2 * KH * D:]], 1)
        assert float((prep[lo:hi, :C] - want).abs().max()) <= 3e-6 * float(want.abs().max())
        beta = torch.sigmoid(proj[lo:hi, C + H * V:C + H * V + H].double())
        pre = decay[lo:hi] if channel else proj[lo:hi, C + H * V + H:]
        rate = torch.exp(a_log.double()).repeat_interleave(GD)
        decays = torch.exp(-rate * torch.nn.functional.softplus(pre.double() + bias.double()))
        assert float((prep[lo:hi, C:C + H] - beta).abs().max()) <= 1e-6 and float((prep[lo:hi, C + H:] - decays).abs().max()) <= 2e-6
        assert torch.equal(kept[s, H * D * V:].cpu().view(taps - 1, C), torch.cat([before, proj[lo:hi, :C]])[n:])


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("D, V, channel", [(128, 128, False), (20, 40, False), (160, 72, False), (48, 256, True)])
def test_delta_prepare_has_the_same_bits_in_steps_of_any_size(taps, D, V, channel):
    """Runs of rows and a warp a row: sequences in one step, and cut into steps of few rows and of a hundred."""
    H, KH, lengths, slots = 4, 2, [1, 700, 9, 2, 588], [3, 0, 4, 2, 1]
    if channel:                                                # more heads, for a step that takes runs
        H, KH = 14, 7
    T, C, GD = sum(lengths), 2 * KH * D + H * V, D if channel else 1
    takes_runs = lambda rows: bool(ops.lib().citlali_delta_prepare_in_runs(rows, H, KH, D, V, taps, int(channel)))
    assert takes_runs(T) and takes_runs(1) and takes_runs(2) != channel and not takes_runs(100)
    g = torch.Generator().manual_seed(taps * D + 1)
    dev = lambda *shape: torch.randn(*shape, generator=g).to(DEV)
    proj, decay = dev(T, C + H * V + 2 * H), dev(T, H * GD) if channel else None
    w, a_log, bias, state = dev(C, taps), 0.3 * dev(H), dev(H * GD), dev(5, H * D * V + (taps - 1) * C)
    i32 = lambda t: torch.as_tensor(t, dtype=torch.int32, device=DEV)

    def run(kept, rows, counts, of_slots):
        bounds = [sum(counts[:i]) for i in range(len(counts) + 1)]
        prep = torch.full((bounds[-1], C + H + H * GD), float("nan"), device=DEV)
        ops.delta_prepare(proj[rows].contiguous(), w, kept, H * D * V, i32([s for s, n in zip(of_slots, counts) for _ in range(n)]), i32(bounds),
                          i32(of_slots), len(counts), a_log, bias, prep, H, KH, D, V, 1e-6,
                          decay_in=None if decay is None else decay[rows].contiguous(), channel_decay=channel)
        return prep

    kept = state.clone()
    whole = run(kept, slice(0, T), lengths, slots)
    assert torch.isfinite(whole).all()
    for cut in (100, 1 if channel else 2):
        at, parts, part_kept = 0, [], state.clone()
        for n, s in zip(lengths, slots):
            parts += [run(part_kept, slice(at + i, at + min(i + cut, n)), [min(cut, n - i)], [s]) for i in range(0, n, cut)]
            at += n
        assert torch.equal(torch.cat(parts), whole) and torch.equal(part_kept, kept)


@pytest.mark.parametrize("S", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("rows, W", [(3, 64), (5, 30), (130, 2048)])
def test_stream_writes_against_float64(S, rows, W):
    g = torch.Generator().manual_seed(S * W)
    X, y = torch.randn(S, rows, W, generator=g), torch.randn(rows, W, generator=g)
    mix, w_out, w_in, gain = torch.randn(S, S, generator=g), torch.randn(S, generator=g), torch.randn(S, generator=g), torch.randn(W, generator=g)
    want = torch.einsum("st,srw->trw", mix.double(), X.double()) + w_out.double()[:, None, None] * y.double()
    wrote = X.to(DEV)
    ops.hyper_write(wrote, y.to(DEV), mix.to(DEV), w_out.to(DEV))
    assert float((wrote.cpu().double() - want).abs().max()) <= 3e-6 * float(want.abs().max())
    both, h = X.to(DEV), torch.empty(rows, W, device=DEV)
    ops.hyper_write_read_norm(both, y.to(DEV), mix.to(DEV), w_out.to(DEV), w_in.to(DEV), gain.to(DEV), 1e-5, h)
    assert torch.equal(both.cpu(), wrote.cpu())
    u = torch.einsum("s,srw->rw", w_in.double(), want)
    ref = u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-5) * gain.double()
    assert float((h.cpu().double() - ref).abs().max()) <= 2e-5 * float(ref.abs().max())


@pytest.mark.parametrize("V, H, extra", [(128, 5, 0), (36, 9, 4), (512, 2, 8), (300, 3, 0), (7, 4, 1), (516, 2, 0), (128, 3, 2)])
@pytest.mark.parametrize("act", ["silu", "sigmoid"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_delta_output_against_float64(V, H, extra, act, dtype):
    """Values in fours and others, gates on 16-byte boundaries and off them (rows a little wider than the gates)."""
    rows = 11
    g = torch.Generator().manual_seed(V * H)
    o, wide, w = torch.randn(rows, H * V, generator=g), torch.randn(rows, extra + H * V, generator=g), torch.randn(V, generator=g)
    z = wide.to(DEV)
    y = torch.full((rows, H * V), float("nan"), dtype=dtype, device=DEV)
    ops.delta_output(o.to(DEV), z[:, extra:], z.shape[1], w.to(DEV), y, H, V, 1e-5, gate_act=act)
    v, t = o.double().view(rows, H, V), wide[:, extra:].double().view(rows, H, V)
    s = torch.sigmoid(t)
    want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w.double() * (s if act == "sigmoid" else t * s)
    assert float((y.double().cpu().view(rows, H, V) - want).abs().max()) <= (3e-6 if dtype == torch.float32 else 2 ** -8) * float(want.abs().max())


@pytest.mark.parametrize("N, K, odd", [(48, 64, False), (130, 1000, False), (17, 333, False), (1024, 1024, False), (70, 128, True), (1, 1, False)])
def test_32_bit_products_give_a_row_the_same_bits_in_steps_of_any_size(N, K, odd):
    """Few rows, many rows and operands off 16-byte boundaries run different kernels with one chain an element."""
    g = torch.Generator().manual_seed(N + K)
    x, base = torch.randn(97, K, generator=g), torch.randn(97, N, generator=g).to(DEV)
    store = torch.zeros(N * K + 1, device=DEV)
    w = store[1:].view(N, K) if odd else store[:-1].view(N, K)
    w.copy_(torch.randn(N, K, generator=g))
    x, want = x.to(DEV), None
    for rows in (97, 1, 7, 8, 9, 31, 32, 65):
        y = torch.full((rows, N), float("nan"), device=DEV)
        ops.gemm_simt(x[:rows].contiguous(), w, y)
        added = base[:rows].clone()
        ops.gemm_simt(x[:rows].contiguous(), w, added, accumulate=True)
        if want is None:
            want, exact = y, x.double() @ w.double().T
            assert float((y.double() - exact).abs().max()) <= 2e-6 * K ** 0.5 * max(1.0, float(exact.abs().max()))
        assert torch.equal(y, want[:rows]) and torch.equal(added, base[:rows] + y)


@pytest.mark.parametrize("M, N, K, odd", [(64, 1024, 96, False), (65, 1531, 100, False), (682, 1024, 68, False), (500, 1100, 33, False),
                                          (130, 2300, 64, True), (273, 2400, 40, False), (1200, 1024, 36, False)])
def test_narrow_32_bit_products_give_the_bits_of_few_rows(M, N, K, odd):
    """Narrow tiles of 32, 48 and 80 columns, ragged rows, columns and last tiles of k, in pieces and element by element (the other widths and
    forms are in the next test)."""
    g = torch.Generator().manual_seed(M + N + K)
    store = torch.zeros(N * K + 1, device=DEV)
    w = store[1:].view(N, K) if odd else store[:-1].view(N, K)
    w.copy_(torch.randn(N, K, generator=g))
    x, base = torch.randn(M, K, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)
    y, added = torch.full((M, N), float("nan"), device=DEV), base.clone()
    ops.gemm_simt(x, w, y)
    ops.gemm_simt(x, w, added, accumulate=True)
    few = torch.empty(31, N, device=DEV)
    for r in range(0, M, 31):
        n = min(31, M - r)
        ops.gemm_simt(x[r:r + n].contiguous(), w, few[:n])
        assert torch.equal(y[r:r + n], few[:n])
    assert torch.equal(added, base + y)


@pytest.mark.parametrize("M, N, K, odd", [(65, 500, 50, False), (65, 2391, 67, False), (65, 3611, 68, True), (65, 4770, 201, False),
                                          (200, 5929, 101, False), (65, 3611, 36, False), (200, 5929, 72, False), (1400, 1280, 159, False),
                                          (1400, 1280, 161, False), (980, 2300, 100, True), (65, 500, 48, True), (65, 500, 47, False)])
def test_32_bit_products_that_cannot_be_copied_in_pieces_and_the_widest_tiles(M, N, K, odd):
    """Element by element in every width of the narrow tiles (32 to 96 columns) and in the transposed tiles of 64 columns, either side of
    the lines between them; in pieces the two widths that the sizes above do not reach."""
    g = torch.Generator().manual_seed(M + N + K)
    store = torch.zeros(N * K + 1, device=DEV)
    w = store[1:].view(N, K) if odd else store[:-1].view(N, K)
    w.copy_(torch.randn(N, K, generator=g))
    x, base = torch.randn(M, K, generator=g).to(DEV), torch.randn(M, N, generator=g).to(DEV)
    y, added = torch.full((M, N), float("nan"), device=DEV), base.clone()
    ops.gemm_simt(x, w, y)
    ops.gemm_simt(x, w, added, accumulate=True)
    few = torch.empty(31, N, device=DEV)
    for r in range(0, M, 31):
        n = min(31, M - r)
        ops.gemm_simt(x[r:r + n].contiguous(), w, few[:n])
        assert torch.equal(y[r:r + n], few[:n])
    assert torch.equal(added, base + y)


_SHARED_MEMORY_LIMITS = """
import sys
sys.path.insert(0, {root!r})
import torch
import citlali_b200
from citlali_b200 import ops
DEV, d, page = torch.device("cuda:0"), 128, 64
g = torch.Generator().manual_seed(1)
pool = torch.randn(191, 1, page, d, generator=g).to(DEV)
table = torch.arange(191, dtype=torch.int32, device=DEV)[None].contiguous()
slot = torch.zeros(1, dtype=torch.int32, device=DEV)
close = lambda a, b: float((a.double() - b).abs().max()) <= 1e-5 * float(b.abs().max())      # sums of up to 12,289 in float32


def attention(nq, keys, room):
    q = torch.randn(1, nq * d, generator=torch.Generator().manual_seed(keys)).to(DEV)
    out = torch.full((1, nq * d), float("nan"), device=DEV)
    ops.attention_rows(q, nq * d, pool, pool, table, slot, slot + (keys - 1), out, nq, 1, d, page, 0, room, d ** -0.5)
    return out


# the form of one head at a time first: the reference below needs more shared memory and leaves a higher limit behind
lengths = [(nq, keys) for nq in (1, 2, 4) for keys in (12128, 12129, 12144, 12160, 12161)]
lengths += [(4, n) for n in range(2451, 2459)] + [(2, n) for n in range(4090, 4098)] + [(1, n) for n in range(6140, 6146)]
for (nq, keys), out in [(c, attention(*c, c[1])) for c in lengths]:
    assert torch.isfinite(out).all() and torch.equal(out, attention(nq, keys, 40000)), (nq, keys)

for W in (12255, 12256, 12264, 12270, 12288, 12289):          # a row of floats beside a block sum's 128 bytes
    X, y = torch.randn(3, 2, W, generator=g).to(DEV), torch.randn(2, W, generator=g).to(DEV)
    ones, eye = torch.ones(3, device=DEV), torch.eye(3, device=DEV)
    gain = torch.ones(W, device=DEV)
    norm = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    h = torch.empty(2, W, device=DEV)
    ops.hyper_read_norm(X, ones, gain, 1e-5, h)
    assert close(h, norm(X.double().sum(0))), W
    wrote = X.clone()
    ops.hyper_write_read_norm(wrote, y, eye, ones, ones, gain, 1e-5, h)
    assert close(h, norm((X.double() + y.double()).sum(0))), W
    x = torch.zeros(2, W, device=DEV)
    ops.layer_norm_add(y, gain, 1e-5, x)
    ops.layer_norm_rows(y, gain, 1e-5, h)
    centred = y.double() - y.double().mean(-1, keepdim=True)
    assert close(x, norm(centred)) and close(h, norm(centred)), W
for bw in (1280, 1281, 1536):                                  # eight rows of a gate block beside 8 KB of partial sums
    u, wa, wi = torch.randn(3, bw, generator=g).to(DEV), *(torch.randn(1, bw, bw, generator=g).to(DEV) / bw ** 0.5 for _ in range(2))
    zero, a, coef = torch.zeros(bw, device=DEV), torch.empty(3, bw, device=DEV), torch.empty(3, bw, device=DEV)
    ops.lru_gates(u, wa, zero, wi, zero, zero, a, coef, 1)
    log_a = -8.0 * torch.sigmoid(u.double() @ wa[0].double()) * torch.log(torch.tensor(2.0, dtype=torch.float64))
    assert close(a, torch.exp(log_a)) and close(coef, torch.sqrt(-torch.expm1(2 * log_a)) * torch.sigmoid(u.double() @ wi[0].double()) * u.double()), bw
print("every length ran")
"""


def test_every_length_around_the_default_limit_of_shared_memory_runs():
    """48 KB a block count a kernel's own arrays too.  In a process of its own: a launch that raises a kernel's limit raises it for later
    ones, so another test's longer rows would hide what is looked for."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SHARED_MEMORY_LIMITS.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "every length ran" in r.stdout, r.stdout + r.stderr
