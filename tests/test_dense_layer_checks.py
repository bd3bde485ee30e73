"""What a layer from one call refuses before anything is launched: tensors of other types, sizes or places than its kernels read and
write.  The tensors are stand-ins without memory, so nothing here needs a GPU."""
import os
import re
import struct
import types

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from citlali_b200 import ops
from citlali_b200.csrc import build
from citlali_b200.errors import CitlaliError
from citlali_b200.parts.base import StepBatch

ROWS, HIDDEN, INTER, NQ, NKV, D = 23, 64, 48, 4, 2, 16


def _given():
    """The arguments of a call that is taken, by name, as stand-ins on a CUDA device."""
    dev = "cuda:0"
    bf = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device=dev)
    f32 = lambda *s: torch.empty(*s, dtype=torch.float32, device=dev)
    i32 = lambda *s: torch.empty(*s, dtype=torch.int32, device=dev)
    wide = (NQ + 2 * NKV) * D
    a = dict(qkv=bf(wide, HIDDEN), o=bf(HIDDEN, NQ * D), gate_up=bf(2 * INTER, HIDDEN), down=bf(HIDDEN, INTER), q_gain=bf(D), k_gain=bf(D),
             inv_freq=f32(D // 2), keys=bf(3, 64, NKV, D), values=bf(3, 64, NKV, D), page_table=i32(2, 3), x=f32(ROWS, HIDDEN),
             s_qkv=bf(ROWS, wide), s_heads=bf(ROWS, NQ * D), s_act=bf(ROWS, INTER), error_flag=i32(4), tokens=i32(ROWS), row_slot=i32(ROWS),
             row_pos=i32(ROWS), seq_start=i32(3), seq_slot=i32(2), seq_past=i32(2))
    for name in ("in", "mid", "out"):
        a[name + "_rows"], a[name + "_sums"] = bf(ROWS, HIDDEN), f32(ROWS, HIDDEN // 32)
    return a


def _call(a):
    batch = StepBatch(tokens=a["tokens"], row_slot=a["row_slot"], row_pos=a["row_pos"], seq_start=a["seq_start"], seq_slot=a["seq_slot"],
                      seq_past=a["seq_past"], want_rows=None, slots=[0, 1], past=[0, 0], n_new=[ROWS - 2, 2])
    cache = types.SimpleNamespace(keys=a["keys"], values=a["values"], page_table=a["page_table"], page_size=64)
    ops.dense_layer((a["qkv"], a["o"], a["gate_up"], a["down"]), (a["q_gain"], a["k_gain"]), a["inv_freq"], D, cache,
                    (HIDDEN, INTER, NQ, NKV, D, 0), (1e-6, 1e-6, 1e-6), a["x"], (a["s_qkv"], a["s_heads"], a["s_act"]),
                    (a["in_rows"], a["in_sums"]), (a["mid_rows"], a["mid_sums"]), (a["out_rows"], a["out_sums"]), batch, a["error_flag"], 0.25)


@pytest.fixture
def launched(monkeypatch):
    calls = []
    monkeypatch.setattr(ops, "lib", lambda: types.SimpleNamespace(citlali_dense_layer=lambda *a: calls.append(a) or 0))
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda device: 148)
    with FakeTensorMode():
        yield calls


_TYPED = ("qkv", "o", "gate_up", "down", "k_gain", "inv_freq", "keys", "values", "page_table", "x", "s_qkv", "s_heads", "s_act", "row_slot",
          "row_pos", "seq_start", "seq_slot", "seq_past", "in_rows", "in_sums", "mid_rows", "mid_sums", "out_rows", "out_sums")
_OTHER = {torch.int32: torch.int64, torch.bfloat16: torch.float32, torch.float32: torch.bfloat16}
_CHANGES = {
    "short": (lambda t: t.new_empty((t.shape[0] - 1,) + tuple(t.shape[1:])),
              ("qkv", "o", "gate_up", "down", "inv_freq", "x", "s_qkv", "s_heads", "s_act", "in_rows", "in_sums", "mid_rows", "mid_sums",
               "out_rows", "out_sums")),
    "narrow": (lambda t: t.new_empty(t.shape[0], t.shape[1] - 1), ("s_qkv", "s_heads", "s_act", "in_sums", "mid_sums", "out_sums", "out_rows")),
    "type": (lambda t: t.to(_OTHER[t.dtype]), _TYPED),
    "place": (lambda t: torch.empty(t.shape, dtype=t.dtype, device="cpu"), _TYPED + ("q_gain", "error_flag")),
    "apart": (lambda t: t.new_empty(tuple(t.shape) + (2,))[..., 0], _TYPED + ("q_gain", "error_flag")),
}


@pytest.mark.parametrize("what, name", [(w, n) for w, (_, names) in _CHANGES.items() for n in names])
def test_a_tensor_that_does_not_fit_is_refused(launched, what, name):
    a = _given()
    a[name] = _CHANGES[what][0](a[name])
    with pytest.raises(CitlaliError):
        _call(a)
    assert not launched


@pytest.mark.filterwarnings("ignore:Accessing the data pointer")
@pytest.mark.parametrize("gains", ["both", "none", "float32"])
def test_what_fits_reaches_the_kernels(launched, gains):
    a = _given()
    if gains != "both":
        a["q_gain"], a["k_gain"] = (None, None) if gains == "none" else (a["q_gain"].float(), a["k_gain"].float())
    _call(a)
    (args,) = launched
    with open(os.path.join(build._HERE, "api.h")) as fh:                # the structure as the header declares it
        body = re.search(r"typedef struct \{([^}]*)\} CitlaliDenseLayer;", re.sub(r"//[^\n]*", "", fh.read())).group(1)
    fields = [(name.strip("* "), "P" if "*" in name else "if"["float" in line])
              for line in body.split(";") if line.strip() for name in re.sub(r"^\s*(const )?\w+", "", line).split(",")]
    given = dict(zip((n.strip() for n, _ in fields), struct.unpack("@" + "".join(k for _, k in fields) + "0P", args[0])))
    want = dict(gain_dtype=int(gains == "both"), rotary_dim=D, page_table_stride=3, pool_pages=3, page_size=64, hidden=HIDDEN, inter=INTER, nq=NQ,
                nkv=NKV, head_dim=D, window=0)
    assert {k: given[k] for k in want} == want and given["scale"] == 0.25 and args[16:19] == (ROWS, 2, ROWS - 2)
