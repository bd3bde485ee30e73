"""A layer from one call against its launches one by one, with the options that its parts may have."""
import copy
import types

import pytest
import torch

import citlali_b200 as cb
from citlali_b200 import ops
from citlali_b200.engine.step import StepEntry
from citlali_b200.parts.block import PreNormResidualBlock

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _dense_config(d, heads, kv):
    return cb.config_from_dict(dict(
        architectures=["Qwen3ForCausalLM"], num_hidden_layers=3, hidden_size=256, num_attention_heads=heads, num_key_value_heads=kv,
        head_dim=d, intermediate_size=352, vocab_size=500, rope_theta=1e4, rms_norm_eps=1e-6, tie_word_embeddings=True,
        max_position_embeddings=512))


def _one_call_against_launches_one_by_one(config, lengths, calls_wanted, monkeypatch, stored_dtype="bfloat16"):
    """Two steps of ``lengths`` new tokens a sequence, the layers from one call each and then launch by launch: the same bits."""
    session = cb.InferenceSession().load_random(config, seed=3, max_context=400, dtype="bfloat16", device=DEV, max_batch=len(lengths),
                                                gain_spread=0.1, stored_dtype=stored_dtype)
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
    assert len(calls) == calls_wanted
    monkeypatch.setattr(PreNormResidualBlock, "_from_one_call", lambda *a: False)
    want = steps()
    session.check_device_errors()
    assert len(calls) == calls_wanted and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("option", ["window", "no head norms", "gains of 32 bits", "part of the head turned", "unequal inner widths"])
def test_a_layer_from_one_call_with_each_option_of_its_parts(d, option, monkeypatch):
    """Windows shorter than what is cached (one run on the tcgen05 attention for heads of 128), no gains, gains in float32, a rotation of
    part of a head, and scratch rows that two layers of a step need in different widths."""
    spec = copy.deepcopy(_dense_config(d, 4, 2).to_model_spec())
    for i, layer in enumerate(spec.layers):
        mixer = layer.parts["mixer"].params
        if option == "window":
            mixer["window"] = (20, 57, None)[i]
        elif option == "no head norms":
            mixer["qk_norm_eps"] = None
        elif option == "part of the head turned":
            mixer["position"]["rotary_dim"] = d // 4 * (i + 1)
        elif option == "unequal inner widths":
            layer.parts["feed_forward"].params["intermediate_size"] = (352, 96, 352)[i]
    _one_call_against_launches_one_by_one(types.SimpleNamespace(to_model_spec=lambda: spec), (60, 33, 2), 6, monkeypatch,
                                          stored_dtype="float32" if option == "gains of 32 bits" else "bfloat16")
