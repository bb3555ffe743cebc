"""Which models a decode step may bypass the modules of: the stock ones, and none of whose parts a program has replaced."""
import struct
import subprocess
import sys
from pathlib import Path
from types import MethodType, SimpleNamespace

import pytest
import torch
import torch.nn as nn

from ttcd_b200 import ops
from ttcd_b200.models import IPTTCDv9Config, IPTTCDv9ForCausalLM, layers
from ttcd_b200.models.base import DecoderForCausalLM
from ttcd_b200.models.decoding import GraphDecoder, pack_projection_weights
from ttcd_b200.models.layers import GatedMLP


class _ReluMLP(GatedMLP):
    def features(self, x):
        return torch.relu(ops.linear(x, self.gate_proj.weight)) * ops.linear(x, self.up_proj.weight)


class _ScaledLogits(IPTTCDv9ForCausalLM):
    def forward(self, *args, **kwargs):
        out = super().forward(*args, **kwargs)
        out.logits = 0.5 * out.logits
        return out


class _HalfEmbedding(nn.Embedding):
    def forward(self, ids):
        return 0.5 * super().forward(ids)


class _Doubled(nn.Module):
    def forward(self, w):
        return 2 * w


def _model(cls=IPTTCDv9ForCausalLM):
    torch.manual_seed(0)
    model = cls(IPTTCDv9Config(hidden_size=128, num_hidden_layers=2, num_heads=2, num_kv_heads=1, head_dim=64, intermediate_size=256,
                               vocab_size=64, window_size=32, ttt_mode=True, ttt_chunk=8, ttt_layers=[1], qk_norm=True,
                               tie_word_embeddings=False)).to(torch.bfloat16).eval()
    pack_projection_weights(model)
    return model


def _fused(model):
    return GraphDecoder._fused_weights(SimpleNamespace(model=model), 2)


def _replace_mlp(model):
    old = model.model.layers[1].mlp
    new = _ReluMLP(128, 256).to(torch.bfloat16).eval()
    for name in ("gate_proj", "up_proj", "down_proj"):
        setattr(new, name, getattr(old, name))
    model.model.layers[1].mlp = new


def _replace_embedding(model):
    model.model.embeddings = _HalfEmbedding.from_pretrained(model.model.embeddings.weight.data)


def _replace_method(path, name):
    def change(model):
        module = model.get_submodule(path)
        original = getattr(module, name)
        setattr(module, name, MethodType(lambda self, *a, **k: original(*a, **k), module))
    return change


CHANGES = {
    "mlp_of_another_kind": _replace_mlp,
    "embedding_of_another_kind": _replace_embedding,
    "mlp_forward_replaced": _replace_method("model.layers.0.mlp", "forward"),
    "mlp_features_replaced": _replace_method("model.layers.0.mlp", "features"),
    "attention_finish_replaced": _replace_method("model.layers.1.attn", "finish"),
    "norm_forward_replaced": _replace_method("model.layers.1.mlp_norm", "forward"),
    "model_forward_replaced": _replace_method("model", "forward"),
    "hook_on_a_block": lambda model: model.model.layers[0].register_forward_hook(lambda *a: None),
    # the weight would be read while the launch that makes it still runs
    "computed_weight": lambda model: nn.utils.parametrize.register_parametrization(model.model.layers[0].attn.o_proj, "weight", _Doubled()),
}


def test_the_stock_model_is_fused():
    assert len(_fused(_model())) == 2


@pytest.mark.parametrize("change", list(CHANGES))
def test_a_changed_model_runs_its_modules(change):
    model = _model()
    CHANGES[change](model)
    assert _fused(model) is None


def test_a_model_with_its_own_forward_runs_it():
    assert _fused(_model(_ScaledLogits)) is None


def test_hooks_on_all_modules_are_run():
    model = _model()
    handle = nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert _fused(model) is None
    finally:
        handle.remove()
    assert _fused(model) is not None


def test_a_tensor_parallel_state_runs_the_modules(monkeypatch):
    model = _model()
    monkeypatch.setattr(layers, "_tp_state", lambda: SimpleNamespace(world=2))
    assert _fused(model) is None


def _plain(model):
    """Which blocks a prompt would run natively (the rule itself needs no GPU)."""
    from ttcd_b200.models.prefill import PlainBlocks
    runner = PlainBlocks(torch.zeros(1, 300, 128, dtype=torch.bfloat16), None)
    return [runner._tensors(block) is not None for block in model.model.layers]


def test_the_stock_blocks_run_natively_but_for_the_fast_weight_one():
    assert _plain(_model()) == [True, False]


@pytest.mark.parametrize("change", ["mlp_forward_replaced", "mlp_features_replaced", "hook_on_a_block", "computed_weight"])
def test_a_changed_block_runs_its_modules_over_a_prompt(change):
    model = _model()
    CHANGES[change](model)
    assert _plain(model) == [False, False]


def test_a_method_replaced_on_a_class_is_run_over_a_prompt(monkeypatch):
    model = _model()
    assert _plain(model) == [True, False]
    monkeypatch.setattr(GatedMLP, "features", lambda self, x: x)
    assert _plain(model) == [False, False]


BEFORE_THE_FIRST_PROMPT = """
import torch
from ttcd_b200.models import layers, modeling_ipttcdv9
cls = {"GatedMLP": layers.GatedMLP, "IPTTCDBlock": modeling_ipttcdv9.IPTTCDBlock}["%s"]
inner = cls.%s
cls.%s = lambda self, *a, **k: inner(self, *a, **k)
from tests.test_fused_decode_rule import _fused, _model, _plain
model = _model()
assert not any(_plain(model)), "a prompt"
assert _fused(model) is None, "a decode step"
"""


@pytest.mark.parametrize("cls,method", [("GatedMLP", "features"), ("IPTTCDBlock", "forward")])
def test_a_method_replaced_on_a_class_before_the_first_prompt_is_run(cls, method):
    """In a process of its own: import, replace, run."""
    root = Path(__file__).resolve().parents[1]
    done = subprocess.run([sys.executable, "-c", BEFORE_THE_FIRST_PROMPT % (cls, method, method)], cwd=root, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr[-2000:]


def test_a_model_class_with_another_forward_runs_it_in_every_decode_step(monkeypatch):
    model = _model()
    inner = DecoderForCausalLM.forward
    monkeypatch.setattr(DecoderForCausalLM, "forward", lambda self, *a, **k: inner(self, *a, **k))
    assert _fused(model) is None


def _with_linears(path, **widths):
    """Modules of other extents in the place of the stock ones, the attributes left as they were."""
    def change(model):
        parent = model.get_submodule(path)
        for name, (n_in, n_out) in widths.items():
            setattr(parent, name, nn.Linear(n_in, n_out, bias=False).to(torch.bfloat16))
    return change


@pytest.mark.parametrize("change", [
    _with_linears("model.layers.0.mlp", gate_proj=(128, 128), up_proj=(128, 128), down_proj=(128, 128)),        # a pruned MLP
    _with_linears("model.layers.0.mlp", up_proj=(128, 264)),
    _with_linears("model.layers.0.attn", k_proj=(128, 128), v_proj=(128, 128)),
    _with_linears("model.layers.0.attn", o_proj=(64, 128)),
    lambda model: setattr(model.model.layers[0].attn, "q_norm", layers.RMSNorm(32).to(torch.bfloat16)),
    lambda model: setattr(model.model.layers[0], "mlp_norm", layers.RMSNorm(64).to(torch.bfloat16)),
    lambda model: setattr(model.model.layers[0].mlp, "intermediate_size", 512)])
def test_a_block_with_weights_of_other_extents_runs_its_modules_over_a_prompt(change):
    model = _model()
    change(model)
    assert _plain(model) == [False, False]


def test_a_pruned_mlp_still_works():
    model = _model()
    ids = torch.arange(40).view(1, 40) % 64
    _with_linears("model.layers.0.mlp", gate_proj=(128, 64), up_proj=(128, 64), down_proj=(64, 128))(model)
    with torch.no_grad():
        assert model(input_ids=ids).logits.isfinite().all()


@pytest.mark.parametrize("table", [(200, 32), (300, 33), (300, 64)])
def test_a_rotary_table_that_does_not_cover_the_prompt_is_left_to_the_modules(table, monkeypatch):
    from ttcd_b200.models import prefill
    model = _model()
    block = model.model.layers[0]
    monkeypatch.setattr(prefill.nv, "call", lambda *a: pytest.fail("launched"))
    monkeypatch.setattr(block.attn.rotary, "tables", lambda *a: (torch.zeros(table, dtype=torch.bfloat16),) * 2)
    x = torch.zeros(1, 300, 128, dtype=torch.bfloat16)
    assert prefill.PlainBlocks(x, None)(block, x) is None


@pytest.mark.parametrize("change", [lambda x: x[:, ::2].contiguous(), lambda x: x.float(), lambda x: x[..., :64].contiguous(), lambda x: (x, None)])
def test_what_another_block_hands_on_is_looked_at_before_every_block(change, monkeypatch):
    """A hook on a block may drop tokens, or change the type; the blocks that follow must not go by the prompt's extents."""
    from ttcd_b200.models import prefill
    monkeypatch.setattr(prefill.nv, "call", lambda *a: pytest.fail("launched"))
    model = _model()
    x = torch.zeros(1, 300, 128, dtype=torch.bfloat16)
    runner = prefill.PlainBlocks(x, None)
    assert runner(model.model.layers[0], change(x)) is None


def _one_projection(model):
    """q, k and v from one linear of the program's own, the three taken out."""
    attn = model.model.layers[0].attn
    attn.qkv_proj = nn.Linear(128, 256, bias=False).to(torch.bfloat16)
    for name in ("q_proj", "k_proj", "v_proj"):
        delattr(attn, name)
    attn.project_qkv = MethodType(lambda self, x, *a, **k: tuple(t.unflatten(-1, (-1, 64)) for t in self.qkv_proj(x).split((128, 64, 64), -1)), attn)


def _no_norm(model):
    block = model.model.layers[0]
    del block.mlp_norm
    block.forward = MethodType(lambda self, x, *a, **k: x + self.mlp(self.attn_norm(x)), block)


@pytest.mark.parametrize("change", [_one_projection, _no_norm])
def test_a_block_without_a_stock_part_runs_its_modules_over_a_prompt(change):
    model = _model()
    change(model)
    assert _plain(model) == [False, False]
    with torch.no_grad():
        assert model(input_ids=torch.arange(40).view(1, 40) % 64, use_cache=False).logits.isfinite().all()


def test_scratch_of_native_blocks_is_given_back_to_a_block_that_runs_its_modules(monkeypatch):
    from ttcd_b200.models import prefill
    launches = []
    monkeypatch.setattr(prefill.nv, "call", lambda symbol, record, *a: launches.append(struct.unpack("34q", record)))
    monkeypatch.setattr(prefill.nv, "stream_ptr", lambda: None)
    plain, fast_weight = _model().model.layers
    x = torch.zeros(1, 300, 128, dtype=torch.bfloat16)
    runner = prefill.PlainBlocks(x, None)
    assert runner(plain, x) is not None and runner.scratch
    assert runner(fast_weight, x) is None and not runner.scratch
    # one piece of memory: the sum lies over q, which is done with by then, o behind both, the MLP's features behind the sum
    q, o, total, z = (launches[0][i] for i in (5, 7, 9, 10))
    assert total == q and o == q + 300 * 128 * 2 and z == total + 300 * 128 * 2
