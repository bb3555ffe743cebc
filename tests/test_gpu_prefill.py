"""A prompt through native blocks against the same model run module by module: the same bits."""
import pytest
import torch

from ttcd_b200 import _native as nv
from ttcd_b200.models import IPTTCDv9Config, IPTTCDv9ForCausalLM, TransformerConfig, TransformerForCausalLM, prefill
from ttcd_b200.models.decoding import pack_projection_weights
from ttcd_b200.models.layers import WindowKVCache

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _model(heads, kv_heads, dim, hidden, inter, window, qk_norm, ttt_layers=(), family="ipttcd"):
    torch.manual_seed(heads + dim)
    cfg = dict(hidden_size=hidden, num_hidden_layers=3, num_heads=heads, num_kv_heads=kv_heads, head_dim=dim, intermediate_size=inter,
               vocab_size=512, window_size=window, max_position_embeddings=64, qk_norm=qk_norm, tie_word_embeddings=False)
    if family == "transformer":
        cfg.pop("head_dim")
        return TransformerForCausalLM(TransformerConfig(**cfg)).to(DEV, torch.bfloat16).eval()
    cfg.update(ttt_mode=bool(ttt_layers), ttt_layers=list(ttt_layers), ttt_chunk=128)
    return IPTTCDv9ForCausalLM(IPTTCDv9Config(**cfg)).to(DEV, torch.bfloat16).eval()


@torch.no_grad()
def _run(model, ids, native, monkeypatch, cache=True):
    calls = []
    with monkeypatch.context() as m:
        if native:
            inner = prefill.PlainBlocks.__call__
            m.setattr(prefill.PlainBlocks, "__call__", lambda self, block, x: (calls.append(out := inner(self, block, x)), out)[1])
        else:
            m.setattr(prefill, "plain_blocks", lambda *a: None)
        past = WindowKVCache() if cache else None
        out = model(input_ids=ids, past_key_values=past, use_cache=cache)
    return out.logits, [] if past is None else [t for kv in past.layers.values() for t in kv], [c is not None for c in calls]


@pytest.mark.parametrize("batch,seq,heads,kv_heads,dim,hidden,inter,window,qk_norm,packed", [
    (1, 128, 4, 2, 128, 256, 384, 64, True, False), (2, 301, 4, 4, 64, 192, 520, None, False, False), (1, 777, 3, 1, 64, 264, 1000, 200, True, True),
    (3, 131, 8, 2, 64, 512, 128, 4096, False, True)])
def test_native_blocks_match_the_modules(batch, seq, heads, kv_heads, dim, hidden, inter, window, qk_norm, packed, monkeypatch):
    model = _model(heads, kv_heads, dim, hidden, inter, window, qk_norm)
    if packed:
        pack_projection_weights(model)
    ids = torch.randint(0, 512, (batch, seq), device=DEV)
    for cache in (True, False):
        got, kv, ran = _run(model, ids, True, monkeypatch, cache)
        want, kv_want, _ = _run(model, ids, False, monkeypatch, cache)
        assert ran == [True] * 3 and torch.equal(got, want)
        assert len(kv) == len(kv_want) and all(torch.equal(a, b) for a, b in zip(kv, kv_want))


def test_fast_weight_blocks_and_other_families_take_their_own_way(monkeypatch):
    model = _model(4, 2, 64, 256, 256, 128, True, ttt_layers=(1,))
    for seq, want_ran in ((300, [True, False, True]), (127, [])):        # 127: no tile of queries; the fast-weight layer needs a chunk
        ids = torch.randint(0, 512, (1, seq), device=DEV)
        got, kv, ran = _run(model, ids, True, monkeypatch)
        want, kv_want, _ = _run(model, ids, False, monkeypatch)
        assert ran == want_ran and torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(kv, kv_want))
    model = _model(4, 4, 64, 256, 512, 256, False, family="transformer")
    ids = torch.randint(0, 512, (2, 200), device=DEV)
    assert _run(model, ids, True, monkeypatch)[2] == [True] * 3
    assert torch.equal(_run(model, ids, True, monkeypatch)[0], _run(model, ids, False, monkeypatch)[0])
    with torch.no_grad():                                                # a second call on a filled cache: the modules
        past = WindowKVCache()
        model(input_ids=ids, past_key_values=past, use_cache=True)
        with monkeypatch.context() as m:
            m.setattr(nv, "call", lambda symbol, *a, _c=nv.call: (_ for _ in ()).throw(AssertionError(symbol)) if symbol == "ttcd_block_prefill" else _c(symbol, *a))
            model(input_ids=ids, past_key_values=past, use_cache=True)


@pytest.mark.parametrize("seq", [300, 700, 9000, 13000])
def test_weights_that_leave_narrow_tiles_only(seq, monkeypatch):
    """q|k|v of 960 + 320 + 320 columns: from three matrices, over one and several tiles per CTA, or copied side by side (13000 rows)."""
    model = _model(15, 5, 64, 960, 256, 4096, False)
    ids = torch.randint(0, 512, (1, seq), device=DEV)
    got, kv, ran = _run(model, ids, True, monkeypatch)
    want, kv_want, _ = _run(model, ids, False, monkeypatch)
    assert ran == [True] * 3 and torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(kv, kv_want))


@pytest.mark.parametrize("seq,inter,ttt_layers", [(20000, 1536, (1,)), (20000, 512, ()), (9000, 1536, (2,))])
def test_a_prompt_takes_no_more_memory_than_its_modules(seq, inter, ttt_layers, monkeypatch):
    model = _model(8, 4, 64, 512, inter, 4096, True, ttt_layers=ttt_layers)
    ids = torch.randint(0, 512, (1, seq), device=DEV)
    peak = []
    for native in (True, False):
        with monkeypatch.context() as m, torch.no_grad():
            if not native:
                m.setattr(prefill, "plain_blocks", lambda *a: None)
            model(input_ids=ids[:, :256], logits_to_keep=1)         # (what stays: rotary tables)
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            torch.cuda.reset_peak_memory_stats()
            at = torch.cuda.memory_allocated()
            model(input_ids=ids, logits_to_keep=1)
            peak.append(torch.cuda.max_memory_allocated() - at)
    assert peak[0] <= 1.02 * peak[1], peak


@pytest.mark.parametrize("seq", [128, 300, 511, 512])
def test_a_fast_weight_block_below_its_chunk_is_a_plain_one(seq, monkeypatch):
    """What every chat-sized prompt of the shipped models is (chunks of 4096)."""
    model = _model(4, 2, 64, 256, 384, 256, True, ttt_layers=(1,))
    model.model.layers[1].ttt_chunk = model.model.layers[1].mlp.ttt_chunk = 512
    ids = torch.randint(0, 512, (2, seq), device=DEV)
    got, kv, ran = _run(model, ids, True, monkeypatch)
    want, kv_want, _ = _run(model, ids, False, monkeypatch)
    assert ran == [True, seq < 512, True] and torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(kv, kv_want))
