"""The work that users of this framework have it do, as timed cases.

Four kinds of work, each through the calls that a user's program makes:

* ``train``   one optimizer step (``TrainEngine.train_step``): forward, backward, clip, AdamW (or Muon + AdamW);
* ``prefill`` a whole model over a prompt: with the key/value cache and the last position's logits (``cache``: what precedes
  generation), or all positions' logits (``score``: perplexity evaluation);
* ``decode``  greedy decoding of a number of tokens after a prompt (``GraphDecoder``: what ``generate`` runs);
* ``attn``    dual-window attention on its own (``ops.dual_window_attention``), forward or forward and backward.

Widths, head counts, windows and vocabularies are those of the shipped model configurations.  Training cases keep one
period of the layer pattern (a fast-weight layer and the plain layers up to the next one), so that the mix of work is the
full model's while a step stays short; prefill and decoding run every layer.
"""
from __future__ import annotations

import math

import torch

from ttcd_b200 import ops
from ttcd_b200.models import decoding
from ttcd_b200.models.layers import WindowKVCache
from ttcd_b200.train.engine import EngineConfig, TrainEngine, build_model, load_model_config

QWEN = "configs/ipttcd/ipttcdv9_qwen3_0.6B_ct_64k_v2_swa8k.json"
LLAMA = "configs/ipttcd/ipttcdv9_llama32_1B_ct_64k_v2_fullattn.json"
SCRATCH = "configs/ipttcd/ipttcdv9_340M_swa_teacher_student_causalconv.json"
DELTA = "configs/delta_net/delta_net_340M.json"
GATED = "configs/gated_deltanet/gated_deltanet_340M.json"

PERIOD = {QWEN: 7, LLAMA: 5, SCRATCH: 6, DELTA: 3, GATED: 3}       # layers of a training case


def listed() -> list[dict]:
    train = lambda name, config, batch, seq, ac="none", muon=False: dict(      # noqa: E731
        name=name, kind="train", config=config, layers=PERIOD[config], batch=batch, seq=seq, ac=ac, muon=muon)
    return [
        # continued training at 64K context, one sequence per GPU: the recipe the framework is built for
        train("train_qwen_64k", QWEN, 1, 65536),
        # from-scratch pretraining of the 340M model with Muon: short sequences, many of them
        train("train_340m_muon", SCRATCH, 8, 4096, muon=True),
        # continued training of the 1B model (full attention, head_dim 64, grouped 32/8) on one document of its own
        # length, every block recomputed in backward as the recipe has it
        train("train_llama_ragged", LLAMA, 1, 5003, ac="full"),
        # the two delta-rule baselines
        train("train_delta_net", DELTA, 4, 4096),
        train("train_gated_deltanet", GATED, 2, 3001),
        # a long document read before generation, and a chat-sized prompt (latency: launches and small tiles)
        dict(name="prefill_qwen_64k", kind="prefill", config=QWEN, batch=1, seq=65536, mode="cache"),
        dict(name="prefill_qwen_short", kind="prefill", config=QWEN, batch=1, seq=300, mode="cache"),
        # perplexity of a few documents: every position's logits
        dict(name="score_llama", kind="prefill", config=LLAMA, batch=3, seq=2345, mode="score"),
        # greedy generation for one user after a long prompt, and for a batch of eight after shorter ones
        dict(name="decode_one", kind="decode", config=QWEN, batch=1, prompt=9000, tokens=32),
        dict(name="decode_eight", kind="decode", config=QWEN, batch=8, prompt=1500, tokens=32),
        # the dual-window kernel on its own: the prefill microbenchmark's shape, and a training call on an odd length
        # at head_dim 64
        dict(name="attn_32k", kind="attn", batch=1, seq=32768, heads=16, kv_heads=8, dim=128, w_t=8192, w_s=4096,
             backward=False),
        dict(name="attn_d64_bwd", kind="attn", batch=2, seq=10007, heads=15, kv_heads=5, dim=64, w_t=8192, w_s=4096,
             backward=True),
    ]


def _spread(rng, lo: int, hi: int, multiple: int = 1) -> int:
    """Log-uniform whole number of [lo, hi], of a multiple if asked."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v // multiple * multiple))


def draw(rng) -> dict:
    kind = rng.choice(["train", "train", "train", "prefill", "prefill", "decode", "decode", "attn", "attn"])
    if kind == "train":
        config = rng.choice([QWEN, LLAMA, SCRATCH, DELTA, GATED])
        most = {QWEN: 65536, LLAMA: 24000, SCRATCH: 4096, DELTA: 4096, GATED: 4096}[config]
        multiple = rng.choice([1, 1, 512])
        seq = _spread(rng, 600, most, multiple)
        total = 32768 if config in (QWEN, LLAMA, SCRATCH) else 12288
        batch = rng.randint(1, max(1, min(8, total // seq)))
        return dict(kind="train", config=config, layers=PERIOD[config], batch=batch, seq=seq,
                    ac=rng.choice(["none", "none", "full"]), muon=bool(config == SCRATCH and rng.random() < 0.5))
    if kind == "prefill":
        config, mode = rng.choice([(QWEN, "cache"), (QWEN, "cache"), (LLAMA, "score")])
        seq = _spread(rng, 130, 65536 if mode == "cache" else 4096)
        return dict(kind="prefill", config=config, mode=mode, seq=seq, batch=rng.randint(1, max(1, min(4, 8192 // seq))))
    if kind == "decode":
        return dict(kind="decode", config=QWEN, batch=_spread(rng, 1, 16), prompt=_spread(rng, 200, 12000),
                    tokens=rng.randint(16, 48))
    heads, kv_heads, dim = rng.choice([(16, 8, 128), (15, 5, 64), (16, 16, 64)])
    backward = rng.random() < 0.5
    w_t = rng.choice([2048, 4096, 8192])
    seq = _spread(rng, 1000, 65536 if not backward else 24000)
    return dict(kind="attn", batch=rng.randint(1, max(1, min(4, 32768 // seq))), seq=seq, heads=heads, kv_heads=kv_heads,
                dim=dim, w_t=w_t, w_s=w_t // 2, backward=backward)


# ------------------------------------------------------------------------------------------------ state
def _config(case):
    over = {}
    if case["kind"] == "train":
        over["num_hidden_layers"] = case["layers"]
    if case["kind"] == "decode":
        over["tie_word_embeddings"] = False
    cfg = load_model_config(case["config"], **over)
    cfg.max_position_embeddings = max(cfg.max_position_embeddings or 0, case.get("seq", 0) + 64)
    return cfg


@torch.no_grad()
def _trained_like(model, gen, decides: bool = False) -> None:
    """What a trained model has and a fresh one lacks.  Fast-weight layers start with a zero student convolution, which
    switches the update off; ``decides``: the next token stands out from the rest (each token asks for one other token),
    so that greedy decoding does not hang on the last bit of the logits."""
    for name, p in model.named_parameters():
        if name.endswith("ttt_student_conv.weight"):
            p.copy_(0.1 * torch.randn(p.shape, generator=gen, device=p.device))
            p[:, :, -1] += 1.0
    if decides:
        table = model.model.embeddings.weight
        model.lm_head.weight.copy_(table[torch.randperm(table.shape[0], generator=gen, device=table.device)])
        table.mul_(50.0)


def _ids(case, cfg, gen, batch, seq):
    return torch.randint(0, cfg.vocab_size, (batch, seq), generator=gen, device="cuda")


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "attn":
        mk = lambda h: torch.randn(case["batch"], case["seq"], h, case["dim"], device="cuda", generator=gen,    # noqa: E731
                                   dtype=torch.bfloat16)
        q, k, v = mk(case["heads"]), mk(case["kv_heads"]), mk(case["kv_heads"])
        state = dict(case=case, qkv=(q, k, v))
        if case["backward"]:
            state["grads"] = (mk(case["heads"]), mk(case["heads"]))
            for t in state["qkv"]:
                t.requires_grad_()
        return state
    cfg = _config(case)
    if case["kind"] == "train":
        # the learning rate of the recipe's first warm-up step
        engine = TrainEngine(cfg, EngineConfig(lr=1e-7, activation_checkpoint=case["ac"], enable_muon=case["muon"],
                                               seed=seed), device="cuda")
        _trained_like(engine.model, gen)
        engine.sdp.resync_master()
        return dict(case=case, engine=engine, ids=_ids(case, cfg, gen, case["batch"], case["seq"]))
    model = build_model(cfg, "cuda", torch.bfloat16, seed=seed).eval()
    _trained_like(model, gen, decides=case["kind"] == "decode")
    if case["kind"] == "prefill":
        return dict(case=case, model=model, ids=_ids(case, cfg, gen, case["batch"], case["seq"]))
    # decoding: what generate() has in hand after the prompt
    cache = WindowKVCache()
    with torch.no_grad():
        out = model(input_ids=_ids(case, cfg, gen, case["batch"], case["prompt"]), past_key_values=cache, use_cache=True,
                    logits_to_keep=1)
    first = out.logits[:, -1].float().argmax(-1, keepdim=True)
    return dict(case=case, model=model, cache=cache, first=first, decoder=decoding.decoder_for(model, cache, case["tokens"]))


# ------------------------------------------------------------------------------------------------ one pass
def run(state: dict):
    case = state["case"]
    if case["kind"] == "train":
        engine = state["engine"]
        loss = engine.train_step(state["ids"], return_loss_on_host=False)
        params = list(engine.model.parameters())
        # every parameter's gradient, or, for the deeper models, the flat buffers (one per block) that hold them
        grads = [p.grad for p in params] if len(params) <= 56 else [g.flat_grad for g in engine.sdp.groups]
        return dict(loss=loss, grads=grads, weights=[g.flat_param for g in engine.sdp.groups])
    if case["kind"] == "prefill":
        with torch.no_grad():
            if case["mode"] == "score":
                return state["model"](input_ids=state["ids"], use_cache=False).logits
            out = state["model"](input_ids=state["ids"], use_cache=True, logits_to_keep=1)
        return dict(logits=out.logits, cache=[kv for kv in out.past_key_values.layers.values()])
    if case["kind"] == "decode":
        decoder = state["decoder"]
        decoder.load(state["cache"])
        tokens = decoder.run(state["first"], case["tokens"], set())
        return dict(tokens=tokens, logits=decoder.last_logits, cache=[kv for kv in decoder.cache.layers.values()])
    q, k, v = state["qkv"]
    if not case["backward"]:
        with torch.no_grad():
            return ops.dual_window_attention(q, k, v, case["w_t"], case["w_s"])
    outs = ops.dual_window_attention(q, k, v, case["w_t"], case["w_s"])
    grads = torch.autograd.grad(outs, (q, k, v), state["grads"])
    return dict(outs=outs, grads=grads)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _pairs(seq: int, window) -> float:
    """Visible (query, key) pairs of one causal row with a window."""
    w = seq if window is None else min(window, seq)
    return w * (w + 1) / 2 + (seq - w) * w


def _model_terms(cfg, batch, seq):
    """(parameters, forward flops of one pass without the head, key/value values per token)."""
    d, tokens = cfg.hidden_size, batch * seq
    inter = cfg.resolved_intermediate_size
    flops, params, kv = 0.0, 0.0, 0.0
    for i in range(cfg.num_hidden_layers):
        params += 3 * d * inter
        flops += 2.0 * tokens * 3 * d * inter
        if cfg.model_type in ("delta_net", "gated_deltanet"):
            gated = cfg.model_type == "gated_deltanet"
            heads = cfg.num_heads
            dk = cfg.head_dim if gated else d // heads
            dv = int(dk * cfg.expand_v) if gated else d // heads
            proj = d * heads * (2 * dk + (2 if gated else 1) * dv) + heads * dv * d
            # per token and head: the recurrence reads and writes one [dk, dv] state (three products of 2 dk dv flops)
            flops += 2.0 * tokens * proj + tokens * heads * 6.0 * dk * dv
            params += proj
            continue
        hd = cfg.head_dim or d // cfg.num_heads
        kvh = cfg.num_kv_heads or cfg.num_heads
        proj = d * hd * (2 * cfg.num_heads + 2 * kvh)
        ttt = i in set(cfg.ttt_layers) and seq >= cfg.ttt_chunk
        flops += 2.0 * tokens * proj + 4.0 * batch * cfg.num_heads * hd * _pairs(seq, cfg.window_size)
        params += proj
        kv += 2.0 * kvh * hd
        if ttt:         # student stream (o_proj, gate/up), the update's projection, outer product
            flops += 2.0 * tokens * (cfg.num_heads * hd * d + 2 * d * inter) + 4.0 * tokens * d * inter
            params += d * d
    return params, flops, kv


def work(case: dict) -> dict:
    if case["kind"] == "attn":
        b, t, h, hk, dim = (case[x] for x in ("batch", "seq", "heads", "kv_heads", "dim"))
        q, kv = 2.0 * b * t * h * dim, 2.0 * b * t * hk * dim
        flops = 4.0 * b * h * dim * _pairs(t, case["w_t"])        # one softmax pass serves both windows
        if not case["backward"]:
            return dict(bytes=q + 2 * kv + 2 * q, flops=flops)
        return dict(bytes=(q + 2 * kv + 2 * q) + (2 * q + q + 2 * kv), flops=3.5 * flops)
    cfg = _config(case)
    vocab = cfg.vocab_size * cfg.hidden_size
    if case["kind"] == "train":
        params, fwd, _ = _model_terms(cfg, case["batch"], case["seq"])
        tokens = case["batch"] * case["seq"]
        held = params + vocab * (1 if cfg.tie_word_embeddings else 2)
        # bf16 weights in, gradients out; master and two moments in and out, new bf16 weights out
        return dict(bytes=held * (2 + 2 + 2 * 12 + 2) + 8.0 * tokens, flops=3 * (fwd + 2.0 * tokens * vocab))
    if case["kind"] == "prefill":
        params, fwd, kv = _model_terms(cfg, case["batch"], case["seq"])
        tokens = case["batch"] * case["seq"]
        if case["mode"] == "score":
            return dict(bytes=2 * (params + vocab) + 2.0 * tokens * cfg.vocab_size, flops=fwd + 2.0 * tokens * vocab)
        kept = case["batch"] * min(case["seq"], cfg.window_size)
        return dict(bytes=2 * (params + vocab) + 2.0 * kept * kv, flops=fwd + 2.0 * case["batch"] * vocab)
    b, steps = case["batch"], case["tokens"]
    params, _, kv = _model_terms(cfg, 1, 1)
    rows = sum(min(case["prompt"] + i + 1, cfg.window_size) for i in range(steps))
    pair = 4.0 * cfg.num_hidden_layers * cfg.num_heads * cfg.head_dim
    filled = min(case["prompt"], cfg.window_size)
    # every token reads the weights and the filled window once; loading the prompt's rows reads and writes them once
    return dict(bytes=steps * 2 * (params + vocab) + 2.0 * b * kv * rows + 4.0 * b * kv * filled,
                flops=b * (steps * 2.0 * (params + vocab) + pair * rows))


def tolerance(case: dict):
    # measured: attention against float64: rel 0.0022 forward, 0.0031 backward (max 0.03 and 0.2).  Models with every GEMM
    # summed in another order (bf16 outputs, so each layer rounds again): gradients rel 0.008-0.017, max 0.34-0.85 (a
    # frequent token's row of the embedding); prefill rel 0.0076, max 0.14; decoding rel 0.015, max 0.08, same tokens
    if case["kind"] == "attn":
        return {"rel": 0.01, "max": 0.6}
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.99}
    return {"rel": 0.03, "max": 0.5, "differ": 0.01}
