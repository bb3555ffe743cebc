"""Greedy decoding as one captured CUDA graph per token.

Eager decoding of a 28-layer model issues over a thousand small launches per token and is bound by the host; the
device work of a step (one pass over the weights and the key/value windows) is a fraction of a millisecond.  The
decode step therefore runs through ``StaticWindowCache`` (fixed addresses, positions and fill counts on the device),
is captured once per (batch, ring capacities) and replayed per token: the next token is chosen on the device and fed
back without the host seeing it; the host reads the tokens once at the end (or every few steps when it has to look
for an end-of-sequence token).

The reference decodes eagerly through HF ``generate`` (custom_models/ipttcd/modeling_ipttcdv9.py:794-850 for the
model side: fast weights are built during prefill only, a decode step is the plain windowed transformer step).
"""
from __future__ import annotations

import torch

from .layers import Attention, GatedMLP, RMSNorm, StaticWindowCache, WindowKVCache, _slab_view


def pack_projection_weights(model) -> int:
    """Re-house q|k|v and gate|up weights of every block back to back in one buffer each, so that their projections
    run as ONE GEMM / GEMV without concatenating the weights per call.  Only touches weights that own their storage
    (a training runtime that keeps parameters as views of its flat buffers is left alone).  Returns how many groups
    were packed."""
    packed = 0
    for mod in model.modules():
        if isinstance(mod, Attention):
            group = [mod.q_proj, mod.k_proj, mod.v_proj]
        elif isinstance(mod, GatedMLP):
            group = [mod.gate_proj, mod.up_proj]
        else:
            continue
        ws = [lin.weight for lin in group]
        if any(lin.bias is not None for lin in group) or any(w.data._base is not None or not w.is_contiguous() for w in ws):
            continue
        if _slab_view(ws) is not None:      # (neighbours by chance, each in its own storage, are no slab)
            continue
        if len({(w.dtype, w.device, w.shape[1]) for w in ws}) != 1:
            continue
        slab = torch.cat([w.data for w in ws], dim=0)
        row = 0
        for w in ws:
            w.data = slab[row:row + w.shape[0]]
            row += w.shape[0]
        packed += 1
    return packed


def graph_decoding_supported(model, input_ids, attention_mask, do_sample: bool) -> bool:
    if do_sample or not input_ids.is_cuda or getattr(model.model, "cache_class", WindowKVCache) is not WindowKVCache:
        return False
    if attention_mask is not None and not bool(attention_mask.all()):
        return False
    if any(isinstance(m, Attention) and m.use_l2_softmax for m in model.modules()):
        return False
    from .. import _native
    return _native.available() and next(model.parameters()).dtype == torch.bfloat16


# what the fused step computes on behalf of the modules; a program may replace any of these on an instance
_STEP_METHODS = ("forward", "project_qkv", "finish", "features", "_block_kwargs")


def _as_defined(*modules) -> bool:
    """No hook and no method replaced on an instance: calling these modules does what their classes say."""
    from torch.nn.modules import module as hooks
    if hooks._global_forward_hooks or hooks._global_forward_pre_hooks:
        return False
    return not any(m._forward_hooks or m._forward_pre_hooks or any(name in vars(m) for name in _STEP_METHODS) for m in modules)


def _at_rest(linear) -> bool:
    """The weight is the module's own parameter and not made from others in every step (a parametrization)."""
    return linear._parameters.get("weight") is not None and linear.bias is None


def _fused_block_weights(block, batch: int):
    """The weights of a block whose decode step runs as six launches (``_fused_block_step``), or None where the step has
    to go through the modules: another kind of block or of a part of it, an option the step has no kernel for, a hook, a
    replaced method, a weight that is computed."""
    from .layers import _tp_state
    from .modeling_ipttcdv9 import IPTTCDBlock, IPTTCDMLP
    from .modeling_transformer import TransformerBlock
    from .stock import unchanged
    stock = unchanged()                 # (a method may have been replaced on a class)
    if type(block) not in stock & {IPTTCDBlock, TransformerBlock} or block.training or batch > 16 or _tp_state() is not None:
        return None
    if type(block) is IPTTCDBlock and block.is_ttt_layer and block.ttt_chunk <= 1:       # one token would be a whole chunk
        return None
    if not _as_defined(*block.modules()) or type(block.mlp) not in stock & {GatedMLP, IPTTCDMLP}:
        return None
    attn, mlp = block.attn, block.mlp
    if type(attn) is not Attention or not {Attention, RMSNorm} <= stock or attn.use_output_gate or attn.use_l2_softmax or attn.head_dim not in (64, 128):
        return None
    norms = [block.attn_norm, block.mlp_norm] + ([attn.q_norm, attn.k_norm] if attn.qk_norm else [])
    if any(type(n) is not RMSNorm or n.weight is None for n in norms):
        return None
    if not all(_at_rest(m) for m in (attn.q_proj, attn.k_proj, attn.v_proj, attn.o_proj, mlp.gate_proj, mlp.up_proj, mlp.down_proj)):
        return None
    qkv = _slab_view([attn.q_proj.weight, attn.k_proj.weight, attn.v_proj.weight])
    gate_up = _slab_view([mlp.gate_proj.weight, mlp.up_proj.weight])
    ws = [qkv, gate_up, attn.o_proj.weight, mlp.down_proj.weight, *(n.weight for n in norms)]
    hidden = attn.hidden_size
    if hidden % 8 or hidden > 2048 or mlp.intermediate_size % 8:
        return None
    if any(w is None or w.dtype != torch.bfloat16 or not w.is_contiguous() or w.data_ptr() % 16 for w in ws):
        return None
    return qkv, gate_up


def _fused_block_step(block, weights, x: torch.Tensor, cache: StaticWindowCache, turns: torch.Tensor) -> torch.Tensor:
    """One token per sample through a decoder block: x [B, hidden] -> x.  The norms ride in front of the projections that
    read them, SwiGLU and the residual sums behind the ones that produce them, k and v go straight into the rings; the
    roundings are those of the module by module step."""
    from .. import ops
    from ..ops import cuda
    attn, mlp, (qkv_w, gate_up_w) = block.attn, block.mlp, weights
    i = attn.layer_idx
    c = cache.capacity[i]
    rk, rv = cache.layers[i]
    cos = sin = None
    if not attn.use_nope:
        cos, sin = attn.rotary.tables(max(cache.max_position, attn.max_position_embeddings or 0), x.device, x.dtype)
    qw, kw, eps = (attn.q_norm.weight, attn.k_norm.weight, attn.q_norm.eps) if attn.qk_norm else (None, None, 0.0)
    qkv = cuda.gemv(x, qkv_w, norm=(block.attn_norm.weight, block.attn_norm.eps), early_w=True)
    q = cuda.decode_qkv(qkv, rk, rv, cache.slot[c], cache.positions, qw, kw, eps, cos, sin, attn.num_heads)
    o = ops.decode_attention(q, rk, rv, cache.kv_len[c], turns=turns)
    x = cuda.gemv(o.view(x.shape[0], -1), attn.o_proj.weight, residual=x, early_w=True)
    z = cuda.gemv(x, gate_up_w, norm=(block.mlp_norm.weight, block.mlp_norm.eps), swiglu=True, early_w=True)
    return cuda.gemv(z, mlp.down_proj.weight, residual=x, early_w=True)


def _windows(model) -> dict[int, int | None]:
    return {m.layer_idx: m.window_size for m in model.modules() if isinstance(m, Attention)}


class GraphDecoder:
    """One captured decode step of ``model`` over a ``StaticWindowCache``; ``run`` replays it."""

    def __init__(self, model, source: WindowKVCache, max_new_tokens: int):
        self.model = model
        pack_projection_weights(model)
        self.cache = StaticWindowCache(source, _windows(model), max_new_tokens)
        batch = self.cache.positions.shape[0]
        dev = self.cache.pos.device
        self.token = torch.zeros(batch, 1, dtype=torch.long, device=dev)
        self.steps_capacity = max_new_tokens
        self.out = torch.zeros(batch, max_new_tokens, dtype=torch.long, device=dev)
        self.cursor = torch.zeros(1, dtype=torch.int64, device=dev)
        self.weights_at = self._weights_at()
        self.fused = self._fused_weights(batch)
        heads = max(k.shape[2] for k, _ in self.cache.layers.values())
        self.turns = torch.zeros(batch * heads, dtype=torch.int32, device=dev)      # this decoder's merge counters
        self.pick = torch.zeros(8 * batch + 1, dtype=torch.int64, device=dev)
        start = self.cache.start
        # warm-up on a side stream (allocator pools, rotary tables, lazily configured kernels), then rewind and capture
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            self._step()
        torch.cuda.current_stream(dev).wait_stream(side)
        self.cache.reset(start)
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self._step()
        self.load(source)                       # the warm-up step overwrote the oldest row of every ring
        self.tables = [m.rotary._cached for m in model.modules() if isinstance(m, Attention) and not m.use_nope]

    def _weights_at(self):
        return (self.model.lm_head.weight.data_ptr(), next(self.model.model.layers[0].parameters()).data_ptr())

    def _fused_weights(self, batch: int):
        """Per block the weights of its fused step; None if any part of the model has to run module by module."""
        from .base import DecoderForCausalLM, DecoderModel
        from .stock import unchanged
        if not {DecoderForCausalLM, DecoderModel, RMSNorm} <= unchanged():
            return None
        model, core, head = self.model, self.model.model, self.model.lm_head
        if type(model).forward is not DecoderForCausalLM.forward or type(core).forward is not DecoderModel.forward:
            return None
        if type(core)._block_kwargs is not DecoderModel._block_kwargs or type(core.embeddings) is not torch.nn.Embedding:
            return None
        if not _as_defined(model, core, core.norm, core.embeddings, head) or not _at_rest(head):
            return None
        if head.weight.dtype != torch.bfloat16 or not head.weight.is_contiguous() or head.weight.data_ptr() % 16:
            return None
        got = [_fused_block_weights(layer, batch) for layer in core.layers]
        return None if any(w is None for w in got) else got

    def _logits(self) -> torch.Tensor:
        if self.fused is None:
            return self.model(input_ids=self.token, past_key_values=self.cache, use_cache=True, logits_to_keep=1).logits[:, -1]
        from ..ops import cuda
        core = self.model.model
        x = core.embeddings(self.token.view(-1))
        for layer, weights in zip(core.layers, self.fused):
            x = _fused_block_step(layer, weights, x, self.cache, self.turns)
        norm = core.norm
        if type(norm) is RMSNorm and norm.weight is not None and norm.weight.dtype == x.dtype and norm.weight.data_ptr() % 16 == 0:
            return cuda.gemv(x, self.model.lm_head.weight, norm=(norm.weight, norm.eps), early_w=True)
        return cuda.gemv(norm(x), self.model.lm_head.weight, early_w=True)

    @torch.no_grad()
    def _step(self) -> None:
        self.last_logits = self._logits()                # (kept for inspection; lives in the graph's pool)
        cache = self.cache
        if self.fused is not None and len(cache.slot) <= 4:
            from ..ops import cuda
            cuda.decode_pick(self.last_logits, self.token, self.out, self.cursor, cache.pos, cache.positions,
                             [(c, cache.slot[c], cache.kv_len[c]) for c in cache.slot], self.pick)
            return
        nxt = self.last_logits.float().argmax(-1, keepdim=True)
        self.token.copy_(nxt)
        self.out.index_copy_(1, self.cursor, nxt)
        self.cursor.add_(1)
        cache.advance()

    def fits(self, source: WindowKVCache, max_new_tokens: int) -> bool:
        """Whether a new prompt's cache can reuse this capture (same shapes, rings large enough, same weights)."""
        if self._weights_at() != self.weights_at or max_new_tokens > self.steps_capacity:
            return False
        seen = {source.seen[i] for i in source.layers}
        if len(seen) != 1 or set(source.layers) != set(self.cache.layers):
            return False
        start = seen.pop()
        if start + max_new_tokens > self.cache.max_position:
            return False
        windows = _windows(self.model)
        for i, (k, _v) in source.layers.items():
            rk = self.cache.layers[i][0]
            if k.shape[0] != rk.shape[0] or k.shape[2:] != rk.shape[2:] or k.dtype != rk.dtype:
                return False
            cap = self.cache.capacity[i]
            if (windows.get(i) is not None and cap != windows[i]) or k.shape[1] > cap:
                return False
            if windows.get(i) is None and start + max_new_tokens > cap:
                return False
        return True

    def load(self, source: WindowKVCache) -> None:
        """Copy a new prompt's keys and values into the rings (addresses unchanged) and rewind the device state."""
        start = next(iter(source.seen.values()))
        self.cache.fill(source, start)
        self.cache.start = start
        self.cache.reset(start)
        self.cursor.zero_()
        self.taken = 0                          # tokens chosen since: the host's copy of the cursor

    @torch.no_grad()
    def run(self, first_token: torch.Tensor, steps: int, eos: set[int], check_every: int = 16) -> torch.Tensor:
        """``first_token`` [B,1] (chosen from the prefill logits) is fed to the first replay; returns the ``steps``
        tokens that follow it, cut after the step at which every sample had produced an end-of-sequence token."""
        if self.taken + steps > self.out.shape[1]:
            raise ValueError(f"{steps} more tokens after {self.taken} do not fit a decoder made for {self.out.shape[1]}")
        self.token.copy_(first_token)
        eos_t = torch.tensor(sorted(eos), device=self.token.device) if eos else None
        finished = torch.isin(first_token.squeeze(1), eos_t) if eos else None
        done = 0
        while done < steps:
            n = min(steps - done, check_every if eos else steps)
            for _ in range(n):
                self.graph.replay()
            self.cache.host_advance(n)
            self.taken += n
            done += n
            if eos:
                hit = torch.isin(self.out[:, :done], eos_t)
                hit[:, 0] |= finished
                all_done = hit.int().cummax(dim=1).values.bool().all(dim=0)          # per step: has every sample finished by now?
                if bool(all_done.any()):
                    done = int(all_done.float().argmax()) + 1
                    break
        return self.out[:, :done].clone()


def decoder_for(model, source: WindowKVCache, max_new_tokens: int) -> GraphDecoder:
    """The model's cached capture when the new prompt fits it, else a fresh one (kept for the next call)."""
    dec = getattr(model, "_graph_decoder", None)
    if dec is not None and dec.fits(source, max_new_tokens):
        dec.load(source)
        return dec
    model._graph_decoder = None                     # drop the old rings before allocating new ones
    dec = GraphDecoder(model, source, max_new_tokens)
    model._graph_decoder = dec
    return dec
