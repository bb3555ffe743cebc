"""A prompt through the plain decoder blocks of a model (inference) with one native call per block.

A block run module by module takes ~370 us of Python for eleven launches; a chat-sized prompt is bound by that.  Where a block
is the stock one, with nothing hooked or replaced, gradients off and no padding, its launches are issued from C++
(``ttcd_block_prefill``), weights that do not lie side by side need not be put there, SwiGLU and the residual sums ride on the
products that feed them.  Fast-weight blocks that run their dual path, and everything else, go through the modules.

Mirrors the block order of the reference (custom_models/ipttcd/modeling_ipttcdv9.py:794-850,
fla/models/transformer/modeling_transformer.py:43-122); the roundings are the module path's.
"""
from __future__ import annotations

import struct

import torch

from .. import _native as nv
from . import layers, stock
from .decoding import _as_defined
from .layers import Attention, WindowKVCache

_BF16 = torch.bfloat16
_RECORD, _EPS = struct.Struct("34q"), struct.Struct("4f")        # what the native call reads

class PlainBlocks:
    """Runs the blocks it can of one forward pass; made by ``plain_blocks``."""

    def __init__(self, x: torch.Tensor, past):
        self.past, self.device, self.device_index, self.shape = past, x.device, x.get_device(), x.shape
        self.B, self.T, self.hidden = x.shape
        self.scratch: dict = {}
        # classes that still are what this package made them, methods that a program may have replaced on an instance
        self.classes = stock.unchanged() if _as_defined() else set()
        self.blocks = {cls for cls in self.classes if cls.__name__.endswith("Block")}
        self.replaceable = frozenset(stock.METHODS)

    def _buffers(self, q_cols: int, kv_cols: int, inter: int, heads: int) -> tuple:
        """Addresses of the scratch of blocks of these widths: rstd, q, o, lse, sum, z, wide."""
        key = (q_cols, kv_cols, inter, heads)
        got = self.scratch.get(key)
        if got is None:
            self.scratch.clear()
            rows, hidden, dev = self.B * self.T, self.hidden, self.device
            # one piece of memory: q, then the sum in its place; o, read for the last time before z is written beside the sum
            at_o = rows * max(q_cols, hidden)
            piece = torch.empty(max(at_o + rows * q_cols, rows * (hidden + inter)), dtype=_BF16, device=dev)
            rstd, lse = (torch.empty(n, dtype=torch.float32, device=dev) for n in (rows, heads * rows))
            # weights whose widths leave narrow tiles only may be put side by side (the native call decides)
            wide = torch.empty((q_cols + 2 * kv_cols) * hidden, dtype=_BF16, device=dev) if (q_cols | kv_cols) % 128 else None
            q = piece.data_ptr()
            at = (rstd.data_ptr(), q, q + 2 * at_o, lse.data_ptr(), q, q + 2 * rows * hidden, 0 if wide is None else wide.data_ptr())
            self.scratch[key] = got = (at, (piece, rstd, lse, wide))
        return got[0]

    def _tensors(self, block):
        """The addresses of the block's weights in the native call's order, or None where it has to run through its modules.  (Runs per
        block and pass: plain dictionaries, as a module's attribute lookup costs more than what is asked here.)"""
        if type(block) not in self.blocks or block.training:
            return None
        if getattr(block, "is_ttt_layer", False) and self.T >= block.ttt_chunk:
            return None
        parts = block._modules
        attn, mlp = parts.get("attn"), parts.get("mlp")
        if type(attn) is not Attention or attn.use_output_gate or attn.use_l2_softmax or attn.head_dim not in (64, 128) or mlp is None:
            return None
        linears = [attn._modules.get(n) for n in ("q_proj", "k_proj", "v_proj", "o_proj")] + [mlp._modules.get(n) for n in ("gate_proj", "up_proj", "down_proj")]
        norms = [parts.get("attn_norm"), parts.get("mlp_norm")] + ([attn._modules.get("q_norm"), attn._modules.get("k_norm")] if attn.qk_norm else [])
        classes, replaceable = self.classes, self.replaceable
        for m in (block, attn, mlp, *norms):
            if type(m) not in classes or m._forward_hooks or m._forward_pre_hooks or not m.__dict__.keys().isdisjoint(replaceable):
                return None
        for m in linears:                    # (only their weights are looked at, by the modules too)
            if type(m) not in classes:
                return None
        hidden, inter = attn.hidden_size, mlp.intermediate_size
        if hidden != self.hidden or min(hidden, inter) < 128 or hidden % 8 or inter % 8 or attn.num_heads % attn.num_kv_heads:
            return None
        # the native call goes by these extents; modules put in the place of the stock ones (a pruned MLP, say) may have others
        dim, q_cols, kv_cols = attn.head_dim, attn.num_heads * attn.head_dim, attn.num_kv_heads * attn.head_dim
        shapes = ((hidden,), (hidden,), (q_cols, hidden), (kv_cols, hidden), (kv_cols, hidden), (hidden, q_cols), (inter, hidden), (inter, hidden),
                  (hidden, inter), (dim,), (dim,))
        device, at, low_bits = self.device_index, [], 0
        for m, shape in zip((*norms[:2], *linears, *norms[2:]), shapes):
            own = m._parameters              # (a weight that is made from others, by a parametrization, is not in there)
            w = own.get("weight")
            if (type(w) is not torch.nn.Parameter or w.dtype is not _BF16 or w.get_device() != device or w.shape != shape or not w.is_contiguous()
                    or own.get("bias") is not None):
                return None
            address = w.data_ptr()
            low_bits |= address
            at.append(address)
        if low_bits % 16 or getattr(linears[0]._parameters["weight"], "_ttcd_gather", None) is not None:
            return None
        return at if attn.qk_norm else at + [0, 0]

    def __call__(self, block, x: torch.Tensor):
        """The block's output, or None where it has to run through its modules (nothing has been done then)."""
        out = self._run(block, x)
        if out is None:
            self.scratch.clear()        # the modules have need of the memory
        return out

    def _run(self, block, x):
        # (a block that ran through its modules, or a hook on it, may have handed on anything)
        if type(x) is not torch.Tensor or x.shape != self.shape or x.dtype is not _BF16 or x.device != self.device:
            return None
        weights = self._tensors(block)
        if weights is None or not x.is_contiguous() or x.data_ptr() % 16:
            return None
        parts = block._modules
        attn, mlp = parts["attn"], parts["mlp"]
        past, B, T, hidden, inter = self.past, self.B, self.T, self.hidden, mlp.intermediate_size
        H, HK, D = attn.num_heads, attn.num_kv_heads, attn.head_dim
        if past is not None and past.get_seq_length(attn.layer_idx) > 0:
            return None
        tables, half = (0, 0), D // 2
        if not attn.use_nope:
            cos, sin = attn.rotary.tables(max(T, attn.max_position_embeddings or 0), x.device, x.dtype)
            extent, tables = cos.shape, (cos.data_ptr(), sin.data_ptr())
            if len(extent) != 2 or sin.shape != extent or extent[0] < T or 2 * extent[1] > D or (tables[0] | tables[1]) % 16:
                return None
            if cos.dtype is not _BF16 or sin.dtype is not _BF16 or not cos.is_contiguous() or not sin.is_contiguous():
                return None
            half = extent[1]
        q_cols, kv_cols = H * D, HK * D
        rstd, q, o, lse, total, z, wide = self._buffers(q_cols, kv_cols, inter, H)
        qkv = torch.empty(B, T, q_cols + 2 * kv_cols, dtype=_BF16, device=x.device)
        k = torch.empty(B, T, HK, D, dtype=_BF16, device=x.device)
        out = torch.empty_like(x)           # holds the normed rows until it is written
        out_at = out.data_ptr()
        record = _RECORD.pack(x.data_ptr(), out_at, out_at, rstd, qkv.data_ptr(), q, k.data_ptr(), o, lse, total, z, *weights, *tables,
                              B, T, hidden, inter, H, HK, D, attn.window_size or 0, half, wide)
        eps = _EPS.pack(parts["attn_norm"].eps, parts["mlp_norm"].eps, attn._modules["q_norm"].eps if attn.qk_norm else 0.0, D ** -0.5)
        nv.call("ttcd_block_prefill", record, eps, nv.stream_ptr())
        if past is not None:
            if not attn.qk_norm and attn.use_nope:
                k = qkv[..., q_cols:q_cols + kv_cols].view(B, T, HK, D)
            past.update(k, qkv[..., q_cols + kv_cols:].view(B, T, HK, D), attn.layer_idx, attn.window_size)
        return out


def plain_blocks(x: torch.Tensor, attention_mask, past, kwargs) -> PlainBlocks | None:
    """A runner for this forward pass, or None where all of it goes through the modules."""
    from ..ops import cuda, selective
    if attention_mask is not None or torch.is_grad_enabled() or cuda._watched() or any(v is not None for v in kwargs.values()):
        return None
    if type(x) is not torch.Tensor or x.dim() != 3 or x.shape[1] < 128 or not nv.use_native(x) or not nv.has("ttcd_block_prefill"):
        return None
    if past is not None and type(past) is not WindowKVCache:
        return None
    if layers._tp_state() is not None or layers._cp_state() is not None or selective.current() is not None:
        return None
    return PlainBlocks(x, past)
