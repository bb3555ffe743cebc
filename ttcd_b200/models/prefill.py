"""A prompt through the plain decoder blocks of a model (inference) with one native call per block.

A block run module by module takes ~370 us of Python for eleven launches; a chat-sized prompt is bound by that.  Where a block
is the stock one, with nothing hooked or replaced, gradients off and no padding, its launches are issued from C++
(``ttcd_block_prefill``), weights that do not lie side by side need not be put there, SwiGLU and the residual sums ride on the
products that feed them.  Fast-weight blocks that run their dual path, and everything else, go through the modules.

Mirrors the block order of the reference (custom_models/ipttcd/modeling_ipttcdv9.py:794-850,
fla/models/transformer/modeling_transformer.py:43-122); the roundings are the module path's.
"""
from __future__ import annotations

import ctypes

import torch

from .. import _native as nv
from . import layers, stock
from .decoding import _as_defined
from .layers import Attention, WindowKVCache

_BF16 = torch.bfloat16


class PlainBlocks:
    """Runs the blocks it can of one forward pass; made by ``plain_blocks``."""

    def __init__(self, x: torch.Tensor, past):
        self.past, self.device, self.shape = past, x.device, x.shape
        self.B, self.T, self.hidden = x.shape
        self.scratch: dict = {}
        # classes that still are what this package made them, methods that a program may have replaced on an instance
        self.classes = stock.unchanged() if _as_defined() else set()
        self.blocks = {cls for cls in self.classes if cls.__name__.endswith("Block")}
        self.replaceable = frozenset(stock.METHODS)

    def _buffers(self, q_cols: int, kv_cols: int, inter: int, heads: int):
        key = (q_cols, kv_cols, inter, heads)
        got = self.scratch.get(key)
        if got is None:
            self.scratch.clear()
            rows, dev = self.B * self.T, self.device
            new = lambda n: torch.empty(n, dtype=_BF16, device=dev)                  # noqa: E731
            f32 = lambda n: torch.empty(n, dtype=torch.float32, device=dev)          # noqa: E731
            # one piece of memory: q, then the sum in its place; o, read for the last time before z is written beside the sum
            at_o = rows * max(q_cols, self.hidden)
            piece = new(max(at_o + rows * q_cols, rows * (self.hidden + inter)))
            # weights whose widths leave narrow tiles only may be put side by side (the native call decides)
            wide = new((q_cols + 2 * kv_cols) * self.hidden) if (q_cols | kv_cols) % 128 else None
            self.scratch[key] = got = (f32(rows), piece, piece[at_o:], f32(heads * rows), piece, piece[rows * self.hidden:], wide)
        return got

    def _tensors(self, block):
        """The block's weights in the native call's order, or None where it has to run through its modules.  (Runs per block and
        pass: plain dictionaries, as a module's attribute lookup costs more than what is asked here.)"""
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
        for m in (block, attn, mlp, *linears, *norms):
            if type(m) not in self.classes or m._forward_hooks or m._forward_pre_hooks or not self.replaceable.isdisjoint(m.__dict__):
                return None
        hidden, inter = attn.hidden_size, mlp.intermediate_size
        if hidden != self.hidden or min(hidden, inter) < 128 or hidden % 8 or inter % 8 or attn.num_heads % attn.num_kv_heads:
            return None
        if any(m._parameters.get("bias") is not None for m in linears):
            return None
        # a weight that is made from others (a parametrization) is not in _parameters
        ws = [m._parameters.get("weight") for m in (*norms[:2], *linears, *norms[2:])]
        # the native call goes by these extents; modules put in the place of the stock ones (a pruned MLP, say) may have others
        dim, q_cols, kv_cols = attn.head_dim, attn.num_heads * attn.head_dim, attn.num_kv_heads * attn.head_dim
        shapes = ((hidden,), (hidden,), (q_cols, hidden), (kv_cols, hidden), (kv_cols, hidden), (hidden, q_cols), (inter, hidden), (inter, hidden),
                  (hidden, inter), (dim,), (dim,))
        device = self.device
        for w, shape in zip(ws, shapes):
            if (type(w) is not torch.nn.Parameter or w.dtype is not _BF16 or w.device != device or w.shape != shape or not w.is_contiguous()
                    or w.data_ptr() % 16):
                return None
        if getattr(ws[2], "_ttcd_gather", None) is not None:
            return None
        return ws if attn.qk_norm else ws + [None, None]

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
        ws = self._tensors(block)
        if ws is None or not x.is_contiguous() or x.data_ptr() % 16:
            return None
        attn = block.attn
        past, B, T = self.past, self.B, self.T
        H, HK, D = attn.num_heads, attn.num_kv_heads, attn.head_dim
        if past is not None and past.get_seq_length(attn.layer_idx) > 0:
            return None
        cos = sin = None
        if not attn.use_nope:
            cos, sin = attn.rotary.tables(max(T, attn.max_position_embeddings or 0), x.device, x.dtype)
            if cos.dim() != 2 or cos.shape != sin.shape or cos.shape[0] < T or 2 * cos.shape[1] > D:
                return None
            if any(t.dtype is not _BF16 or not t.is_contiguous() or t.data_ptr() % 16 for t in (cos, sin)):
                return None
        q_cols, kv_cols = H * D, HK * D
        rstd, q, o, lse, total, z, wide = self._buffers(q_cols, kv_cols, block.mlp.intermediate_size, H)
        qkv = torch.empty(B, T, q_cols + 2 * kv_cols, dtype=_BF16, device=x.device)
        k = torch.empty(B, T, HK, D, dtype=_BF16, device=x.device)
        out = torch.empty_like(x)           # holds the normed rows until it is written
        at = [t.data_ptr() for t in (x, out, out, rstd, qkv, q, k, o, lse, total, z)]
        at += [0 if w is None else w.data_ptr() for w in ws]
        at += [0, 0] if cos is None else [cos.data_ptr(), sin.data_ptr()]
        at += [B, T, self.hidden, block.mlp.intermediate_size, H, HK, D, attn.window_size or 0, D // 2 if cos is None else cos.shape[-1],
               0 if wide is None else wide.data_ptr()]
        eps = (ctypes.c_float * 4)(block.attn_norm.eps, block.mlp_norm.eps, attn.q_norm.eps if attn.qk_norm else 0.0, D ** -0.5)
        nv.call("ttcd_block_prefill", (ctypes.c_longlong * len(at))(*at), eps, nv.stream_ptr())
        if past is not None:
            if not attn.qk_norm and cos is None:
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
