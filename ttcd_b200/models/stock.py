"""The classes that a native block or a fused decode step stands for, with their methods as this package defines them.

Recorded while the package is imported, before a program can have replaced any of them: what a program puts on one of these
classes later, whether before or after its first prompt, shows as a difference.
"""
from __future__ import annotations

import torch

from .base import DecoderForCausalLM, DecoderModel
from .layers import Attention, GatedMLP, RMSNorm
from .modeling_ipttcdv9 import IPTTCDBlock, IPTTCDMLP
from .modeling_transformer import TransformerBlock

METHODS = ("forward", "project_qkv", "finish", "features", "_block_kwargs", "__call__")      # what is computed on behalf of a class


def _methods(cls) -> tuple:
    return tuple(getattr(cls, n, None) for n in METHODS)


_DEFINED = {cls: _methods(cls) for cls in (IPTTCDBlock, TransformerBlock, IPTTCDMLP, GatedMLP, Attention, RMSNorm, DecoderForCausalLM,
                                           DecoderModel, torch.nn.Linear)}


def unchanged() -> set:
    """The classes that still are what they were defined as."""
    return {cls for cls, methods in _DEFINED.items() if _methods(cls) == methods}
