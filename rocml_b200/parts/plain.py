"""The plain dense decoder's layer, for which steps have ways of their own."""
from __future__ import annotations

from .attention import Attention
from .block import PreNormBlock
from .mlp import GatedMLP


def plain_layer(block) -> bool:
    """A pre-norm layer of grouped-query attention in its plain layout and a gated feed-forward."""
    return type(block) is PreNormBlock and type(block.mixer) is Attention and block.mixer.plain and type(block.ff) is GatedMLP
