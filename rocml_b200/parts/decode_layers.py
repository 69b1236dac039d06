"""All layers of a decode step in one persistent kernel (``kernels.decode_layers``), for models it takes.

The kernel stands for the layers of a plain dense decoder: pre-norm blocks of grouped-query attention (heads of 128 with or
without per-head norm and rotation, every earlier key visible) and a SiLU-gated feed-forward, RMS norms, bfloat16 weights
without biases, all layers alike.  Any other layer, more than eight tokens and a step under the profiler (which times the
kernels of a layer one by one) run layer by layer as always.
"""
from __future__ import annotations

import os

import torch

from .. import kernels
from ..profile import profiler as _profiler
from .attention import Attention
from .block import _defer_enabled
from .norm import RMSNorm
from .plain import plain_layer

# Up to one tile of tokens the one kernel is the faster one: a step before and now, microseconds, 28 layers of 0.6b sizes with 1, 2 and 8
# sequences 758, 853, 856 -> 667, 769, 764; 1.7b with 1 and 4 1,131, 1,159 -> 937, 1,006, with 8 of 700 to 1,300 tokens 1,280 -> 1,248;
# 4b with 1 (900 tokens), 4 and 8 2,080, 2,114, 2,227 -> 1,971, 1,947, 2,068; 8b with 1 and 8 2,961, 3,096 -> 2,761, 3,058.  A second tile of
# tokens: 0.6b with 16 884 -> 880, 8b 3,537 -> 4,000.
MAX_TOKENS = 8


def enabled() -> bool:
    """RB_DECODE_LAYERS=0 runs decode steps layer by layer (RB_DEFER=0, which asks for the norms' own kernels, does too)."""
    return os.environ.get("RB_DECODE_LAYERS", "1") != "0" and _defer_enabled()


def _weight(linear) -> bool:
    w = linear.weight
    return w is not None and w.dtype == torch.bfloat16 and w.is_cuda and w.is_contiguous() and w.data_ptr() % 16 == 0 and \
        linear.bias is None and linear.k % 64 == 0


def _norm(norm, like) -> bool:
    return type(norm) is RMSNorm and norm.weight is not None and norm.weight.is_contiguous() and norm.weight.dtype == like.weight.dtype


def _alike(a: Attention, b: Attention) -> bool:
    pa, pb = a.position, b.position
    return (a.nq, a.nkv, a.hd, a.scale, a.qk_norm, a.qk_norm_eps) == (b.nq, b.nkv, b.hd, b.scale, b.qk_norm, b.qk_norm_eps) and \
        (pa.inv_freq is None) == (pb.inv_freq is None) and \
        all(getattr(pa, f, None) == getattr(pb, f, None) for f in ("rot_dim", "theta", "scaling", "ramp_scaling", "magnitude"))


def _head_norms(m: Attention, first: Attention) -> bool:
    return all(w is not None and w.dtype == first.q_norm_w.dtype and w.is_contiguous() and w.data_ptr() % 16 == 0 for w in (m.q_norm_w, m.k_norm_w))


def _block_fits(block, first, hidden: int) -> bool:
    if not plain_layer(block):
        return False
    m, ff = block.mixer, block.ff
    if not (m.hd == 128 and not m.shares_cache and m._span() == 0 and m.nq // m.nkv <= 8 and _alike(m, first.mixer)):
        return False
    if (m.position.inv_freq is not None and m.position.rot_dim != m.hd) or (m.qk_norm and not _head_norms(m, first.mixer)):
        return False
    if not (ff.act == "silu" and ff.gate_up.paired and ff.inter == first.ff.inter):
        return False
    return all(_weight(w) for w in (m.qkv, m.o, ff.gate_up, ff.down)) and hidden % 64 == 0 and \
        _norm(block.mixer_norm, first.mixer_norm) and _norm(block.ff_norm, first.mixer_norm)


def takes(model, batch, cache) -> bool:
    """Whether this step's layers run as the one kernel."""
    if not batch.is_decode or batch.n_tokens > MAX_TOKENS or model.env.act_dtype != torch.bfloat16 or _profiler.ACTIVE is not None \
            or not enabled():
        return False
    first = None
    for e, view in zip(model.spec.schedule, cache.views):
        if e.add_input or e.add_row is not None or e.reads_cache_of is not None:
            return False
        block = model.blocks[e.layer]
        first = block if first is None else first
        if not _block_fits(block, first, model.hidden) or view.kind != "kv" or not view.writes or view.extras \
                or view.group is not cache.views[0].group or view.k.dtype != torch.bfloat16:
            return False
    if first is None:
        return False
    # every block should have a unit (16 rows) of the first product and of gate | up
    sms = torch.cuda.get_device_properties(model.env.device).multi_processor_count
    return first.mixer.qkv.n >= 16 * sms and 2 * first.ff.inter >= 16 * sms


def forward(model, resid, batch, cache) -> None:
    """Run the layers on the step's residual stream ``resid`` [T, H] float32, which holds the embedding's rows."""
    blocks = [model.blocks[e.layer] for e in model.spec.schedule]
    m, inter = blocks[0].mixer, blocks[0].ff.inter
    splits = kernels.decode_layers_splits(batch.n_tokens * m.nkv, batch.max_kv_len, resid.device)
    layers = []
    for i, (b, view) in enumerate(zip(blocks, cache.views)):
        nxt = blocks[i + 1].mixer_norm if i + 1 < len(blocks) else None
        layers.append((b.mixer.qkv.weight, b.mixer.o.weight, b.ff.gate_up.weight, b.ff.down.weight, b.ff_norm.weight,
                       nxt.weight if nxt is not None else None, b.mixer.q_norm_w, b.mixer.k_norm_w, view.k, view.v,
                       b.ff_norm.eps, b.mixer_norm.eps))
    kernels.decode_layers(resid, blocks[0].mixer_norm.weight, layers, m.nq, m.nkv, inter, m.qk_norm_eps, m.scale,
                          m.position.cos_sin(batch) if m.position.inv_freq is not None else None,
                          batch.seq_slot, batch.kv_len, cache.views[0].block_table, splits)
