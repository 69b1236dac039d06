"""All layers of a decode step in one persistent kernel (``kernels.decode_layers``), for models it takes.

The kernel stands for the layers of a plain dense decoder: pre-norm blocks of grouped-query attention (heads of 128 with or
without per-head norm and rotation, every earlier key visible) and a SiLU-gated feed-forward, RMS norms, bfloat16 weights
without biases, all layers alike.  Any other layer, more than eight tokens, lengths at which it does not pay (``pays``) and a step under the profiler (which times the
kernels of a layer one by one, so its table shows kernels that the step does not launch otherwise) run layer by layer as always.

The kernel holds every multiprocessor from the first layer to the last: what other streams have queued waits for a whole step instead of
running beside its kernels.  ``RB_DECODE_LAYERS=0``, read when a step's size is first run or captured, avoids that.
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

MAX_TOKENS = 8         # a tile; with a second one (9 to 16 sequences) a step of 0.6b sizes took 880 us for 884, of 8b sizes 4,000 for 3,537
# What the kernel's registers were measured with: activations of one pass over k for the products that read the stream or the heads, of three
# for down.  Two passes and seven (32b sizes: 5,120 wide, 64 heads, 25,600) are 1 to 4 % slower than the layers' own kernels with one or two sequences, 5 to 12 %
# with more.
MAX_WIDTH, MAX_INTER = 4096, 12288
# From here on (8b sizes, 4,096) a block reads so much activation with more than four sequences that only short contexts are faster.
WIDE = 3072


def pays(n_tokens: int, hidden: int, longest: int, total: int, room: int) -> bool:
    """Whether a step of ``n_tokens`` sequences (padded), whose keys are ``total`` in all and ``longest`` at most, in a batch sized for ``room`` keys
    a sequence, is faster as one kernel.  Its attention cuts every sequence into as many parts as if all were the longest, and a
    part stays with its block: few long sequences among short ones leave most blocks idle.  The layers' own attention has finer parts, and from four sequences of
    more than 4,096 keys on it deals all pages out equally, which costs more where they are equal anyway: the rule has a step there.
    One kernel over the layers' own, 28 layers of 0.6b and 1.7b sizes, 36 of 4b and 8b, device time of a whole step:
    * one and two sequences, up to 32,000 keys: 0.79 to 1.01;
    * three and four: one long among short ones, up to 2,048 keys 0.81 to 1.01, 3,060 0.96 to 1.03, 4,090 1.00 to 1.04, 6,000 and 8,190 0.83 to 1.01; falling to
      half of the longest, up to 4,096 0.73 to 1.02; three of a length, up to 16,380 0.81 to 1.02; four, up to 32,000 0.72 to 1.01, falling to 0.8 0.92 to 0.97;
      one long with 24,000 1.18 to 1.41;
    * five to eight, up to 4,096 keys: 8b sizes 0.98 to 0.99 with 250 and 1.01 to 1.12 with 500 and more; narrower ones, one long 0.93 to 1.01 with 500, 0.94 to 1.02 with 760,
      1.00 to 1.06 with 2,040; five of a length or six falling to half 0.93 to 1.00 up to 1,530, 0.96 to 1.04 with 2,040; eight of a length 0.88 to 1.00;
    * five to eight beyond: one long 1.14 to 1.50 with 8,190, five of a length 1.08 to 1.14; six of a length or eight falling to half 0.96 to 1.00, seven 0.86 to 0.97,
      eight 0.78 to 0.92, with 16,380 0.92 to 0.96, with 32,000 0.95 to 1.01; eight falling to 0.8, 16,380 0.97 to 1.00, 24,000 1.00 to 1.02."""
    if n_tokens <= 2:
        return True
    full = total / (n_tokens * longest)          # how much of the batch's places times the longest is there
    if n_tokens <= 4:
        if full >= 0.7:
            return full >= 0.9 or room <= 16384
        return room <= (4096 if full >= 0.5 else 2048) or 4096 < room <= 8192
    if room > 4096:
        return full >= (0.7 if room <= 8192 else 0.9 if room <= 16384 else 0.95)
    if hidden > WIDE:
        return room <= 256
    return room <= (4096 if full >= 0.9 else 1536 if full >= 0.4 else 512)


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


def fits(model) -> bool:
    """Whether this model's decode steps may run as the one kernel, as far as its layers' kind and widths say."""
    return model.env.act_dtype == torch.bfloat16 and all(
        plain_layer(b) and max(model.hidden, b.mixer.nq * b.mixer.hd) <= MAX_WIDTH and b.ff.inter <= MAX_INTER for b in model.blocks)


def takes(model, batch, cache) -> bool:
    """Whether this step's layers run as the one kernel."""
    if not batch.is_decode or batch.n_tokens > MAX_TOKENS or not batch.at_once or not fits(model) or _profiler.ACTIVE is not None \
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
    # Every block has a unit (16 rows) of the first product and of gate | up.  (Not where the two ways meet: at 256 to 1,024 wide layers with 64 to 192 units the one
    # kernel takes 0.58 to 0.93 of the others' time too.)
    sms = torch.cuda.get_device_properties(model.env.device).multi_processor_count
    return first.mixer.qkv.n >= 16 * sms and 2 * first.ff.inter >= 16 * sms


def forward(model, resid, batch, cache) -> bool:
    """Run the layers on the step's residual stream ``resid`` [T, H] float32, which holds the embedding's rows.  False where the kernel
    declines: nothing has run then, and the layers' own kernels take the step."""
    blocks = [model.blocks[e.layer] for e in model.spec.schedule]
    m, inter = blocks[0].mixer, blocks[0].ff.inter
    splits = kernels.decode_layers_splits(batch.n_tokens * m.nkv, batch.max_kv_len, resid.device)
    layers = []
    for i, (b, view) in enumerate(zip(blocks, cache.views)):
        nxt = blocks[i + 1].mixer_norm if i + 1 < len(blocks) else None
        layers.append((b.mixer.qkv.weight, b.mixer.o.weight, b.ff.gate_up.weight, b.ff.down.weight, b.ff_norm.weight,
                       nxt.weight if nxt is not None else None, b.mixer.q_norm_w, b.mixer.k_norm_w, view.k, view.v,
                       b.ff_norm.eps, b.mixer_norm.eps))
    return kernels.decode_layers(resid, blocks[0].mixer_norm.weight, layers, m.nq, m.nkv, inter, m.qk_norm_eps, m.scale,
                                 m.position.cos_sin(batch) if m.position.inv_freq is not None else None,
                                 batch.seq_slot, batch.kv_len, cache.views[0].block_table, splits)
