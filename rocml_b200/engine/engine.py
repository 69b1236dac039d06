"""The engine: a model, its cache, and ONE step function.

``step(entries)`` runs exactly the tokens it is given, as one batch, from the cache that
earlier steps left, and returns the logits at the wanted places.  The sequences of a step
may have any lengths (whole prompts of unequal length, pieces of prompts, or one token
each); a step larger than the work space is cut into pieces internally, which changes no
result.  Steps of one token per sequence are replayed from CUDA graphs captured per batch
size and context bucket, with the batch padded up to the bucket; padding changes no result
because padded tokens carry slot -1 and every kernel skips them.

The reference has three entry points for this (one token: rocml/src/forward/mod.rs:246-387;
a chunk of one prompt: chunk_forward.rs:62-189; the chunk loop: :33-53) and no batch.
"""
from __future__ import annotations

from collections import OrderedDict
from dataclasses import dataclass
from typing import Dict, List, Optional, Sequence, Tuple

import numpy as np
import torch

from ..cache import SequenceCache
from ..config import load_model_spec
from ..errors import CacheError, ConfigError, KernelError, RocmlError
from ..parts import BuildEnv, decode_layers
from ..parts.plain import plain_layer
from ..profile import profiler as _profiler
from .batch import BatchBuffers, HostBatch, StepBatch, pack_entries
from .model import Model

_DTYPES = {"bfloat16": torch.bfloat16, "bf16": torch.bfloat16, "float32": torch.float32, "fp32": torch.float32}


@dataclass
class StepEntry:
    slot: int
    tokens: Sequence[int]
    want: Sequence[int] = ()


def _bucket(n: int, floor: int = 1) -> int:
    b = floor
    while b < n:
        b *= 2
    return b


def _batch_bucket(n: int, ctx: int, waves: Sequence[int]) -> int:
    """How many sequences a captured decode graph for ``n`` of them and a context of ``ctx`` is sized for: the next power of two, or
    one of ``waves`` below it that holds them.  With fewer than eight pages decode attention runs a block a (sequence, head
    group), and its launch does not know which of them are padding: 33 to 55 sequences on 8 heads, which run as one wave,
    would be taken for the 64 that do not, whose blocks keep one page in flight instead of two (28 layers of 0.6b sizes, 44
    sequences of 43, 103, 168 and 231 keys padded to 64: 1,226, 1,293, 1,360 and 1,426 us a step, to 55: 1,185, 1,220, 1,266 and 1,326; 36 layers of 4b sizes 2,773 to 2,994 and 2,678 to 2,859)."""
    b = _bucket(n)
    if ctx < 8 * 64:
        b = min([b] + [w for w in waves if n <= w])
    return b


def _ctx_bucket(n: int) -> int:
    """Context length a captured decode graph is sized for: the next multiple of 256 (of 1024 beyond
    4096).  Fine steps matter: decode attention deals its blocks out over the bucket, and blocks
    that lie past the sequences' real end do nothing."""
    step = 256 if n <= 4096 else 1024
    return max(step, -(-n // step) * step)


# Prompts of few tokens (all sequences of a piece together) are replayed from captured graphs too, where their kernels take less time than the host
# takes to launch them one by one (9 launches a layer): the layers' weights decide that.  Milliseconds of a step alone, launched and replayed, at 61,
# 128 and 256 tokens: 28 layers of 0.6b sizes (31 MB a layer) 4.1, 4.0, 3.8 and 1.7, 2.3, 2.5; 28 of 1.7b (101 MB) 4.2, 4.3, 3.9 and 2.1, 2.8, 3.1; 36 of 4b
# (202 MB) 5.3, 5.3, 6.1 and 3.4, 4.4, 5.6, but with 129 tokens 5.7 for 5.5; 36 of 8b (386 MB) 5.4, 5.4, 7.2 and 4.5, 5.1, 6.9, with 129 tokens 6.5 for 7.0.
# A capture takes 3 to 6 ms more than the step that it stands for (at times 30 to 190), which a few replays pay for: a size is captured the fourth time
# that it comes.  (Streams of prompts on new engines, ms a prompt, launched, captured the first time with four kept as they came, and by these rules: 64 lengths
# at random up to 256, 0.6b 3.96, 5.87, 3.49, 4b 5.58, 9.05, 5.58; five lengths in turn 4.03, 9.47, 2.89 and 5.36, 21.1, 4.98; one length 4.15, 2.03, 2.22 and 5.37, 3.67,
# 4.01; the prompts of ten turns of a chat 4.26, 8.53, 4.24 and 6.44, 64.9, 6.03.)
PROMPT_GRAPH_RULES = ((128 << 20, 256), (400 << 20, 128))      # (bytes of a layer at most, tokens at most)
PROMPT_GRAPH_TIMES = 4
PROMPT_GRAPHS = 8                                              # how many are kept at most


def _prompt_graph_tokens(layer_bytes: int) -> int:
    return next((tokens for most, tokens in PROMPT_GRAPH_RULES if layer_bytes <= most), 0)


def _prompt_pads(n_tokens: int, n_seqs: int, n_want: int, longest: int):
    """What a captured prompt graph is sized for, tokens, sequences, wanted rows, longest piece, longest sequence (which decides the order of
    blocks only), or None where the step has no graph: more wanted places than sequences.  Powers of two, few of them: padding 33
    tokens to 64 costs 4 % of a replay, a size more a capture."""
    t, b = _bucket(n_tokens, 16), _bucket(n_seqs)
    return (t, b, b if n_want else 0, t, _bucket(longest, 4096), False) if n_want <= b else None


class GraphSizes:
    """Which sizes of short prompts are worth a captured graph.  The first steps of a size are launched kernel by kernel; the ``times``-th is captured
    while there is room, and later only if the size has come more often than the rarest of those kept by as many times:
    sizes that take turns do not drive one another out.  Counts are halved now and then, so that what was common long ago gives way."""

    def __init__(self, kept: int, times: int = PROMPT_GRAPH_TIMES):
        self.kept, self.times = kept, times
        self.seen: Dict[tuple, int] = {}
        self._total = 0

    def due(self, size, graphs: "OrderedDict") -> bool:
        """Whether a step of this size runs as a graph, of which ``graphs`` are there; the one that has to go for it is then the first of them."""
        if size in graphs:
            return True
        n = self.seen.get(size, 0) + 1
        if n < self.times or self.kept < 1:
            return False
        if len(graphs) >= self.kept:
            rarest = min(graphs, key=lambda k: self.seen.get(k, 0))
            if n < self.seen.get(rarest, 0) + self.times:
                return False
            graphs.move_to_end(rarest, last=False)
        return True

    def note(self, size) -> None:
        """A step of this size has run."""
        self.seen[size] = self.seen.get(size, 0) + 1
        self._total += 1
        if self._total >= 256:
            self.seen = {k: n // 2 for k, n in self.seen.items() if n > 1}
            self._total = sum(self.seen.values())


class Engine:
    def __init__(self, model: Model, max_tokens: int, max_slots: Optional[int] = None,
                 max_step_tokens: int = 4096, use_graphs: bool = True, max_seq_len: Optional[int] = None,
                 max_graphs: int = 8):
        """``max_graphs``: how many captured decode graphs are kept (one per batch bucket and context
        bucket, least recently used dropped first); each holds its own activations and logits.  As many graphs of short prompts, up to
        ``PROMPT_GRAPHS`` and as the memory left over allows, are kept beside them."""
        self.model = model
        self.env = model.env
        self.device = model.env.device
        self.max_step_tokens = int(max_step_tokens)
        if self.max_step_tokens < 1:
            raise ConfigError("max_step_tokens must be at least 1")
        self.max_graphs = max(1, int(max_graphs))
        max_tokens = int(max_tokens)
        if max_slots is None:
            # every live sequence holds a page at least, so the pages bound the sequences (a slot costs a row
            # of the block table and, where a layer keeps fixed-size state, its state)
            max_slots = max(1, min((max_tokens + 63) // 64, 4096))
        self.use_graphs = bool(use_graphs) and model.graph_safe and self.device.type == "cuda"
        # (layers whose prompt kernels take nothing from the host but the step's sizes)
        self._prompt_graph_tokens = 0
        if self.use_graphs and self.env.act_dtype == torch.bfloat16 and all(plain_layer(b) for b in model.blocks):
            self._prompt_graph_tokens = _prompt_graph_tokens(max(b.weight_bytes() for b in model.blocks))
        self._one_kernel = decode_layers.fits(model)
        self._prompt_sizes = GraphSizes(self._check_budget(max_tokens, max_slots))
        self.cache = SequenceCache(
            model.cache_requirements(), model.reads_cache_of(), max_tokens, max_slots,
            min(model.spec.max_position, max_seq_len or model.spec.max_position), self.env.act_dtype,
            self.device, self.max_step_tokens)
        # how many sequences run as one wave of the decode attention that can keep two pages in flight (heads of 128 in
        # bfloat16), for each of the model's counts of key/value heads
        self._waves = []
        if self.use_graphs and self.env.act_dtype == torch.bfloat16:
            from .. import kernels
            self._waves = sorted({kernels.decode_wave(g.req.n_kv_heads, self.device) for g in self.cache.kv_groups
                                  if g.req.head_dim == 128})
        self._eager: Dict[Tuple[int, int], BatchBuffers] = {}
        self._graphs: "OrderedDict[Tuple[int, ...], dict]" = OrderedDict()
        self._prompt_graphs: "OrderedDict[Tuple[int, ...], dict]" = OrderedDict()
        self._capture_stream = None
        self.graphs_captured = 0
        self.launches = 0          # steps issued (sub-steps counted)
        self.last_h2d_bytes = 0
        self._sampler = None
        self._device_tokens = None
        self._replayed = False     # the last piece's logits are a graph's
        self.graph_kernel_launches = 0  # kernels run by graph replays

    # After the weights are resident: does the cache fit what is left, with head room for a step's
    # activations?  (The reference's check: rocml/src/forward/mod.rs:145-168, 768 MiB of head room,
    # rocml/src/budget/mod.rs:37.)  What a step needs is asked of the parts, so it holds for any
    # arrangement: the widest step's buffers, one more set and its logits for every captured decode
    # graph that may be kept, and the groups of fixed-size state.  Returns how many graphs of short prompts
    # fit beside all that.
    def _check_budget(self, max_tokens: int, max_slots: int) -> int:
        if self.device.type != "cuda":
            return 0
        esz = 4 if self.env.act_dtype == torch.float32 else 2
        per_token = state = 0
        from ..cache.requirements import simple_requirements
        for r in [x for r, src in zip(self.model.cache_requirements(), self.model.reads_cache_of()) if src is None
                  for x in simple_requirements(r)]:
            if hasattr(r, "n_kv_heads"):
                per_token += (1 if getattr(r, "shared_values", False) else 2) * r.n_kv_heads * r.head_dim * esz
            elif hasattr(r, "shape"):
                n = 1
                for d in r.shape:
                    n *= int(d)
                state += n * torch.empty((), dtype=r.dtype).element_size() * max_slots
        step = self.model.workspace_bytes(self.max_step_tokens, min(self.max_step_tokens, max_slots))
        graphs = 0
        if self.use_graphs:
            graphs = self.max_graphs * self.model.workspace_bytes(_bucket(max_slots), _bucket(max_slots))
        headroom = (768 << 20) + step + graphs
        free, total = torch.cuda.mem_get_info(self.device)
        need = ((max_tokens + 63) // 64 * 64) * per_token + state
        if need + headroom > free:
            from ..errors import MemoryBudget
            fit = max(0, (free - headroom - state) // per_token // 64 * 64) if per_token else 0
            raise MemoryBudget(max_tokens, int(fit), (
                f"{need / 2**30:.1f} GiB of keys, values and state ({per_token} bytes per token) + "
                f"{headroom / 2**30:.1f} GiB head room (a step of {self.max_step_tokens} tokens: {step / 2**30:.2f}, "
                f"{self.max_graphs if self.use_graphs else 0} decode graphs: {graphs / 2**30:.2f}) against "
                f"{free / 2**30:.1f} GiB free of {total / 2**30:.1f} GiB"))
        if not self._prompt_graph_tokens:
            return 0
        each = self.model.workspace_bytes(self._prompt_graph_tokens, min(_bucket(max_slots), self._prompt_graph_tokens))
        return min(PROMPT_GRAPHS, self.max_graphs, (free - need - headroom) // each)

    # ---- construction ----------------------------------------------------------------------------
    @staticmethod
    def from_folder(folder: str, dtype: str = "bfloat16", device="cuda:0", **kw) -> "Engine":
        if dtype not in _DTYPES:
            raise ConfigError(f"dtype must be one of {sorted(set(_DTYPES))}, found {dtype!r}")
        dev = torch.device(device)
        if dev.type != "cuda":
            raise KernelError("the engine runs on a CUDA device only; there is no CPU path")
        spec = load_model_spec(folder)
        model = Model(spec, BuildEnv(dev, _DTYPES[dtype]))
        with torch.cuda.device(dev):
            model.load_folder(folder)
            return Engine(model, **kw)

    # ---- slots ---------------------------------------------------------------------------------------
    def new_sequence(self) -> int:
        return self.cache.alloc_slot()

    def release(self, slot: int) -> None:
        self.cache.free_slot(slot)

    def length(self, slot: int) -> int:
        return self.cache.length(slot)

    # ---- the step --------------------------------------------------------------------------------------
    def step(self, entries: Sequence[StepEntry], device_tokens: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
        """Run the entries' tokens; return float32 logits [wanted places, vocab] in the order of
        the entries and of each entry's ``want`` (None when nothing is wanted).  The tensor may
        be reused by the next step: read it before stepping again.

        ``device_tokens`` (int32 on the device, one per entry) replaces the entries' token ids
        for a step of one token per sequence: the ids a sampling kernel has just written are
        fed back without passing through the host."""
        if device_tokens is not None and any(len(e.tokens) != 1 for e in entries if isinstance(e, StepEntry)):
            raise RocmlError("device_tokens needs exactly one token per entry")
        entries = [e if isinstance(e, StepEntry) else StepEntry(*e) for e in entries]
        if not entries:
            return None
        seen = set()
        vocab = self.model.vocab
        for e in entries:
            if e.slot in seen:
                raise CacheError(f"slot {e.slot} appears twice in one step")
            seen.add(e.slot)
            if len(e.tokens) == 0:
                raise RocmlError(f"slot {e.slot}: a step entry needs at least one token")
            if len(e.tokens) > 64:
                arr = np.asarray(e.tokens)
                bad = arr[(arr < 0) | (arr >= vocab)][:1].tolist()
            else:
                bad = [t for t in e.tokens if not 0 <= int(t) < vocab]
            if bad:
                raise RocmlError(f"slot {e.slot}: token id {bad[0]} is outside the vocabulary of {vocab}")
            for w in e.want:
                if not 0 <= w < len(e.tokens):
                    raise RocmlError(f"slot {e.slot}: wanted place {w} is outside the {len(e.tokens)} tokens given")
        total = sum(len(e.tokens) for e in entries)
        if total <= self.max_step_tokens:
            pieces = [[(i, 0, len(e.tokens)) for i, e in enumerate(entries)]]
        else:
            pieces = self._cut(entries)
        # Room for everything, before anything launches.  Pages are then taken piece by piece: a
        # layer that keeps a window of keys gives pages back between the pieces of a long prompt, and
        # its group holds only a window and a piece for each sequence.
        self.cache.plan([[(entries[i].slot, b - a) for i, a, b in piece] for piece in pieces])

        with torch.cuda.device(self.device):
            outs, order = [], []
            for piece in pieces:
                slots, olds, toks, wants = [], [], [], []
                for i, a, b in piece:
                    e = entries[i]
                    slots.append(e.slot)
                    olds.append(self.cache.grow(e.slot, b - a))
                    toks.append(e.tokens[a:b])
                    w_here = sorted(w for w in set(e.want) if a <= w < b)
                    wants.append([w - a for w in w_here])
                    order.extend((i, w) for w in w_here)
                # (one token per entry: a piece's entries are a run of them)
                self._device_tokens = None if device_tokens is None else device_tokens[piece[0][0]:piece[-1][0] + 1]
                logits = self._run(slots, olds, toks, wants)
                for (i, a, b) in piece:
                    self.cache.commit(entries[i].slot, b - a)
                if logits is not None:
                    # (a replayed graph's logits live until the next replay, which may be the next piece's)
                    outs.append(logits.clone() if self._replayed and len(pieces) > 1 else logits)
            if not outs:
                return None
            result = outs[0] if len(outs) == 1 else torch.cat(outs, dim=0)
            wanted = [(i, w) for i, e in enumerate(entries) for w in e.want]
            if wanted != order:
                where = {key: r for r, key in enumerate(order)}
                idx = torch.tensor([where[k] for k in wanted], dtype=torch.long, device=self.device)
                result = result.index_select(0, idx)
            return result

    def _cut(self, entries):
        """Cut a step that is larger than the work space into pieces of at most
        max_step_tokens tokens, sequence after sequence, a sequence continuing in the next
        piece where it was cut (what the reference's chunk loop does for one prompt,
        rocml/src/forward/chunk_forward.rs:41-51)."""
        pieces, cur, room = [], [], self.max_step_tokens
        for i, e in enumerate(entries):
            a, n = 0, len(e.tokens)
            while a < n:
                take = min(room, n - a)
                cur.append((i, a, a + take))
                a += take
                room -= take
                if room == 0:
                    pieces.append(cur)
                    cur, room = [], self.max_step_tokens
        if cur:
            pieces.append(cur)
        return pieces

    # ---- one piece: eager launches or a graph replay ------------------------------------------------------
    def _run(self, slots, old_lens, token_lists, wants) -> Optional[torch.Tensor]:
        packed = pack_entries(slots, old_lens, token_lists, wants)
        token_ids, positions, slot_of_token, cu_q, kv_len, want_rows = packed
        T, B, W = len(token_ids), len(slots), len(want_rows)
        q_lens = [len(t) for t in token_lists]
        is_decode = all(n == 1 for n in q_lens)
        host = HostBatch(list(slots), q_lens, list(kv_len), list(want_rows))
        self.cache.flush()
        self.launches += 1
        self._replayed = False
        prof = _profiler.ACTIVE
        if prof is not None:
            # a profiled step runs its kernels one by one, without a graph (rocml_b200.profile.profiler)
            with prof.step("decode" if is_decode else "prefill", q_lens, kv_len):
                return self._run_eager(packed, host, slots, q_lens, T, B, W, is_decode)
        if is_decode and self.use_graphs:
            ctx_pad = _ctx_bucket(max(kv_len))
            b_pad = _batch_bucket(B, ctx_pad, self._waves)
            at_once = self._at_once(b_pad, kv_len, ctx_pad)
            key = (b_pad, ctx_pad) if at_once else (b_pad, ctx_pad, False)
            return self._run_graph(self._graphs, self.max_graphs, key, packed, host, W, (b_pad, b_pad, b_pad, 1, ctx_pad, True), at_once)
        pads = _prompt_pads(T, B, W, max(kv_len)) if not is_decode and T <= self._prompt_graph_tokens and self._prompt_sizes.kept else None
        if pads is not None:
            if self._prompt_sizes.due(pads, self._prompt_graphs):
                out = self._run_graph(self._prompt_graphs, self._prompt_sizes.kept, pads, packed, host, W, pads)
            else:
                # (padded as the graph will be: an answer does not depend on how often its size has come)
                out = self._run_eager(packed, host, slots, q_lens, T, B, W, is_decode, pads)
            self._prompt_sizes.note(pads)
            return out
        return self._run_eager(packed, host, slots, q_lens, T, B, W, is_decode)

    def _at_once(self, n_tokens: int, kv_len, room: int) -> bool:
        """``StepBatch.at_once`` of a decode step.  (Where there is no one kernel it says nothing: one graph a bucket.)"""
        return not self._one_kernel or n_tokens > decode_layers.MAX_TOKENS or decode_layers.pays(n_tokens, self.model.hidden, max(kv_len), sum(kv_len), room)

    def _run_eager(self, packed, host, slots, q_lens, T, B, W, is_decode, pads=None) -> Optional[torch.Tensor]:
        kv_len = packed[4]
        key = (_bucket(T, 64), _bucket(B, 8))
        if key not in self._eager:
            self._eager[key] = BatchBuffers(key[0], key[1], key[0], self.device)
        buf = self._eager[key]
        t_pad, b_pad, w_pad, max_q, max_kv, _ = pads or (T, B, W, max(q_lens), max(kv_len), is_decode)
        buf.fill(*packed, slots, pad_tokens=t_pad, pad_seqs=b_pad, pad_want=w_pad)
        if self._device_tokens is not None:
            buf.token_ids[:B].copy_(self._device_tokens, non_blocking=True)
        self.last_h2d_bytes = buf.h2d_bytes
        at_once = not is_decode or self._at_once(T, kv_len, max_kv)
        out = self.model.forward(self._batch(buf, t_pad, b_pad, w_pad, max_q, max_kv, is_decode, host, at_once), self.cache)
        return out[:W] if W else None

    @staticmethod
    def _batch(buf: BatchBuffers, T, B, W, max_q, max_kv, is_decode, host, at_once=True, capturing=False) -> StepBatch:
        return StepBatch(
            n_tokens=T, n_seqs=B, n_want=W, max_q_len=max_q, max_kv_len=max_kv, is_decode=is_decode,
            token_ids=buf.token_ids, positions=buf.positions, slot_of_token=buf.slot_of_token,
            seq_slot=buf.seq_slot, cu_q=buf.cu_q, kv_len=buf.kv_len, want_rows=buf.want_rows, host=host,
            capturing=capturing, at_once=at_once)

    def _run_graph(self, graphs, kept: int, key, packed, host, W, pads, at_once=True) -> Optional[torch.Tensor]:
        """Replay the graph of ``key`` among ``graphs``, of which ``kept`` are kept, after capturing it if need be.  ``pads``: the
        tokens, sequences and wanted rows that it is sized for, the longest piece of a sequence, the longest sequence, whether it is
        a step of single tokens."""
        t_pad, b_pad, w_pad, max_q, ctx_pad, is_decode = pads
        B = len(host.seq_slots)
        g = graphs.get(key)
        if g is None:
            while len(graphs) >= kept:
                # the least recently used bucket goes; its memory returns to the graphs' pool.  Work that
                # is still queued may read it: wait before it is released.
                _, old = graphs.popitem(last=False)
                torch.cuda.current_stream().synchronize()
                if old["graph"] is not None:
                    old["graph"].reset()
                old.clear()
            g = {"buffers": BatchBuffers(t_pad, b_pad, w_pad, self.device), "graph": None, "logits": None, "plain": False}
            graphs[key] = g
        else:
            graphs.move_to_end(key)
        buf: BatchBuffers = g["buffers"]
        buf.fill(*packed, host.seq_slots, pad_tokens=t_pad, pad_seqs=b_pad, pad_want=w_pad)
        if self._device_tokens is not None:
            buf.token_ids[:B].copy_(self._device_tokens, non_blocking=True)
        self.last_h2d_bytes = buf.h2d_bytes
        def batch(capturing=False):
            return self._batch(buf, t_pad, b_pad, w_pad, max_q, ctx_pad, is_decode, None if capturing else host, at_once, capturing)
        if g["graph"] is None and not is_decode and not g["plain"]:
            self._capture(g, batch(capturing=True))              # (a prompt of this size has run before)
        if g["graph"] is None:
            # First use of a decode bucket: run it plainly (this also loads every kernel), then
            # capture the same launches for the next time.  Capturing executes nothing.
            out = self.model.forward(batch(), self.cache)
            if is_decode and not g["plain"]:
                torch.cuda.current_stream().synchronize()
                self._capture(g, batch(capturing=True))
                self.graphs_captured += g["graph"] is not None
            return out[:W] if W else None
        g["graph"].replay()
        self._replayed = True
        self.graph_kernel_launches += g["kernels"]
        return g["logits"][:W] if W else None

    def _capture(self, g: dict, batch: StepBatch) -> None:
        """Capture the launches of ``batch`` as g["graph"].  Blocks that the allocator holds for later are not given back first, as
        ``torch.cuda.graph`` does (an engine with 28 layers of 1.7b sizes made its first graph in 60 ms that way, in 22 without): only where the device has no memory left, which the allocator cannot help
        during a capture, are they, and the capture is tried again.  If that fails too, steps of this size run plainly (g["plain"])."""
        from .. import kernels
        if self._capture_stream is None:
            # (one for all captures: the allocator hands a block out again only on the stream that it was made for)
            self._capture_stream = torch.cuda.Stream(self.device)
        before = kernels.launch_count
        for _ in range(2):
            # (graphs share their memory, as no two run side by side; it goes with the last of them)
            pool = next((x["graph"].pool() for t in (self._graphs, self._prompt_graphs) for x in t.values() if x["graph"] is not None), None)
            graph = torch.cuda.CUDAGraph()
            try:
                with torch.cuda.stream(self._capture_stream):
                    # (only this thread's calls are watched: others may allocate meanwhile)
                    graph.capture_begin(pool, "thread_local")
                    try:
                        logits = self.model.forward(batch, self.cache)
                    finally:
                        graph.capture_end()
                g["graph"], g["logits"], g["kernels"] = graph, logits, kernels.launch_count - before
                return
            except RuntimeError as e:              # (the allocator's own type is one, what an instantiation raises is not that type)
                if "out of memory" not in str(e):
                    raise
            finally:
                kernels.launch_count = before      # captured, not launched
            logits = None
            graph.reset()
            torch.cuda.empty_cache()
        g["plain"] = True

    # ---- generation: the engine as the loop's executor ------------------------------------------------------
    @property
    def max_seq_len(self) -> int:
        return self.cache.max_seq_len

    def capacity_tokens(self) -> int:
        return self.cache.n_pages * 64

    def capacity_slots(self) -> int:
        return self.cache.max_slots

    def launch(self, slots, tokens, params, rngs, histories, feed_from=None):
        """Enqueue a step of the sequences with their next tokens and the sampling of one token
        each, and return a handle at once.  With ``feed_from`` (the handle of the step before,
        over the same sequences in the same order) the next tokens are the ones that step
        sampled, taken on the device: ``tokens`` is not read."""
        device_tokens = None
        if feed_from is not None:
            if feed_from.n != len(slots):
                raise RocmlError("feed_from must hold one token for each sequence of the step")
            tokens = [[0]] * len(slots)
            device_tokens = feed_from.device_tokens
        if self._sampler is None:
            from ..sampling import Sampler
            self._sampler = Sampler(self.device, max_batch=max(self.cache.max_slots, 1))
        from .. import kernels
        prof = _profiler.ACTIVE
        if prof is not None:
            # the sampling belongs to the step it follows (one piece assumed; a cut prompt opens steps of its own)
            phase = "decode" if all(len(t) == 1 for t in tokens) else "prefill"
            single = sum(len(t) for t in tokens) <= self.max_step_tokens
            if single:
                with prof.step(phase, [], []):
                    logits = self.step([StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, tokens)],
                                       device_tokens=device_tokens)
                    with prof.scope(op="sampling"):
                        return self._sampler.launch(logits, params, rngs, histories,
                                                    status=kernels.status_word(self.device))
        logits = self.step([StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, tokens)], device_tokens=device_tokens)
        return self._sampler.launch(logits, params, rngs, histories, status=kernels.status_word(self.device))

    def collect(self, handle) -> List[int]:
        """Wait for a launched step and bring its token ids (nothing else) back to the host."""
        return self._sampler.collect(handle)

    def run(self, slots, tokens, params, rngs, histories) -> List[int]:
        """Step the sequences with their next tokens, sample one token each on the GPU, and
        bring the token ids back to the host."""
        return self.collect(self.launch(slots, tokens, params, rngs, histories))

    def generate(self, prompts, max_new_tokens: int = 64, sampling=None, stop_tokens=None,
                 ignore_eos: bool = False, max_batch: int = 64, on_token=None, stats=None, run_ahead: bool = True):
        """Generate for a list of prompts (token id lists).  Returns a list of Completion.
        ``sampling`` is one SamplingParams for all or a list; stop tokens default to the model's."""
        from ..sampling import SamplingParams
        from .generate import Request, generate
        if sampling is None:
            sampling = SamplingParams()
        per = sampling if isinstance(sampling, (list, tuple)) else [sampling] * len(prompts)
        reqs = [Request(list(p), max_new_tokens, sp, stop_tokens, ignore_eos) for p, sp in zip(prompts, per)]
        return generate(self, reqs, default_stop=self.model.spec.stop_tokens, max_batch=max_batch,
                        on_token=on_token, stats=stats, run_ahead=run_ahead)

    # ---- facts for measurement --------------------------------------------------------------------------------
    def kv_bytes_per_token(self) -> int:
        """Bytes of keys and values one token adds over all layers
        (rocml/src/budget/mod.rs:47-59: 2 * layers * kv heads * head size * element size)."""
        n = 0
        for g in self.cache.kv_groups:
            n += (1 if g.req.shared_values else 2) * g.n_entries * g.req.n_kv_heads * g.req.head_dim * g.k.element_size()
        return n
