"""The persistent kernel of a decode step's layers against the same layers in float64: edges of its units, passes over k, stages
of keys and parts of a sequence; then through the engine; and a wait that runs out."""
import pytest
import torch

from tiny_models import CONFIGS, prompt, write_model

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
# Rows pass through bfloat16 about six times a layer (2^-9 of a value each time); entries are compared with their row's largest, as in the
# other tests of bfloat16 layers.
TOL = 2.5e-2


def make(T, H, inter, nq, nkv, lens, layers=2, norms=torch.bfloat16, rope=True, seed=1):
    g = torch.Generator(device=DEV).manual_seed(seed)

    def rnd(*shape, std=1.0, dtype=torch.bfloat16, centre=0.0):
        return (torch.randn(shape, generator=g, device=DEV) * std + centre).to(dtype)
    pages = sum((n + 63) // 64 for n in lens) + 1
    table = torch.full((T + 1, max((n + 63) // 64 for n in lens) + 1), -1, dtype=torch.int32)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(seed)).tolist()
    for t, n in enumerate(lens):
        for i in range((n + 63) // 64):
            table[t, i] = order.pop()
    out = []
    for _ in range(layers):
        vec = lambda n: rnd(n, std=0.1, dtype=norms, centre=1.0)  # noqa: E731
        out.append(dict(q=rnd(nq * 128, H, std=H ** -0.5), k=rnd(nkv * 128, H, std=H ** -0.5), v=rnd(nkv * 128, H, std=H ** -0.5),
                        o=rnd(H, nq * 128, std=(nq * 128) ** -0.5), gate=rnd(inter, H, std=2 * H ** -0.5), up=rnd(inter, H, std=2 * H ** -0.5),
                        down=rnd(H, inter, std=inter ** -0.5), n1=vec(H), n2=vec(H), qn=vec(128), kn=vec(128),
                        ck=rnd(pages, nkv, 64, 128), cv=rnd(pages, nkv, 64, 128)))
    # behind a sequence's last key a page holds anything
    for L in out:
        for t, n in enumerate(lens):
            if n % 64:
                L["ck"][table[t, n // 64], :, n % 64:] = float("nan")
                L["cv"][table[t, n // 64], :, n % 64:] = float("inf")
    x = rnd(T, H, dtype=torch.float32)
    angle = torch.rand((T, 64), generator=g, device=DEV) * 6.0
    cs = torch.stack([angle.cos(), angle.sin()], dim=-1).contiguous() if rope else None
    return out, x, table.to(DEV), cs


def rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps) * w.double()


def want(layers, x, table, cs, lens, nq, nkv, eps, heads_normed):
    """(the stream, new keys and values of every layer) in float64."""
    x = x.double()
    new = []
    for L in layers:
        h = rms(x, L["n1"], eps)
        q, k, v = (h @ L[n].double().T for n in "qkv")
        q, k, v = q.view(len(lens), nq, 128), k.view(len(lens), nkv, 128), v.view(len(lens), nkv, 128)
        if heads_normed:
            q, k = rms(q, L["qn"], eps), rms(k, L["kn"], eps)
        if cs is not None:
            c, s = cs[..., 0].double()[:, None], cs[..., 1].double()[:, None]
            q, k = (torch.cat([a[..., :64] * c - a[..., 64:] * s, a[..., :64] * s + a[..., 64:] * c], dim=-1) for a in (q, k))
        o = torch.zeros((len(lens), nq * 128), dtype=torch.float64, device=DEV)
        for t, n in enumerate(lens):
            if n == 0:
                continue
            ids = table[t, : (n + 63) // 64].long()
            keys = L["ck"][ids].double().transpose(0, 1).reshape(nkv, -1, 128)[:, : n - 1]
            vals = L["cv"][ids].double().transpose(0, 1).reshape(nkv, -1, 128)[:, : n - 1]
            keys, vals = torch.cat([keys, k[t][:, None]], dim=1), torch.cat([vals, v[t][:, None]], dim=1)
            keys, vals = (a.repeat_interleave(nq // nkv, dim=0) for a in (keys, vals))
            p = torch.softmax((keys @ q[t][:, :, None])[..., 0] * 128 ** -0.5, dim=-1)
            o[t] = (p[:, None] @ vals).flatten()
        new.append((k, v))
        x = x + o @ L["o"].double().T
        h = rms(x, L["n2"], eps)
        x = x + (torch.nn.functional.silu(h @ L["gate"].double().T) * (h @ L["up"].double().T)) @ L["down"].double().T
    return x, new


def run(layers, x, table, cs, lens, nq, nkv, inter, eps, heads_normed, splits, wait_limit=0):
    from rocml_b200 import kernels
    T, H = x.shape
    resid = x.clone()
    args = []
    for i, L in enumerate(layers):
        pairs = torch.stack([L["gate"].view(-1, 16, H), L["up"].view(-1, 16, H)], dim=1).reshape(2 * inter, H).contiguous()
        args.append((torch.cat([L["q"], L["k"], L["v"]]).contiguous(), L["o"], pairs, L["down"], L["n2"],
                     layers[i + 1]["n1"] if i + 1 < len(layers) else None, L["qn"] if heads_normed else None,
                     L["kn"] if heads_normed else None, L["ck"].clone(), L["cv"].clone(), eps, eps))
    slots = torch.tensor([t if n else -1 for t, n in enumerate(lens)], dtype=torch.int32, device=DEV)
    kernels.decode_layers(resid, layers[0]["n1"], args, nq, nkv, inter, eps, 128 ** -0.5, cs, slots,
                          torch.tensor(lens, dtype=torch.int32, device=DEV), table, splits, wait_limit)
    return resid, args


CASES = [
    # lens, H, inter, nq, nkv, splits: one token and no old keys; keys short of a stage, a stage, one more, pages; several parts
    ([1], 64, 64, 1, 1, 1),
    ([16, 17, 18, 64, 65, 66, 2, 129], 192, 320, 16, 2, 1),             # all tokens of a tile; 8 heads a group
    ([300], 512, 1216, 16, 8, 5),                                       # parts, and five pages for them
    ([1, 700, 65], 576, 1088, 6, 3, 4),                                 # a sequence with fewer pages than parts; k 64 past a stage
    ([40, 0, 100, 0], 1024, 192, 5, 5, 2),                              # places without a sequence; four units in work
    ([10 + 37 * i for i in range(8)], 320, 512, 14, 2, 1),              # seven heads a group
    ([200 - 11 * i for i in range(8)], 2112, 704, 12, 4, 3),
    ([77, 5], 4160, 4672, 33, 33, 1),                                   # two passes over k; 33 heads
    ([3] * 8, 4608, 8256, 40, 8, 1),                                   # two and three passes
    ([130, 7, 64], 5120, 25600, 64, 8, 2),                              # more units a block than are kept: groups
    ([900], 768, 2560, 8, 8, 1),                                        # more stages of keys than the ring has
    ([600, 1], 192, 320, 8, 2, 9),                                      # parts that are merged in two rounds of eight, the second ragged
    ([2300], 256, 512, 8, 4, 18),                                       # three rounds
    ([3000, 800, 100, 17], 512, 1216, 16, 4, 9),                        # lengths as unequal as they come, with parts that have no page
    ([1040], 128, 192, 2, 1, 16),                                       # two whole rounds
]


def check(lens, H, inter, nq, nkv, splits, case, layers=2):
    from rocml_b200 import kernels
    eps, normed, rope = 1e-6, case % 3 != 2, case % 4 != 3
    layers, x, table, cs = make(len(lens), H, inter, nq, nkv, lens, layers, torch.float32 if case % 2 else torch.bfloat16, rope, seed=case)
    ref, new = want(layers, x, table, cs, lens, nq, nkv, eps, normed)
    got, args = run(layers, x, table, cs, lens, nq, nkv, inter, eps, normed, splits)
    again, _ = run(layers, x, table, cs, lens, nq, nkv, inter, eps, normed, splits)
    kernels.check_status(DEV)
    live = torch.tensor([n > 0 for n in lens], device=DEV)
    assert torch.isfinite(got).all() and torch.equal(got, again)
    err = ((got.double() - ref).abs() / ref.abs().amax(dim=-1, keepdim=True))[live].max()
    assert err < TOL, float(err)
    for L, a, (k, v) in zip(layers, args, new):
        for old, now, rows in ((L["ck"], a[8], k), (L["cv"], a[9], v)):
            expected = old.clone()
            for t, n in enumerate(lens):
                if n:
                    page, r = int(table[t, (n - 1) // 64]), (n - 1) % 64
                    assert float((now[page, :, r].double() - rows[t]).abs().max()) < TOL * float(rows[t].abs().max())
                    expected[page, :, r] = now[page, :, r]
            assert torch.equal(now.view(torch.int16), expected.view(torch.int16))          # and nothing else in the cache


@pytest.mark.parametrize("case", range(len(CASES)))
def test_layers_against_float64(case):
    check(*CASES[case], case)


def test_more_layers_than_a_launch_takes():
    """40 layers: two launches, the second of which takes the first's rows up.  Errors of a layer add up at random: sqrt(20) times two layers'."""
    global TOL
    keep, TOL = TOL, TOL * 4.5
    try:
        check([70, 3], 192, 256, 4, 2, 1, 4, layers=40)
    finally:
        TOL = keep


def test_a_wait_that_runs_out_is_reported():
    """A limit of one clock cycle: the waits give up, the kernel ends, the status word says why, and the next call is sound."""
    from rocml_b200 import KernelError, kernels
    lens, H, inter, nq, nkv = [90, 200], 512, 1216, 16, 8
    layers, x, table, cs = make(2, H, inter, nq, nkv, lens)
    run(layers, x, table, cs, lens, nq, nkv, inter, 1e-6, True, 2, wait_limit=1)
    with pytest.raises(KernelError, match="wait"):
        kernels.check_status(DEV)
    got, _ = run(layers, x, table, cs, lens, nq, nkv, inter, 1e-6, True, 2)
    kernels.check_status(DEV)
    ref, _ = want(layers, x, table, cs, lens, nq, nkv, 1e-6, True)
    assert float(((got.double() - ref).abs() / ref.abs().amax(dim=-1, keepdim=True)).max()) < TOL


def test_a_step_whose_waits_run_out_ends_soon():
    """Thirty layers, many rounds of the ring each: once a wait has run out the others give up at their next look, so the kernel ends in no more than a few
    steps' time (a step takes about 1 ms)."""
    from rocml_b200 import KernelError, kernels
    lens, H, inter, nq, nkv = [90, 200], 2048, 6144, 16, 8
    layers, x, table, cs = make(2, H, inter, nq, nkv, lens)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    real, times = kernels.decode_layers, []

    def often(resid, first, args, *rest):
        # (thirty layers: the two alternate, the last has no next norm)
        args = [args[0]] * 29 + [args[1]]
        a.record()
        real(resid, first, args, *rest)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    kernels.decode_layers = often
    try:
        for limit in (0, 1, 1):
            run(layers, x, table, cs, lens, nq, nkv, inter, 1e-6, True, 2, wait_limit=limit)
            if limit:
                with pytest.raises(KernelError, match="wait"):
                    kernels.check_status(DEV)
            else:
                kernels.check_status(DEV)
    finally:
        kernels.decode_layers = real
    assert times[2] < 20.0, times


@pytest.mark.parametrize("graphs", [False, True])
def test_decode_through_the_engine(tmp_path, monkeypatch, graphs):
    """Sequences of unequal lengths decoded together, two ending early; the same with the layers' own kernels, which a model too
    narrow for the one kernel always takes."""
    from plain_qwen3 import PlainQwen3
    from rocml_b200 import Engine, StepEntry, kernels
    config = {**CONFIGS["E"], "use_sliding_window": False, "layer_types": ["full_attention"] * 2, "num_attention_heads": 16,
              "num_key_value_heads": 2, "intermediate_size": 1216}
    folder = str(tmp_path / "m")
    write_model(folder, config, seed=9, std=0.05)
    plain = PlainQwen3(folder, dtype=torch.float64)
    calls = []
    real = kernels.decode_layers
    monkeypatch.setattr(kernels, "decode_layers", lambda *a, **k: calls.append(a[0].shape[0]) or real(*a, **k))
    ids = [prompt(70 + i, n, config["vocab_size"]) for i, n in enumerate((400, 50, 40))]
    starts = [340, 20, 1]
    for on in ("1", "0"):
        monkeypatch.setenv("RB_DECODE_LAYERS", on)
        calls.clear()
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1024, use_graphs=graphs)
        slots = [eng.new_sequence() for _ in ids]
        eng.step([StepEntry(s, x[:n], []) for s, x, n in zip(slots, ids, starts)])
        rows = [[] for _ in ids]
        for t in range(60):
            live = [j for j in range(3) if starts[j] + t < len(ids[j])]
            out = eng.step([StepEntry(slots[j], [ids[j][starts[j] + t]], [0]) for j in live])
            for r, j in enumerate(live):
                rows[j].append(out[r].clone())
        kernels.check_status(DEV)
        assert bool(calls) == (on == "1")
        for x, n, got in zip(ids, starts, rows):
            ref = plain.logits(x)[n: n + len(got)].to(torch.float64)
            err = ((torch.stack(got).double().cpu() - ref).abs() / ref.abs().amax(dim=-1, keepdim=True)).max()
            assert float(err) < TOL, float(err)


@pytest.mark.parametrize("graphs", [False, True])
def test_lengths_decide_which_way_a_step_goes(tmp_path, monkeypatch, graphs):
    """One long sequence among seven short ones runs layer by layer, a batch of a length as one kernel, in one engine after another."""
    from plain_qwen3 import PlainQwen3
    from rocml_b200 import Engine, StepEntry, kernels
    config = {**CONFIGS["E"], "use_sliding_window": False, "layer_types": ["full_attention"] * 2, "num_attention_heads": 16,
              "num_key_value_heads": 2, "intermediate_size": 1216, "max_position_embeddings": 2048}
    folder = str(tmp_path / "m")
    write_model(folder, config, seed=13, std=0.05)
    plain = PlainQwen3(folder, dtype=torch.float64)
    calls = []
    real = kernels.decode_layers
    monkeypatch.setattr(kernels, "decode_layers", lambda *a, **k: calls.append(a[0].shape[0]) or real(*a, **k))
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=4096, use_graphs=graphs)
    for lens, taken in (([600] + [20] * 7, False), ([200] * 8, True), ([600], True), ([599] + [21] * 7, False)):
        calls.clear()
        ids = [prompt(70 + i, n, config["vocab_size"]) for i, n in enumerate(lens)]
        slots = [eng.new_sequence() for _ in ids]
        eng.step([StepEntry(s, x[:-3], []) for s, x in zip(slots, ids)])
        rows = torch.stack([eng.step([StepEntry(s, [x[t]], [0]) for s, x in zip(slots, ids)]).clone() for t in (-3, -2, -1)], dim=1)
        assert (bool(calls) == taken) or (graphs and not calls), lens          # (a replay of an earlier capture calls nothing)
        for x, got in zip(ids, rows):
            ref = plain.logits(x)[-3:].to(torch.float64)
            assert float(((got.double().cpu() - ref).abs() / ref.abs().amax(dim=-1, keepdim=True)).max()) < TOL
        for s in slots:
            eng.release(s)
    kernels.check_status("cuda:0")


def test_what_the_kernel_declines_leaves_the_stream_alone():
    """A weight off 16 bytes, and more query heads a key/value head than a block takes."""
    from rocml_b200 import kernels
    lens, H, inter = [30, 9], 512, 1216
    for nq, nkv, shift in ((16, 2, 1), (18, 2, 0)):
        layers, x, table, cs = make(2, H, inter, nq, nkv, lens)
        for L in layers:
            w = torch.empty(H * nq * 128 + 1, dtype=torch.bfloat16, device=DEV)[shift:][:H * nq * 128].view(H, nq * 128)
            L["o"] = w.copy_(L["o"])
        took = []
        real, kernels.decode_layers = kernels.decode_layers, lambda *a: took.append(real(*a))
        try:
            got, args = run(layers, x, table, cs, lens, nq, nkv, inter, 1e-6, True, 1)
        finally:
            kernels.decode_layers = real
        assert took == [False] and torch.equal(got, x)
        for L, a in zip(layers, args):
            assert torch.equal(a[8].view(torch.int16), L["ck"].view(torch.int16)) and torch.equal(a[9].view(torch.int16), L["cv"].view(torch.int16))


@pytest.mark.parametrize("graphs", [False, True])
def test_a_step_that_the_kernel_declines_runs_layer_by_layer(tmp_path, monkeypatch, graphs):
    """The library refuses the step: the answers are those of the layers' own kernels, bit for bit."""
    from rocml_b200 import Engine, StepEntry, kernels
    config = {**CONFIGS["E"], "use_sliding_window": False, "layer_types": ["full_attention"] * 2, "num_attention_heads": 16,
              "num_key_value_heads": 2, "intermediate_size": 1216}
    folder = str(tmp_path / "m")
    write_model(folder, config, seed=9, std=0.05)
    ids = prompt(70, 40, config["vocab_size"])
    rows, refused = {}, []
    monkeypatch.setattr(kernels._lib(), "rb_decode_layers", lambda *a: refused.append(1) or 10003)
    for on in ("1", "0"):
        monkeypatch.setenv("RB_DECODE_LAYERS", on)
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1024, use_graphs=graphs)
        slot = eng.new_sequence()
        eng.step([StepEntry(slot, ids[:35], [])])
        rows[on] = torch.stack([eng.step([StepEntry(slot, [i], [0])]).clone() for i in ids[35:]])
        assert bool(refused) == (on == "1") or on == "0"
    assert torch.equal(rows["1"], rows["0"])


def test_a_long_sequence_through_the_engine(tmp_path, monkeypatch):
    """One sequence of some 2,300 tokens: its pages are taken in more than eight parts."""
    from plain_qwen3 import PlainQwen3
    from rocml_b200 import Engine, StepEntry, kernels
    config = {**CONFIGS["E"], "use_sliding_window": False, "layer_types": ["full_attention"] * 2, "num_attention_heads": 16,
              "num_key_value_heads": 2, "intermediate_size": 1216, "max_position_embeddings": 4096}
    folder = str(tmp_path / "m")
    write_model(folder, config, seed=11, std=0.05)
    ids = prompt(3, 2310, config["vocab_size"])
    ref = PlainQwen3(folder, dtype=torch.float64).logits(ids)[-8:].to(torch.float64)
    parts = []
    real = kernels.decode_layers
    monkeypatch.setattr(kernels, "decode_layers", lambda *a, **k: parts.append(a[12]) or real(*a, **k))
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=2560)
    slot = eng.new_sequence()
    eng.step([StepEntry(slot, ids[:-8], [])])
    got = torch.cat([eng.step([StepEntry(slot, [i], [0])]).clone() for i in ids[-8:]])
    kernels.check_status("cuda:0")
    assert parts and min(parts) > 8
    assert float(((got.double().cpu() - ref).abs() / ref.abs().amax(dim=-1, keepdim=True)).max()) < TOL
