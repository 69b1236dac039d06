"""Short prompts replayed from captured graphs: padded up to a bucket, against the plain implementation, the first time and again."""
import pytest
import torch

from tiny_models import CONFIGS, prompt, write_model

pytestmark = pytest.mark.gpu

TOL = 2.5e-2        # as the other tests of bfloat16 layers


def rel_err(got, want):
    want = want.to(torch.float64)
    return float(((got.double().cpu() - want).abs() / want.abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)).max())


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    from plain_qwen3 import PlainQwen3
    config = {**CONFIGS["E"], "use_sliding_window": False, "layer_types": ["full_attention"] * 2}
    folder = str(tmp_path_factory.mktemp("prompt_graphs"))
    write_model(folder, config, seed=17, std=0.05)
    return config, folder, PlainQwen3(folder, dtype=torch.float64)


@pytest.mark.parametrize("use_graphs", [True, False])
def test_short_prompts(model, use_graphs):
    """Lengths at the edges of the buckets, one sequence and several, new sequences and pieces behind a cache, wanted places in
    any number (none too), a prompt too long for a graph, and more buckets than are kept."""
    from rocml_b200 import Engine, StepEntry, kernels
    from rocml_b200.engine.engine import PROMPT_GRAPHS
    config, folder, plain = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=2048, max_slots=6, use_graphs=use_graphs)
    batches = [[2], [15], [16], [17], [64, 1], [65], [3, 40, 20], [1, 2, 60, 9, 30], [128], [129, 100], [256], [250, 7], [2], [61], [60], [62, 2]]
    for n, lens in enumerate(batches * 2):
        ids = [prompt(1000 + 37 * n + i, m + 30, config["vocab_size"]) for i, m in enumerate(lens)]
        slots = [eng.new_sequence() for _ in ids]
        want = [plain.logits(x) for x in ids]
        places = [[m - 1] if i % 2 == 0 else [0, m - 1] for i, m in enumerate(lens)]
        got = eng.step([StepEntry(s, x[:m], w) for s, x, m, w in zip(slots, ids, lens, places)]).clone()
        assert rel_err(got, torch.cat([x[w] for x, w in zip(want, places)])) < TOL, lens
        assert eng.step([StepEntry(s, x[m:m + 7], []) for s, x, m in zip(slots, ids, lens)]) is None
        got = eng.step([StepEntry(s, x[m + 7:m + 29], [21, 3]) for s, x, m in zip(slots, ids, lens)]).clone()
        assert rel_err(got, torch.cat([x[[m + 28, m + 10]] for x, m in zip(want, lens)])) < TOL, lens
        got = eng.step([StepEntry(s, x[m + 29:m + 30], [0]) for s, x, m in zip(slots, ids, lens)]).clone()
        assert rel_err(got, torch.cat([x[[m + 29]] for x, m in zip(want, lens)])) < TOL, lens
        for s in slots:
            eng.release(s)
        assert len(eng._prompt_graphs) <= (PROMPT_GRAPHS if use_graphs else 0)
    kernels.check_status("cuda:0")
    assert bool(eng._prompt_graphs) == use_graphs


def test_pieces_that_replay_one_graph(model):
    """A step cut into pieces of one size: every piece's logits are its own, though they replay the same graph."""
    from rocml_b200 import Engine, StepEntry
    config, folder, plain = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1024, max_slots=3, max_step_tokens=64)
    ids = prompt(5, 330, config["vocab_size"])
    want = plain.logits(ids)
    for _ in range(2):
        slot = eng.new_sequence()
        assert rel_err(eng.step([StepEntry(slot, ids, list(range(330)))]), want) < TOL
        eng.release(slot)


def test_pieces_that_replay_one_graph_with_one_place_each(model):
    """As above with one wanted place a piece, which is what has a graph."""
    from rocml_b200 import Engine, StepEntry
    config, folder, plain = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1024, max_slots=3, max_step_tokens=64)
    ids = prompt(6, 330, config["vocab_size"])
    want = plain.logits(ids)[[5, 100, 130, 200, 319, 329]]
    for _ in range(2):
        slot = eng.new_sequence()
        assert rel_err(eng.step([StepEntry(slot, ids, [5, 100, 130, 200, 319, 329])]), want) < TOL
        eng.release(slot)
    assert len(eng._prompt_graphs) == 1          # (of 64 tokens; the rest of ten has come twice)


def test_a_size_that_comes_back_is_captured_and_answers_alike(model):
    """No capture for a size seen three times; the same bits before, when it is captured and from then on; never more graphs than
    max_graphs, and sizes that take turns are not captured over and over."""
    from rocml_b200 import Engine, StepEntry
    config, folder, _ = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1024, max_slots=3, max_graphs=2)
    captured, capture = [], eng._capture
    eng._capture = lambda g, batch: captured.append(batch.n_tokens) or capture(g, batch)
    first = {}
    for turn in range(7):
        for n in (2, 30, 61, 100, 200):
            slot = eng.new_sequence()
            got = eng.step([StepEntry(slot, prompt(n, n, config["vocab_size"]), [n - 1])]).clone()
            eng.release(slot)
            assert torch.equal(first.setdefault(n, got), got), (turn, n)
        assert len(captured) == (0 if turn < 3 else 2) and len(eng._prompt_graphs) == len(captured)


def test_graphs_of_prompts_take_only_memory_that_is_left(model, monkeypatch):
    """An engine that just fits keeps none, and is not refused for them."""
    from rocml_b200 import Engine, MemoryBudget, StepEntry
    config, folder, plain = model
    refused = None
    for spare in (0, 1, 2, 3):
        monkeypatch.undo()
        eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=1024, max_slots=3)
        each = eng.model.workspace_bytes(256, 4)
        if refused is None:
            # the least free memory that is accepted, found through the refusals
            lo, hi = 0, 4 << 30
            while hi - lo > 1:
                mid = (lo + hi) // 2
                monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a, m=mid: (m, 180 << 30))
                try:
                    eng._check_budget(1024, 3)
                    hi = mid
                except MemoryBudget:
                    lo = mid
            refused = hi
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (refused + spare * each, 180 << 30))
        assert eng._check_budget(1024, 3) == spare
        eng = Engine(eng.model, max_tokens=1024, max_slots=3)
        ids = prompt(8, 50, config["vocab_size"])
        for _ in range(5):
            slot = eng.new_sequence()
            assert rel_err(eng.step([StepEntry(slot, ids, [49])]), plain.logits(ids)[-1:]) < TOL
            eng.release(slot)
        assert len(eng._prompt_graphs) == min(spare, 1)
