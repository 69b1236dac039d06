"""The memory of captured graphs: shared while there is a graph, given back, and bounded over many captures."""
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
    folder = str(tmp_path_factory.mktemp("graph_memory"))
    write_model(folder, config, seed=23, std=0.05)
    return config, folder, PlainQwen3(folder, dtype=torch.float64)


def decode(eng, ids, steps=3):
    """The logits of ``steps`` single tokens behind the rest of each of ``ids``, [sequences][steps, vocab]."""
    from rocml_b200 import StepEntry
    slots = [eng.new_sequence() for _ in ids]
    eng.step([StepEntry(s, x[:-steps], []) for s, x in zip(slots, ids)])
    rows = [eng.step([StepEntry(s, [x[t - steps]], [0]) for s, x in zip(slots, ids)]).clone() for t in range(steps)]
    for s in slots:
        eng.release(s)
    return torch.stack(rows, dim=1)


def test_one_graph_is_kept_and_another_size_takes_its_place(model):
    """max_graphs=1: with the only graph goes the memory that it shared, and the next size's graph begins anew."""
    from rocml_b200 import Engine
    config, folder, plain = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=2048, max_slots=4, max_graphs=1)
    for n in (1, 3, 1, 2, 1):
        ids = [prompt(40 + n + i, 300 + i, config["vocab_size"]) for i in range(n)]
        got = decode(eng, ids)
        for i, x in enumerate(ids):
            assert rel_err(got[i], plain.logits(x)[-3:]) < TOL


def test_memory_stops_growing_over_many_captures(model):
    """More sizes than are kept, over and over: what earlier graphs held is used again."""
    from rocml_b200 import Engine
    config, folder, _ = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=4096, max_slots=8, max_graphs=2)
    batches = [[prompt(60 + i, 300 * k + i, config["vocab_size"]) for i in range(n)] for n in (1, 2, 4, 8) for k in (1, 2) if n * k <= 8]
    held = []
    for _ in range(8):
        for ids in batches:
            decode(eng, ids)
        torch.cuda.synchronize()
        held.append(torch.cuda.memory_reserved())
    assert eng.graphs_captured >= 8 * 6 and held[-1] == held[2], held


@pytest.mark.parametrize("failures", [1, 2])
def test_a_capture_that_runs_out_of_memory_loses_no_step(model, monkeypatch, failures):
    """The memory that the allocator holds goes back and the capture is tried again; if that does not help, the size runs without a
    graph.  Every step gives its logits."""
    from rocml_b200 import Engine
    config, folder, plain = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=2048, max_slots=4)
    forward, left, emptied = eng.model.forward, [failures], []

    def short_of_memory(batch, cache):
        if batch.capturing and left[0] > 0:
            left[0] -= 1
            raise torch.OutOfMemoryError("out of memory (made up)")
        return forward(batch, cache)
    monkeypatch.setattr(eng.model, "forward", short_of_memory)
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: emptied.append(1))
    ids = [prompt(90 + i, 310 + i, config["vocab_size"]) for i in range(2)]
    for _ in range(2):
        got = decode(eng, ids)
        for i, x in enumerate(ids):
            assert rel_err(got[i], plain.logits(x)[-3:]) < TOL
    assert left == [0] and len(emptied) == failures and eng.graphs_captured == 2 - failures


def test_another_thread_may_allocate_during_captures(model):
    """Fresh device memory for another thread while sizes are captured: neither disturbs the other."""
    import threading
    import time
    from rocml_b200 import Engine
    config, folder, plain = model
    eng = Engine.from_folder(folder, dtype="bfloat16", max_tokens=4096, max_slots=8, max_graphs=1)
    stop, failed, held = threading.Event(), [], []

    def allocate():
        try:
            while not stop.is_set() and len(held) < 500:
                held.append(torch.empty(32 << 20, dtype=torch.uint8, device="cuda:0"))       # (more than is cached: from the device each time)
                time.sleep(0.001)
        except Exception as e:  # noqa: BLE001
            failed.append(e)
    other = threading.Thread(target=allocate)
    other.start()
    try:
        for n in (1, 2, 4, 8) * 4:
            ids = [prompt(120 + n + i, 300 + i, config["vocab_size"]) for i in range(n)]
            got = decode(eng, ids)
            for i, x in enumerate(ids[:1]):
                assert rel_err(got[i], plain.logits(x)[-3:]) < TOL
    finally:
        stop.set()
        other.join()
    assert not failed and len(held) > 50, failed
    held.clear()
    torch.cuda.empty_cache()
