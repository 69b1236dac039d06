"""Which sizes of short prompts are captured: host logic, no GPU needed."""
import random
from collections import OrderedDict

import pytest

from rocml_b200.engine.engine import GraphSizes, _bucket, _prompt_graph_tokens, _prompt_pads


def serve(sizes, stream):
    """(captures, replays) of a stream of sizes."""
    graphs, captures, replays = OrderedDict(), 0, 0
    for s in stream:
        if sizes.due(s, graphs):
            if s in graphs:
                replays += 1
                graphs.move_to_end(s)
            else:
                while len(graphs) >= sizes.kept:
                    graphs.popitem(last=False)
                graphs[s] = True
                captures += 1
        sizes.note(s)
        assert len(graphs) <= sizes.kept
    return captures, replays


def test_a_size_is_captured_when_it_has_come_often_enough():
    assert serve(GraphSizes(4, 2), [1, 2, 3, 4, 5]) == (0, 0)
    assert serve(GraphSizes(4, 2), [1, 1, 1, 2]) == (1, 1)
    assert serve(GraphSizes(4, 4), [1, 2, 1, 2, 1, 2]) == (0, 0)
    assert serve(GraphSizes(4, 4), [1] * 6) == (1, 2)
    assert serve(GraphSizes(0, 4), [1] * 9) == (0, 0)


@pytest.mark.parametrize("times", [2, 4, 12])
def test_sizes_that_take_turns_do_not_drive_one_another_out(times):
    captures, replays = serve(GraphSizes(4, times), list(range(5)) * 40)
    assert captures == 4 and replays >= 4 * (40 - times)


@pytest.mark.parametrize("times", [4, 12])
@pytest.mark.parametrize("seed", range(4))
def test_captures_are_few_in_a_mixed_stream(seed, times):
    """Twelve sizes at random, eight kept: a capture for each of the kept and now and then one more."""
    rng = random.Random(seed)
    stream = [rng.randrange(12) for _ in range(800)]
    captures, replays = serve(GraphSizes(8, times), stream)
    assert captures <= 8 + 800 // (8 * times) and replays > 300


def test_what_was_common_gives_way():
    captures, replays = serve(GraphSizes(2, 4), [1, 2] * 500 + [3, 4] * 500)
    assert captures == 4 and replays > 1000


def test_padded_sizes():
    for n in range(2, 257):
        for b in (1, 2, 3, n // 2, n):
            if not 1 <= b <= n:
                continue
            for w in {0, 1, b}:
                t, seqs, want, longest, ctx, decode = _prompt_pads(n, b, w, n + 5000)
                assert t >= n and seqs >= b and want >= w and longest == t and ctx >= n + 5000 and not decode
                assert (w == 0) == (want == 0)
                assert t <= _bucket(n, 64) and seqs <= _bucket(b, 8) and want <= _bucket(n, 64)       # what a plain step's buffers hold
            assert _prompt_pads(n, b, _bucket(b) + 1, n) is None
    assert len({_prompt_pads(n, 1, 1, n) for n in range(2, 257)}) == 5


def test_wide_layers_have_shorter_graphs_or_none():
    assert [_prompt_graph_tokens(n << 20) for n in (1, 96, 128, 129, 256, 368, 400, 401, 940)] == [256] * 3 + [128] * 4 + [0, 0]
