"""A ring of stages whose waits may run out: a warp that gave up must not hand its stage back, since the copy into it may still be on its way
and the producer would arm the stage's barrier a second time.  Read off the source; no GPU is needed."""
import os
import re

import rocml_b200

PATH = os.path.join(os.path.dirname(rocml_b200.__file__), "csrc", "decode_layers.cu")


def body(text, head):
    """The braces behind ``head`` and what stands between them."""
    at = text.index("{", text.index(head))
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[at:end]


def test_no_stage_is_handed_back_once_a_wait_has_run_out():
    with open(PATH) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    # what is handed back was looked at behind the wait for its copy
    taken, back = body(text, "bool taken("), body(text, "void give_back(")
    assert taken.index("waits.barrier(&s.full[") < taken.index("return !waits.gave_up()")
    assert "if (lane == 0 && whole) sm100::mbar_arrive(&s.empty[" in back
    compute = body(text, "struct Compute ")
    assert compute.count("&s.full[") == taken.count("&s.full[") == 1 and compute.count("&s.empty[") == 1
    uses = re.findall(r"const bool whole = taken\(at\);|give_back\(at, whole\);", compute)
    assert uses == ["const bool whole = taken(at);", "give_back(at, whole);"] * 2
    # a warp that leaves a wait without success has raised the flag or seen it
    assert "return false" in body(text, "bool barrier(") and "gave_up()) return true" in body(text, "bool over(")
    # and one place arms a stage, behind the wait for it
    room = body(text, "bool room()")
    assert room.index("waits.barrier(&s.empty[") < room.index("mbar_arrive_expect_tx(") and text.count("mbar_arrive_expect_tx(") == 1
