"""A ring of stages whose waits may run out: warps that give up hand their stages back though the copies may still be on their way, so the
producer looks at the flag behind every wait for a free stage, before it arms the stage's barrier.  Read off the source; no GPU is needed."""
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


def test_no_stage_is_armed_once_a_wait_has_run_out():
    with open(PATH) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    room = body(text, "bool room()")
    waited, armed = room.index("waits.barrier("), room.index("mbar_arrive_expect_tx(")
    looked = [m.start() for m in re.finditer(r"waits\.gave_up\(\)", room)]
    assert any(waited < at < armed for at in looked)
    assert text.count("mbar_arrive_expect_tx(") == 1          # nothing else arms a stage
    # and the warps that compute raise or read the flag before they hand a stage back without success
    assert "return false" in body(text, "bool barrier(") and "gave_up()) return true" in body(text, "bool over(")
