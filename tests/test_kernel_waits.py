"""Source rules of the solver kernels' bounded waits that no run can show
without hanging a GPU when they are broken."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOLVER = os.path.join(ROOT, "mille-feillue_b200", "csrc", "solver.cu")


def _block(text, start):
    """The braced block that opens at or after `start`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i + 1:j]
    raise AssertionError("unbalanced braces")


def test_producer_warp_leaves_its_loop_together():
    """The copy ring's producer runs as a whole warp with warp barriers in its loop, and each lane's wait has its
    own time limit: a lane may leave only on a vote of all lanes."""
    text = re.sub(r"//[^\n]*", "", open(SOLVER).read())
    producers = [_block(text, m.end()) for m in re.finditer(r"if \(w == PRODUCER_WARP\)", text)]
    assert len(producers) == 2  # the streaming ring, the resident kernels
    for body in producers:
        assert "__syncwarp()" in body
        for m in re.finditer(r"\b(?:break|return)\b", body):
            line = body[body.rfind("\n", 0, m.start()) + 1:m.start()]
            assert "__all_sync(0xffffffffu" in line, line
