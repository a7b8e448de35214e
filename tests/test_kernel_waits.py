"""Warps that share named barriers leave their loops together. The bounded waits of the tensor-core kernels can run out for
one warp and not for another; named barriers have no bound, so a warp that left on its own verdict would leave the others
standing at the next one for good. Such a run-out cannot be produced on demand, so the rule is checked where it is written:
between a wait's verdict and the barrier that votes on it, or the barriers that the warps which stay will come to, nothing
leaves the loop."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ascend-moe-engine_b200", "csrc")

# file, first and last text of the role whose warps share barriers
ROLES = {
    "mla_decode_cluster.cu": ("= softmax =", "if (warp == 5 || warp == 6)"),
    "mla_decode_tc.cu": ("= softmax + epilogue warps =", "// ---- teardown"),
    "kv_indexer_tc.cu": ("// ---- epilogue: thread = token", "TmemDealloc"),
}

EVENT = re.compile(
    # a barrier over the role's warps that carries their verdicts, or a warp going through those that the others come to
    r"(?P<vote>NamedBarrierOr\([^;{]*!ok\)|leave_with_the_others\()"
    r"|(?P<wait>\bok = [^;]*Wait\()"               # a bounded wait's verdict
    r"|(?P<leave>\bbreak;|\breturn;|\bfor \([^;{]*;[^;{]*\bok\b[^;{]*;)")


def undecided_exits(text):
    """Places that leave a loop, in source order, after a wait's verdict and before the vote on it."""
    undecided, found = False, []
    for event in EVENT.finditer(text):
        if event.lastgroup == "wait":
            undecided = True
        elif event.lastgroup == "vote":
            undecided = False
        elif undecided:
            found.append(event.group(0))
    return found


@pytest.mark.parametrize("name", ROLES)
def test_warps_that_share_a_barrier_leave_together(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    first, last = ROLES[name]
    start = text.index(first)
    role = re.sub(r"//[^\n]*", "", text[start:text.index(last, start)])
    assert "NamedBarrierOr" in role and re.search(r"\bok = [^;]*Wait\(", role)
    assert undecided_exits(role) == []


def test_the_rule_catches_an_exit_on_a_warps_own_verdict():
    assert undecided_exits("ok = WarpWait(a); if (!ok) break; NamedBarrierOr(1, 128, r);") == ["break;"]
    assert undecided_exits("ok = WarpWait(a); v = NamedBarrierOr(1, 128, r || !ok); if (v) break;") == []
    assert undecided_exits("ok = WarpWait(a); if (!ok) { leave_with_the_others(false); break; }") == []
