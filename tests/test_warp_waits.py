"""Bounded waits by whole warps, checked in the source on the CPU.

A bounded mbarrier wait can give up. If each lane of a warp decides that for itself, one lane can
give up in the moment in which another sees the phase complete; the first leaves, and the other
waits for it in the next warp-wide instruction (elect.sync, __syncwarp, tcgen05.ld) for good: the
wait that was to end in an error status ends in a hang. It takes a stall of a second and a
coincidence, so no test on a GPU can show it (or may). The source has to keep to this: a wait that one
lane alone makes (inside `if (lane == 0)`, or elected) decides alone; a warp's wait is
mbar_wait_warp() (in the column sums staged_wait_warp()), or every lane goes on whatever it found,
and they agree by __all_sync() before any of them leaves.
"""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).parent.parent / "flint_b200" / "csrc"


def waits(text, name):
    """(statement with the wait, headers of the blocks around it) of every call of `name`."""
    text = re.sub(r"//[^\n]*", "", text)
    for call in re.finditer(rf"\b{name}\(", text):
        if text[:call.start()].rstrip().endswith("bool"):
            continue                                    # its definition
        headers, depth = [], 0
        for at in range(call.start(), -1, -1):
            if text[at] == "}":
                depth += 1
            elif text[at] == "{":
                if depth == 0:
                    start = max(text.rfind(c, 0, at) for c in ";{}")
                    headers.append(" ".join(text[start + 1:at].split()))
                else:
                    depth -= 1
        start = max(text.rfind(c, 0, call.start()) for c in ";{}")
        yield " ".join(text[start + 1:text.index(";", call.start())].split()), headers


@pytest.mark.parametrize("source, name", [("gemm.cu", "sm100::mbar_wait"), ("attention.cu", "sm100::mbar_wait"),
                                          ("reductions.cu", "staged_wait")])
def test_lanes_of_a_warp_do_not_decide_for_themselves(source, name):
    found = list(waits((CSRC / source).read_text(), name))
    assert found
    for statement, headers in found:
        alone = any(re.search(r"\blane == 0\b|if \(sm100::elect_one\(\)", header) for header in headers)
        agreed = re.search(r"\b(there|ok) = .*(&& (there|ok))?$", statement) and "if (" not in statement
        assert alone or agreed, statement


@pytest.mark.parametrize("source, name, least", [("gemm.cu", "sm100::mbar_wait_warp", 2),
                                                 ("attention.cu", "sm100::mbar_wait_warp", 11),
                                                 ("reductions.cu", "staged_wait_warp", 1)])
def test_the_warps_waits_are_found(source, name, least):
    assert len(list(waits((CSRC / source).read_text(), name))) >= least


def test_lanes_that_go_along_agree_before_the_next_step():
    text = (CSRC / "attention.cu").read_text()
    loops = re.findall(r"bool there = sm100.*?\n( *)ok = __all_sync\(0xffffffffu, there\);\n\1?\s*\}", text, re.S)
    assert len(loops) == len(re.findall(r"\bbool there = sm100", text)) == 2


def test_forward_softmax_warps_leave_their_loops_only_at_the_end():
    """Two warps share the rows of a query tile and meet at a barrier without a limit."""
    text = (CSRC / "attention.cu").read_text()
    begin = text.index("bool there = true;")
    loops = re.sub(r"//[^\n]*", "", text[begin:text.index("fb::dependency_release()", begin)])
    assert loops.count("quadrant_sync(pair_barrier)") == 3
    assert not re.search(r"\b(break|continue|return)\b", loops)
    assert "if (there && stores" in loops


@pytest.mark.parametrize("source, function", [("sm100.cuh", "mbar_wait_warp"), ("reductions.cu", "staged_wait_warp")])
def test_a_warps_wait_has_one_outcome(source, function):
    text = (CSRC / source).read_text()
    body = text[re.search(rf"bool {function}\(", text).start():]
    body = body[:body.index("\n}\n")]
    for outcome in re.finditer(r"return (true|false);", body):
        condition = body[body.rfind("if (", 0, outcome.start()):outcome.start()]
        assert "__all_sync" in condition or "__any_sync" in condition
