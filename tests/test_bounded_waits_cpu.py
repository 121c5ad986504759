"""Bounded waits of the tensor-core kernels, by reading their source: a wait that runs out, or
sees another role's abort, ends on each lane by itself.  A role that a whole warp runs must
therefore leave it by a vote, or lanes that give up go to the CTA's last barrier while the
others stay at a warp-wide operation, and the CTA never ends.  So every call of a wait is either
inside a vote or made by one elected lane."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vapoursynth-zipcu_b200", "csrc")
WAITS = {"zb3d_dct_tc.cu": "wait_phase", "zb3d_pilot_tc.cu": "wait_bar", "zb3d_match_tc.cu": "mbar_wait"}


def waits_of(text, name):
    """(line, statement so far, headers of the enclosing blocks) of every call."""
    text = re.sub(r"//[^\n]*", "", text)
    heads, start, calls = [], 0, []
    depth = 0  # parentheses: the ; of a for header ends no statement
    for m in re.finditer(r"[{}();]|\b" + name + r"\(", text):
        t = m.group()
        if t == "(":
            depth += 1
        elif t == ")":
            depth -= 1
        elif t == "{":
            heads.append(text[start:m.start()])
            start = m.end()
        elif t == "}":
            heads.pop()
            start = m.end()
        elif t == ";" and depth == 0:
            start = m.end()
        elif t.startswith(name):
            calls.append((text.count("\n", 0, m.start()) + 1, text[start:m.start()], list(heads)))
            depth += 1
    return calls


def one_lane(head):
    return re.search(r"\b(lane|tid|threadIdx\.x) == 0\b", head) is not None


@pytest.mark.parametrize("name", sorted(WAITS))
def test_a_warp_leaves_a_wait_together(name):
    calls = [c for c in waits_of(open(os.path.join(CSRC, name)).read(), WAITS[name])
             if "__device__" not in c[1]]  # the definition
    assert len(calls) >= 2
    alone = [line for line, stmt, heads in calls
             if "__all_sync(" not in stmt and not one_lane(stmt) and not any(one_lane(h) for h in heads)]
    assert not alone, f"{name}: waits on lines {alone} end lane by lane in a role of whole warps"
