"""The loops that issue tensor-core products, read as text (nothing of them can be seen to go wrong without a GPU that hangs): a whole warp runs them and one
elected lane issues."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cake_b200", "csrc")
KERNELS = {"gemm_tc.cuh": 2, "gemm_skinny.cuh": 1, "attn_prefill_tc.cuh": 3, "attn_window_tc.cuh": 3}   # waits of the issuing warp


def lines(name):
    with open(os.path.join(CSRC, name)) as f:
        return [re.sub(r"//.*", "", x) for x in f]


def issuing_branch(name):
    """The lines from `one = elect_one()` to the end of the warp's branch."""
    src = lines(name)
    first = next(i for i, x in enumerate(src) if re.search(r"\bone = elect_one\(\)", x))
    last = next(i for i in range(first, len(src)) if re.match(r"  }( else|$)", src[i]))
    return src[first:last]


@pytest.mark.parametrize("name", KERNELS)
def test_every_lane_has_seen_a_phase_before_one_issues(name):
    """What a lane issues lets barriers run on to their next phase; a lane that still waits for the one before would find it gone by (parities repeat) and
    keep the warp until its wait runs out.  So the warp comes together between its waits and the issue, whatever the compiler makes of the loops."""
    waits, open_wait = 0, False
    for x in issuing_branch(name):
        if "mbar_wait_lim" in x and "q_full" not in x:   # (of q_full there is one phase only)
            waits, open_wait = waits + 1, True
        if "__syncwarp()" in x:
            open_wait = False
        if re.search(r"\bif \(one\)", x):
            assert not open_wait, f"{name}: a lane issues behind a wait that others may still be in"
    assert waits == KERNELS[name]


@pytest.mark.parametrize("name", KERNELS)
def test_the_lane_that_issues_is_the_one_that_commits(name):
    """A commit counts the products of its own thread: one by another lane completes at once, and a CTA that gave up would hand its tensor memory back
    under products in flight."""
    guard, commits = [], 0   # the lines that opened the enclosing blocks
    for x in lines(name):
        if re.search(r"\btc_commit(_pair)?\(", x) and "__device__" not in x:
            commits += 1
            assert any("if (one)" in g or "elect_one()" in g for g in guard + [x]), f"{name}: {x.strip()}"
        for ch in x:
            if ch == "{":
                guard.append(x)
            elif ch == "}":
                guard.pop()
    assert commits >= 3
