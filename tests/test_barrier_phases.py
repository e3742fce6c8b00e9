"""Parity waits of the two-CTA chunk kernel and of the 9- to 24-row stream kernel on the completion of their output products, checked on
the CPU from the kernels' own expressions.

An mbarrier wait names a phase by its parity alone: it returns when the barrier's last completed phase has that parity, so it is
sound only while at most that one phase can have completed.  A consumer warp may be held up for any time between two
instructions (a slow instruction fetch, a context switch) while the tensor cores go on; what bounds them is that the output
product of block i needs this warp's weights of block i."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warp34_b200", "csrc", "prefill_pair.cuh")


def _expr(text):
    return text.replace("(uint32_t)", "").strip()


def _operand(text, name):
    """The parenthesised argument list that follows `name(` in text."""
    at = text.index(name + "(") + len(name) + 1
    depth, end = 1, at
    while depth:
        depth += {"(": 1, ")": -1}.get(text[end], 0)
        end += 1
    return text[at:end - 1]


def _split(args):
    """Top-level commas of an argument list."""
    out, depth, last = [], 0, 0
    for i, ch in enumerate(args):
        depth += {"(": 1, ")": -1}.get(ch, 0)
        if ch == "," and depth == 0:
            out.append(args[last:i])
            last = i + 1
    return out + [args[last:]]


def _pv_uses():
    with open(SRC) as f:
        lines = [x.split("//")[0] for x in f if "kPpPv" in x and "bar(" in x]
    commits = [_expr(_operand(_operand(x, "tc2_commit_both"), "bar")) for x in lines if "tc2_commit_both" in x]
    waits = [[_expr(a) for a in _split(_operand(x, "wait_all"))] for x in lines if "wait_all" in x]
    return commits, [(_operand(a[0], "bar"), a[1]) for a in waits]


# where the four waits stand: the block whose product is waited for, and the last block whose weights this warp has delivered
WAITS = [("start of block j", lambda j, n: (j - 2, j - 1)), ("rescale in block j", lambda j, n: (j - 1, j - 1)),
         ("end, last but one", lambda j, n: (n - 2, n - 1)), ("end, last", lambda j, n: (n - 1, n - 1))]


@pytest.mark.parametrize("which", range(4))
def test_a_delayed_consumer_warp_still_sees_the_phase_it_waits_for(which):
    commits, waits = _pv_uses()
    assert len(commits) == 1 and len(waits) == 4, (commits, waits)
    slot_of = lambda i: eval(commits[0], {"kPpPv": 0, "i": i})  # noqa: E731
    bar_expr, parity_expr = waits[which]
    name, place = WAITS[which]
    for n in range(1, 12):
        for j in range(n):
            block, delivered = place(j, n)
            if block < 0:
                continue
            env = {"kPpPv": 0, "j": j, "nblocks": n}
            slot, parity = eval(bar_expr, env), eval(parity_expr, env)
            assert slot == slot_of(block), (name, j, n)
            for done in range(block, delivered + 1):           # products completed when the warp gets to look: at least, at most
                phases = sum(slot_of(i) == slot for i in range(done + 1))
                assert (phases - 1) & 1 == parity, f"{name}: j {j} of {n}, products up to {done} completed"


# The stream kernel has a barrier for each half of a block's keys; the products of block c are number 2 c and 2 c + 1 and complete in
# order.  Per wait, in the order of the source: the last product that is known to have completed, and the last that can have.
XT_SRC = os.path.join(os.path.dirname(SRC), "tq4_stream_tc.cuh")
XT_WAITS = [("start of block c", lambda c, half: 2 * (c - 2) + half, lambda c, half: 2 * c + half - 1),   # its own weights are still due
            ("rescale in block c", lambda c, half: 2 * (c - 1) + half, lambda c, half: 2 * c - 1),        # all four warps' weights are due
            ("end, first half", lambda c, half: 2 * (c - 2) + half, lambda c, half: 2 * c - 1),
            ("end, second half", lambda c, half: 2 * (c - 1), lambda c, half: 2 * c - 1)]


@pytest.mark.parametrize("which", range(4))
def test_a_delayed_softmax_warp_still_sees_the_phase_it_waits_for(which):
    with open(XT_SRC) as f:
        code = "".join(x.split("//")[0] for x in f)
    waits = re.findall(r"wait_all\(bar\((kXtPvDone[^,]*)\), ([^,;]*?1u)\)", code)
    commits = re.findall(r"tc_commit\(bar\((kXtPvDone[^;]*)\)\);", code)
    assert len(waits) == 4 and commits == ["kXtPvDone + kk"], (waits, commits)
    (bar_expr, parity_expr), (name, known, most) = waits[which], XT_WAITS[which]
    for c in range(1, 12):
        for khalf in range(2):
            env = {"kXtPvDone": 0, "khalf": khalf, "c": c}
            half, parity = eval(bar_expr, env), eval(parity_expr.replace("1u", "1"), env)
            for done in range(max(known(c, khalf), -1), most(c, khalf) + 1):
                phases = sum(i % 2 == half for i in range(done + 1))
                passes = (phases - 1) & 1 == parity
                assert passes == (done >= 2 * (c - 1) + half), f"{name}: block {c}, half {khalf}, products up to {done} completed"
