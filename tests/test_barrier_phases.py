"""Parity waits of the two-CTA chunk kernel on the completion of its output products, checked on the CPU from the kernel's own
expressions.

An mbarrier wait names a phase by its parity alone: it returns when the barrier's last completed phase has that parity, so it is
sound only while at most that one phase can have completed.  A consumer warp may be held up for any time between two
instructions (a slow instruction fetch, a context switch) while the tensor cores go on; what bounds them is that the output
product of block i needs this warp's weights of block i."""
import os

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
