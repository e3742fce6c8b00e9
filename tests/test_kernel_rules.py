"""Rules of the kernels' source whose breach no run is sure to show: orderings between pipeline stages that hold by timing until
they do not.  Read from the text, on the CPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warp34_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return [x.split("//")[0] for x in f]


@pytest.mark.parametrize("name", ["tq4_stream_tc.cuh", "prefill_pair.cuh", "tq4_prefill_tc.cuh"])
def test_tensor_memory_accesses_are_fenced_from_the_wait_before_them(name):
    """An access to tensor memory behind a wait on an mbarrier needs tcgen05.fence::after_thread_sync in between: the wait alone does
    not order the access behind the MMAs whose completion it saw.  (Waits on other barriers in between are no matter; the
    rescaling and epilogue accesses that follow a fenced one without a new wait are covered by it.)"""
    waited = None
    for i, line in enumerate(_code(name), 1):
        if re.match(r"__device__|template|static", line):
            waited = None
        if re.search(r"\b(wait_all|mbar_wait)\(bar\(", line) and not re.search(r"Raw|KScale|QFull|QFree|KXtQ|Drain|RawFull|RawFree", line):
            waited = i
        if "tc_fence_after()" in line:
            waited = None
        if re.search(r"\btc_(ld|st)\w*\(", line) and "tc_wait" not in line and waited is not None:
            raise AssertionError(f"{name}:{i}: access to tensor memory, unfenced since the wait in line {waited}")


def test_what_the_kernel_in_front_writes_is_not_read_through_the_non_coherent_path():
    """Kernels launched behind each other overlap (tq4_common.cuh), so the plan's output (query fragments, prefix arrays) and the
    partials change during the lifetime of the kernel that reads them: no __ldg and no const __restrict__ on them."""
    for name in ("tq4_stream_exact.cuh", "tq4_stream_tc.cuh", "prefill_pair.cuh"):
        for i, line in enumerate(_code(name), 1):
            assert "__ldg(" not in line and ".nc." not in line, f"{name}:{i}: {line.strip()}"
    for line in _code("tq4_common.cuh"):
        if "last_not_above(" in line and "__device__" in line:
            assert "__restrict__" not in line, line.strip()


@pytest.mark.parametrize("name", ["tq4_stream_tc.cuh", "prefill_pair.cuh", "tq4_prefill_tc.cuh"])
def test_a_loop_that_votes_is_left_by_a_vote(name):
    """Every lane takes part in each __all_sync of a polling loop, so the clock and the abort flag, which lanes read at different
    times, may end the loop through a vote only."""
    code = "".join(_code(name))
    for m in re.finditer(r"\b(do|for \(;;\))\s*\{", code):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(code[end], 0)
            end += 1
        body = code[m.end():end - 1] + code[end:code.index(";", end) + 1] if m.group(1) == "do" else code[m.end():end - 1]
        if "__all_sync" not in body:
            continue
        for line in body.splitlines() if "\n" in body else [body]:
            if "clock64()" in line and "t0 =" not in line:
                assert re.search(r"__any_sync|__all_sync", line), f"{name}: {line.strip()}"
