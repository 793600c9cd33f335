"""What the tensor-core product (csrc/gemm.cu: k_qgemm) does when a bounded wait runs out, checked as a state
machine over every interleaving.

Two of the epilogue's warps stand for the four.  A warp waits for its accumulators with a limit of its own (the
wait may run out at any moment, also just before the accumulators arrive), goes on to a named barrier that all
epilogue warps meet at, and ends at the CTA's last barrier.  The accumulators may arrive at any moment or never.
Which of the steps the kernel has is read from its source, so the model follows the code."""
import os
import re
from collections import deque

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ornith-rs_b200", "csrc")
WARPS = 2


def kernel_source():
    src = open(os.path.join(CSRC, "gemm.cu")).read()
    return src[src.index("k_qgemm(const __grid_constant__"):src.index("grouped form: sorting and row movement")]


def epilogue_source():
    src = kernel_source()
    return src[src.index("// ---- epilogue"):]


def protocol():
    return {"vote": "mbar_wait_epilogue(acc_full" in epilogue_source()}


def explore(vote):
    """Every reachable state; raises on a state that nothing can leave."""
    # per warp (step, ok): wait -> [vote ->] emit barrier -> last barrier -> gone
    start = (False, tuple(("wait", True) for _ in range(WARPS)))
    seen, todo = {start}, deque([start])
    ends = set()
    while todo:
        acc, warps = todo.popleft()
        nxt = []
        if not acc:
            nxt.append((True, warps))
        for i, (step, ok) in enumerate(warps):
            def to(*new):
                return (acc, warps[:i] + (tuple(new),) + warps[i + 1:])
            if step == "wait":
                for got in ([True] if acc else []) + [False]:
                    nxt.append(to("vote" if vote else "emit" if got else "last", got))
        at = [s for s, _ in warps]
        if all(s == "vote" for s in at):
            good = all(o for _, o in warps)
            nxt.append((acc, tuple(("emit" if good else "last", good) for _ in warps)))
        if all(s == "emit" for s in at):
            nxt.append((acc, tuple(("last", o) for _, o in warps)))
        if all(s == "last" for s in at):
            nxt.append((acc, tuple(("gone", o) for _, o in warps)))
        if all(s == "gone" for s in at):
            ends.add(tuple(o for _, o in warps))
            continue
        progress = [n for n in nxt if n[1] != warps]
        assert progress or any(n[0] for n in nxt), ("hangs", acc, warps)
        if acc:
            assert progress, ("hangs", acc, warps)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return ends


def test_a_wait_that_runs_out_leaves_nobody_behind():
    ends = explore(**protocol())
    assert (True,) * WARPS in ends and (False,) * WARPS in ends
    assert len(ends) == 2          # the warps always agree


def test_the_model_finds_the_warp_that_is_left_behind():
    """Without the common outcome one warp leaves and the others meet at a barrier that never fills."""
    with pytest.raises(AssertionError, match="hangs"):
        explore(vote=False)


def test_only_single_lanes_wait_for_themselves():
    """Outside the two producers (one lane each) every wait of the kernel is agreed on by the threads that go on
    together."""
    body = kernel_source()
    roles = re.split(r"\n    // ---- ", body)
    plain = {r.split("\n")[0][:24]: len(re.findall(r"\bmbar_wait\(", r)) for r in roles[1:]}
    assert sum(plain.values()) == sum(n for r, n in plain.items() if r.startswith(("raw weight", "token tiles"))), plain
