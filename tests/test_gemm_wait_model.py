"""What the tensor-core product (csrc/gemm.cu: k_qgemm) and the streaming kernels (csrc/fused.cu) do when a bounded
wait runs out, checked as a state machine over every interleaving.

One CTA: two of the epilogue's warps stand for the four.  A warp waits for its accumulators with a limit of its own (the
wait may run out at any moment, also just before the accumulators arrive), goes on to a named barrier that all
epilogue warps meet at, and ends at the CTA's last barrier.  The accumulators may arrive at any moment or never.

A cluster: each CTA requests a box of weights, adds up, pushes a share of its sums into every other CTA's shared
memory, waits for the shares pushed to it and leaves.  Boxes and pushes land at any later moment; a CTA that has
left must not be their target.

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


def cluster_protocol():
    src = open(os.path.join(CSRC, "gemm.cu")).read()
    body = kernel_source()
    tail = body[body.rindex("__syncthreads"):]
    late = src[src.index("void leave_late("):src.index("k_qgemm(const __grid_constant__")] if "void leave_late(" in src else ""
    called = bool(re.search(r"if \(s_leave.quit\) \{.*leave_late\(", tail, re.S)) and "if (!ok) s_leave.quit = 1;" in epilogue_source()
    return {"meet": called and bool(re.search(r"cluster_arrive\(\);\s*cluster_wait\(\);\s*if \(threadIdx.x == 128\) mbar_wait\(part_full", late)),
            "drain": called and "landed(raw_full" in late and "landed(full" in late and "tc_commit(mma_done);\n    mbar_wait_warp(mma_done" in late}


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


def explore_cluster(C, meet, drain):
    """Every reachable state of C CTAs; raises where something lands in a CTA that has left, or nothing can move."""
    # a CTA: (step, ok, box, got) with box in flight or landed, got = the peers whose share has landed
    start = (tuple(("sum", True, "flying", frozenset()) for _ in range(C)), frozenset())   # and the pushes in flight
    seen, todo = {start}, deque([start])
    ends = set()
    while todo:
        ctas, flying = todo.popleft()
        nxt = []

        def to(i, step, ok, box, got, fl=flying):
            nxt.append((ctas[:i] + ((step, ok, box, got),) + ctas[i + 1:], fl))
        for i, (step, ok, box, got) in enumerate(ctas):
            peers = frozenset(range(C)) - {i}
            if box == "flying":
                assert step != "gone", ("a box lands in a CTA that has left", ctas)
                to(i, step, ok, "landed", got)
            if step == "sum":
                if box == "landed":
                    to(i, "push", True, box, got)
                to(i, "end", False, box, got)
            elif step == "push":
                to(i, "share", ok, box, got, flying | {(i, j) for j in peers})
            elif step == "share":
                if got == peers:
                    to(i, "end", ok, box, got)
                to(i, "end", False, box, got)
            elif step == "end":
                if ok or not drain or box == "landed":
                    to(i, "met" if meet and not ok else "gone", ok, box, got)
            elif step == "met":      # the others have pushed, given up or left; what they pushed has landed
                if all(c[0] in ("met", "gone") for c in ctas) and not any(j == i for _, j in flying):
                    to(i, "gone", ok, box, got)
        for a, b in flying:
            step, ok, box, got = ctas[b]
            assert step != "gone", ("a share lands in a CTA that has left", ctas)
            to(b, step, ok, box, got | {a}, flying - {(a, b)})
        if all(c[0] == "gone" for c in ctas):
            ends.add(tuple(c[1] for c in ctas))
        else:
            assert nxt, ("hangs", ctas)
        for n in nxt:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return ends


@pytest.mark.parametrize("C", [1, 2, 3])
def test_a_cta_stays_while_anything_can_land_in_it(C):
    ends = explore_cluster(C, **cluster_protocol())
    assert (True,) * C in ends and (False,) * C in ends


@pytest.mark.parametrize("meet,drain,what", [(False, True, "share lands"), (True, False, "box lands")])
def test_the_model_finds_what_lands_too_late(meet, drain, what):
    with pytest.raises(AssertionError, match=what):
        explore_cluster(2, meet, drain)


def test_a_streaming_warp_stays_while_its_copies_are_in_flight():
    """The rings of the streaming kernels: a warp waits as a whole, and one that gives up waits for what it has
    requested.  As above with one CTA: the warp is the CTA, a tile is the box."""
    src = open(os.path.join(CSRC, "fused.cu")).read()
    wait = src[src.index("// lane 0: two bulk copies"):src.index("// carve the rings of all warps")]
    assert len(re.findall(r"__all_sync\(0xffffffffu, mbar_try_wait\(", wait)) == len(re.findall(r"\bmbar_try_wait\(", wait)) > 0
    assert len(re.findall(r"\bmbar_try_wait\(", src)) == 1 + len(re.findall(r"\bmbar_try_wait\(", wait))   # no wait elsewhere
    explore_cluster(1, meet=True, drain=bool(re.search(r"for \(int i = 0; i < depth && ring_poll\(", wait)))


def test_only_single_lanes_wait_for_themselves():
    """Outside the two producers (one lane each) every wait of the roles is agreed on by the threads that go on
    together."""
    body = kernel_source()
    roles = re.split(r"\n    // ---- ", body)
    plain = {r.split("\n")[0][:24]: len(re.findall(r"\bmbar_wait\(", r)) for r in roles[1:]}
    assert sum(plain.values()) == sum(n for r, n in plain.items() if r.startswith(("raw weight", "token tiles"))), plain
