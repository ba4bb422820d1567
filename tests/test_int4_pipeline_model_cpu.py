"""Host model of the weight ring of the INT4 GEMM (csrc/kernels/int4_gemm.cu), explored over every interleaving of a small
instance without a GPU.

One thread loads the steps' weights into a ring (`raw_full` / `raw_empty`); two groups of converting warps take the steps in turn,
each from its ring slot into one of the operand slots (`b_full` / `b_empty`), which the MMA thread uses up in order.  A wait is
told by the parity of the phase it waits for, so it also returns while the phase before the last one is still open: a group must
not come to a slot before the slot's earlier step, which with a ring of odd depth is the other group's, has arrived.  The place in
the ring and its parity are stepped as the kernel steps them.
"""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "csrc" / "kernels" / "int4_gemm.cu").read_text()


def constant(name):
    text = re.search(rf"\b{name} = ([^,;]+)[,;]", SOURCE).group(1)
    return eval(re.sub(r"[A-Z_]{2,}", lambda m: str(constant(m.group(0))), text))


GROUPS, B_STAGES = constant("GROUPS"), constant("B_STAGES")


def faults(depth, steps=14):
    """What goes wrong with a ring of `depth` steps: places outside the ring, steps converted before they have arrived."""
    found = set()
    # places and parities as the converting warps step them
    place = {}
    for g in range(GROUPS):
        r, par = g, 0
        if r >= depth:
            r, par = r - depth, par ^ 1
        for i in range(g, steps, GROUPS):
            if r >= depth:
                found.add("outside the ring")
            place[i] = (r, par)
            r += GROUPS
            if r >= depth:
                r, par = r - depth, par ^ 1
    if found:
        return found
    # state: loads issued, loads landed (bits), per group (next step, polled the weights), steps converted (bits), steps multiplied
    start = (0, 0, tuple((g, False) for g in range(GROUPS)), 0, 0)
    seen, stack = {start}, [start]
    while stack:
        issued, landed, groups, converted, multiplied = stack.pop()
        moves = []
        if issued < steps and (issued < depth or converted >> (issued - depth) & 1):
            moves.append((issued + 1, landed, groups, converted, multiplied))
        for i in range(issued):                                 # copies land in any order
            if not landed >> i & 1:
                moves.append((issued, landed | 1 << i, groups, converted, multiplied))
        if converted >> multiplied & 1:
            moves.append((issued, landed, groups, converted, multiplied + 1))
        for g, (i, polled) in enumerate(groups):
            if i >= steps:
                continue
            r, par = place[i]
            if not polled:
                phases = sum(landed >> k & 1 for k in range(r, issued, depth))
                if (phases & 1) != par:                         # the open phase has the other parity
                    moves.append((issued, landed, groups[:g] + ((i, True),) + groups[g + 1:], converted, multiplied))
            elif i < B_STAGES or multiplied > i - B_STAGES:
                if not landed >> i & 1:
                    found.add("converted before it arrived")
                    continue
                moves.append((issued, landed, groups[:g] + ((i + GROUPS, False),) + groups[g + 1:], converted | 1 << i, multiplied))
        for m in moves:
            if m not in seen:
                seen.add(m)
                stack.append(m)
        if not moves and multiplied < steps:
            found.add("stuck")
    return found


@pytest.mark.parametrize("depth", range(constant("MIN_RAW_STAGES"), constant("MIN_RAW_STAGES") + 4))
def test_weight_ring_of_the_least_depth_and_deeper(depth):
    assert not faults(depth)


@pytest.mark.parametrize("depth,fault", [(1, "outside the ring"), (3, "converted before it arrived")])
def test_weight_ring_that_is_too_short(depth, fault):
    assert depth < constant("MIN_RAW_STAGES") and fault in faults(depth)
