"""The orders in which the roles of the tcgen05 attention kernels may run, tried one by one on the CPU: a
warp held up at any point must not read another tile's maxima.  What each role does, in order, is
restated here; the number of slots comes from the kernel's source."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sparse-attention-hub_b200" / "csrc"


def explore(programs):
    """Every reachable tuple of program counters.  A program is a list of steps; a step is called with
    the counters and says whether it can be taken now."""
    start = (0,) * len(programs)
    seen, todo = {start}, [start]
    while todo:
        at = todo.pop()
        for who, program in enumerate(programs):
            if at[who] < len(program) and program[at[who]](at):
                after = at[:who] + (at[who] + 1,) + at[who + 1:]
                if after not in seen:
                    seen.add(after)
                    todo.append(after)
    return seen


def maxima_read(slots, warps=3, tiles=4):
    """(tile that a warp works on, tile whose maximum it finds in another's slot), over all orders.

    A group of warps and the issuing warp of `masked_attention_umma_kernel`.  Per tile a warp waits for the
    scores, frees them, leaves its maximum, arrives, waits for all maxima, reads them, waits for the product
    before, and hands over P; the issuer runs the next tile's scores in front of the present product."""
    issued = [("s", 0)] + [x for j in range(tiles) for x in ([("s", j + 1)] if j + 1 < tiles else []) + [("p", j)]]
    scores = {j: issued.index(("s", j)) for j in range(tiles)}
    product = {j: issued.index(("p", j)) for j in range(tiles)}
    STEPS = 8  # of a warp per tile: scores, free, leave, arrive, all arrived, read, product before, hand over
    found = set()

    def past(at, who, j, step):
        return at[who] > j * STEPS + step

    def warp(me):
        program = []
        for j in range(tiles):
            program += [lambda at, j=j: at[-1] > scores[j]] + [lambda at: True] * 3
            program += [lambda at, j=j: all(past(at, w, j, 3) for w in range(warps))]

            def read(at, j=j):
                for w in range(warps):
                    left = [t for t in range(tiles) if past(at, w, t, 2) and t % slots == j % slots]
                    found.add((j, left[-1]))
                return True

            program += [read, lambda at, j=j: j == 0 or at[-1] > product[j - 1], lambda at: True]
        return program

    def issuer():
        free, full = 1, 7
        return [(lambda at, j=j: j == 0 or all(past(at, w, j - 1, free) for w in range(warps))) if kind == "s" else
                (lambda at, j=j: all(past(at, w, j, full) for w in range(warps))) for kind, j in issued]

    reached = explore([warp(w) for w in range(warps)] + [issuer()])
    assert (tiles * STEPS,) * warps + (len(issued),) in reached
    return found


def test_every_warp_reads_the_maxima_of_its_own_tile():
    slots = int(re.search(r"WMAX_SLOTS = (\d+)", (CSRC / "sah_attention_umma.cuh").read_text()).group(1))
    assert all(mine == theirs for mine, theirs in maxima_read(slots))
    assert any(mine != theirs for mine, theirs in maxima_read(1))  # one slot does not do
