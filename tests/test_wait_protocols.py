"""The orders in which the roles of the tcgen05 attention kernels may run, tried one by one on the CPU: a
warp held up at any point must not read another tile's maxima, and whichever bounded wait runs out, every
role must come to its end.  What each role does, in order, is restated here; the number of slots and the
exits that let a partner go come from the kernels' sources."""

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


def stuck(let_go, tiles=3):
    """Whether some order and some choice of waits that run out leaves a warp of
    `masked_attention_stream_kernel` at an exchange without its partner.

    Two warps that share lanes and the issuing warp.  A bounded wait passes when its condition holds and may
    run out at any time before or after (a role can be held up for longer than the limit), and so does every later
    wait.  The exchange of maxima and the barrier behind the loops have no limit.  `let_go`: the waits,
    "scores" and "product", whose exit arrives at the exchange."""
    issued = [("s", 0)] + [x for j in range(tiles) for x in ([("s", j + 1)] if j + 1 < tiles else []) + [("p", j)]]
    # state: per warp (tile, step, left), exchanges arrived at by (warp or exit), issuer's position, issuer left
    start = (((0, 0, False),) * 2, (0, 0), 0, False)
    seen, todo = {start}, [start]
    while todo:
        warps, arrived, pos, gone = todo.pop()
        nexts = []

        def freed(j):  # s_free: both warps have tile j's scores in registers
            return all(w[0] > j or (w[0] == j and w[1] >= 1) for w in warps)

        def handed(j):  # p_full: both have stored P of tile j
            return all(w[0] > j for w in warps)

        def complete(kind, j):
            return issued.index((kind, j)) < pos

        if not gone and pos < len(issued):
            kind, j = issued[pos]
            if (kind == "s" and (j == 0 or freed(j - 1))) or (kind == "p" and handed(j)):
                nexts.append((warps, arrived, pos + 1, False))
            nexts.append((warps, arrived, pos, True))
        for me in range(2):
            j, step, left = warps[me]

            def to(tile, step, left=False, arrive=0):
                w = tuple((tile, step, left) if i == me else x for i, x in enumerate(warps))
                a = tuple(x + arrive if i == me else x for i, x in enumerate(arrived))
                nexts.append((w, a, pos, gone))

            if left or j == tiles:
                continue
            if step == 0:  # the tile's scores
                if complete("s", j):
                    to(j, 1)
                to(j, 0, True, int("scores" in let_go))
            elif step == 1:  # arrives at the exchange ...
                to(j, 2, False, 1)
            elif step == 2:  # ... and waits for the other: no limit
                if arrived[1 - me] > j:
                    to(j, 3)
            elif step == 3:  # the product before; then P is handed over
                if j == 0 or complete("p", j - 1):
                    to(j + 1, 0)
                if j > 0:
                    to(j, 3, True, int("product" in let_go))
        if not nexts and not all(w[2] or w[0] == tiles for w in warps):
            return True
        for n in nexts:
            if n not in seen:
                seen.add(n)
                todo.append(n)
    return False


def test_a_wait_that_runs_out_leaves_nobody_at_an_exchange():
    source = (CSRC / "sah_attention_stream.cuh").read_text()
    loop = source[source.index("for (int t = gg; t < n_tiles; t += 2, ++j)"):source.index("have_o = ok && j > 0")]
    exits = re.findall(r"(let_go\(\);\s*)?break;", loop)
    assert len(exits) == 2
    assert not stuck([name for name, lets_go in zip(("scores", "product"), exits) if lets_go])
    assert stuck(["scores"]) and stuck(["product"]) and stuck([])
