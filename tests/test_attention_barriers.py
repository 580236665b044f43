"""The order that the barriers of the tcgen05 prefill kernels keep between the MMA warp and the softmax warps, by a walk through every
interleaving of them (no GPU): P V of a key block is issued only when every softmax warp has written that block's P, and no wait is left
behind by its barrier's phases.  The number of barriers for P is read from the kernel's source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpt_fast_b200", "csrc", "attention_tc.cu")


def p_barriers(struct):
    body = re.search(r"struct %s \{(.*?)\n\};" % struct, open(SOURCE).read(), re.S).group(1)
    found = re.search(r"^ *unsigned long long (?:[^;/]*, )?p_ready(?:\[(\d+)\])?[,;]", body, re.M)
    return int(found.group(1) or 1)


def walk(blocks, warps, n_bars, reads_counted):
    """All reachable states of one work item.  MMA warp: S(0); for every block j: S(j + 1) (its buffer read by every warp, if
    `reads_counted`), wait for P(j), P V(j).  Softmax warp: for every block j: wait for S(j), [read it,] write P(j), arrive.  S counts as
    done at once, the earliest it can be.  A barrier is (phases completed, arrivals of the current phase) and a wait for phase n sees only
    their parity, as mbarrier.try_wait.parity does.  Returns what went wrong, as a set."""
    program = [("S", 0)]
    for j in range(blocks):
        program += ([("S", j + 1)] if j + 1 < blocks else []) + [("wait", j), ("PV", j)]
    # a warp's position: 2 j = waits for S(j), 2 j + 1 = has read S(j); arriving for block j ends at 2 (j + 1)
    start = (0, (0,) * warps, ((0, 0),) * n_bars)
    seen, todo, wrong = {start}, [start], set()

    def push(state):
        if state not in seen:
            seen.add(state)
            todo.append(state)

    while todo:
        pc, at, bars = todo.pop()
        issued = sum(1 for op, _ in program[:pc] if op == "S")
        moved = False
        if pc < len(program):
            op, j = program[pc]
            go = True
            if op == "S" and reads_counted and j >= 2:
                go = all(a > 2 * (j - 2) for a in at)
            if op == "wait":
                go = bars[j % n_bars][0] % 2 != (j // n_bars) % 2
            if op == "PV" and any(a < 2 * (j + 1) for a in at):
                wrong.add("P V before every warp's P")
            if go:
                moved = True
                push((pc + 1, at, bars))
        for w, a in enumerate(at):
            if w and a == at[w - 1] or a == 2 * blocks:             # (equal neighbours: the same state up to their names)
                continue
            j, reading = divmod(a, 2)
            if not reading and j >= issued:
                continue
            moved, new = True, bars
            if reading:
                done, n = bars[j % n_bars]
                n += 1
                new = bars[:j % n_bars] + (((done + 1, 0) if n == warps else (done, n)),) + bars[j % n_bars + 1:]
            push((pc, tuple(sorted(at[:w] + (a + 1,) + at[w + 1:])), new))
        if not moved and (pc < len(program) or any(a < 2 * blocks for a in at)):
            wrong.add("a wait that nothing ends")
    return wrong


@pytest.mark.parametrize("struct,warps,reads_counted", [("Bars", 4, True), ("LatBars", 4, False)])
def test_no_product_runs_ahead_of_its_weights(struct, warps, reads_counted):
    assert walk(6, warps, p_barriers(struct), reads_counted) == set()


def test_the_walk_sees_what_one_barrier_does():
    assert "P V before every warp's P" in walk(4, 4, 1, False)
    assert "P V before every warp's P" in walk(4, 4, 1, True)
