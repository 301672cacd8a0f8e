"""The counters of the two-level replica reductions (replica_reduce, post_reduce)
over two consecutive steps, every interleaving of the blocks.

Each group's last block arrives at the replica's counter; the replica's last
block finishes the step, after which the next step's blocks may start (k_flow
queues them at once, while blocks of the step before may still be between two
of their counter operations).  The operations' order is taken from the source;
no interleaving may lose a count, which would leave the replica waiting for a
block that never comes."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "rumd_b200", "csrc", "kernels.cuh")
OPS = [("g_add", r"atom_add_acq_rel\(&(?:a\.)?gctr\["), ("g_reset", r"\bgctr\[[^\]]*\] = 0u"),
       ("r_add", r"atom_add_acq_rel\(&(?:a\.)?rctr\["), ("r_reset", r"\brctr\[[^\]]*\] = 0u")]


def source_order(name):
    """The counter operations of the function's body, in the order of its text
    (the first of each kind: the path of a replica with several groups)."""
    text = open(SRC).read()
    body = text[text.index(" bool " + name + "("):]
    body = body[: body.index("\n}\n")]
    found = sorted((m.start(), op) for op, pat in OPS for m in re.finditer(pat, body))
    return list(dict.fromkeys(op for _, op in found))


def stuck_states(order, groups):
    """Walks every interleaving of one replica's blocks (groups: the number of
    tiles of each of its groups) over two steps.  Returns the number of states
    in which nothing can move although the second step is unfinished."""
    blocks = [(step, g) for step in (0, 1) for g, tiles in enumerate(groups) for _ in range(tiles)]
    # each block's operations still to do, the counters, the finished steps
    start = ((tuple(order),) * len(blocks), (0,) * len(groups), 0, 0)
    seen, todo, stuck = {start}, [start], 0
    while todo:
        left, gctr, rctr, finished = todo.pop()
        moved = False
        for b, (step, g) in enumerate(blocks):
            if not left[b] or step > finished:
                continue
            moved = True
            op, rest, gc, rc, fin = left[b][0], left[b][1:], list(gctr), rctr, finished
            if op == "g_add":
                rest = rest if gc[g] == groups[g] - 1 else ()  # only its group's last block goes on
                gc[g] += 1
            elif op == "g_reset":
                gc[g] = 0
            elif op == "r_add":
                if rc != len(groups) - 1:  # only the replica's last block finishes the step
                    rest = tuple(k for k in rest if k != "r_reset")
                rc += 1
            else:
                rc, fin = 0, step + 1
            s = (left[:b] + (rest,) + left[b + 1:], tuple(gc), rc, fin)
            if s not in seen:
                seen.add(s)
                todo.append(s)
        stuck += not moved and finished < 2
    return stuck


@pytest.mark.parametrize("groups", [(1, 1), (2, 1), (2, 2)])
@pytest.mark.parametrize("name", ["replica_reduce", "post_reduce"])
def test_no_interleaving_loses_a_count(name, groups):
    order = source_order(name)
    assert set(order) == {op for op, _ in OPS} and order[-1] == "r_reset"
    assert stuck_states(order, groups) == 0


def test_the_walk_finds_a_late_reset():
    assert stuck_states(["g_add", "r_add", "g_reset", "r_reset"], (1, 1)) > 0
