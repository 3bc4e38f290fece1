"""The sets of partial sums that the solve kernel's blocks exchange at its grid
barriers (csrc/ggb_partials.h), checked without a GPU: the header's rule is
compiled and run by a model of two blocks, and every interleaving of their steps
has to give each block the sums of the barrier that it reads for."""
import itertools
import os
import subprocess

import pytest

from conftest import PKG

PROBE = r"""
#include <cstdio>
#include "ggb_partials.h"
int main() {
  for (int e = 0; e < 64; e++) printf("%d ", ggb::part_set(e));
  printf("%d %zu\n", ggb::kPartSets, ggb::part_doubles(148));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("partials")
    src, exe = d / "probe.cpp", d / "probe"
    src.write_text(PROBE)
    subprocess.run(["/usr/bin/g++", "-std=c++17", f"-I{os.path.join(PKG, 'csrc')}", "-o", str(exe), str(src)],
                   check=True)
    out = [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    return out[:64], out[64], out[65]


def wrong_read(kinds, part_set):
    """Two blocks through the barriers `kinds` ('n': no sums, 's': sums read
    after the barrier, 'l': sums read beside the next barrier).  A block's first
    warp writes its row, arrives, waits and reads; the second warp reads a late
    sum at any time between the two block barriers of the next grid barrier.
    True when some interleaving lets a block read another barrier's row."""
    last = len(kinds)

    def steps(e):  # the first warp's steps at barrier e
        return (["write"] if kinds[e] != "n" else []) + ["arrive", "wait"] + (["read"] if kinds[e] == "s" else [])

    # per block: barrier, steps of the first warp done, second warp's read done
    start = ((0, 0, False), (0, 0, False), (0, 0), ())
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        blocks, arrived, rows = list(state[:2]), state[2], dict(state[3])
        for b in (0, 1):
            e, pc, late_done = blocks[b]
            if e == last:
                continue
            late = e > 0 and kinds[e - 1] == "l"
            moves = []
            if pc < len(steps(e)):
                op = steps(e)[pc]
                if op == "wait" and min(arrived) <= e:
                    op = None
                if op == "read" and rows.get((part_set(e), 1 - b)) != e:
                    return True
                if op:
                    new_rows, new_arrived = rows, arrived
                    if op == "write":
                        new_rows = {**rows, (part_set(e), b): e}
                    if op == "arrive":
                        new_arrived = tuple(e + 1 if x == b else arrived[x] for x in (0, 1))
                    moves.append(((e, pc + 1, late_done), new_arrived, new_rows))
            if late and not late_done:
                if rows.get((part_set(e - 1), 1 - b)) != e - 1:
                    return True
                moves.append(((e, pc, True), arrived, rows))
            if pc == len(steps(e)) and (late_done or not late):
                moves.append(((e + 1, 0, False), arrived, rows))
            for block, new_arrived, new_rows in moves:
                pair = list(blocks)
                pair[b] = block
                nxt = (pair[0], pair[1], new_arrived, tuple(sorted(new_rows.items())))
                if nxt not in seen:
                    seen.add(nxt)
                    todo.append(nxt)
    return False


SEQUENCES = [k for n in range(1, 6) for k in itertools.product("nsl", repeat=n) if k[-1] != "l"]


def test_every_interleaving_reads_its_own_sums(rule):
    sets, _, _ = rule
    bad = ["".join(k) for k in SEQUENCES if wrong_read(k, lambda e: sets[e])]
    assert not bad, bad


def test_the_model_sees_a_set_reused_too_early():
    """Two alternating sets: a late |r|^2 read beside a barrier without sums and
    the sum at the barrier after it (the solve's exit) share a set."""
    assert wrong_read("lns", lambda e: e & 1)
    assert not wrong_read("sss", lambda e: e & 1)


def test_partials_hold_every_set(rule):
    sets, count, doubles = rule
    assert set(sets) == set(range(count)) and doubles == count * 2 * 148
