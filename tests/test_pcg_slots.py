"""The partial sums of the two PCG kernels: between two reductions of a solve lies one grid
barrier, after which every block reads the first's slots and may go on to write the second's.
A block that is slow to read must find them untouched, whatever the others do."""
from __future__ import annotations

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "boiling-sim_b200", "csrc")
KERNELS = {"pcg.cu": r"block_partials<(\d)>\(v, a\.partials( \+ ([\w ]+?) \* a\.stride| \+ a\.stride|)",
           "pcgr.cu": r"pr_barrier<(\d)>\(s, a, \w, a\.partials( \+ ([\w ]+?) \* gridDim\.x| \+ gridDim\.x|)"}


def _reductions(name):
    """Slots that each reduction of the kernel publishes, in program order."""
    header = open(os.path.join(CSRC, "pcgr.cuh")).read()
    first = {k: int(v) for k, v in re.findall(r"constexpr int (PCG_SUM_\w+) = (\d+);", header)}
    out = []
    for count, offset, slot in re.findall(KERNELS[name], open(os.path.join(CSRC, name)).read()):
        lo = first[slot] if slot else (1 if offset else 0)
        out.append(set(range(lo, lo + int(count))))
    assert len(out) == 3  # the initial sums, then A and B of an iteration
    return out


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_a_reduction_keeps_off_the_slots_of_the_one_before(name):
    init, a, b = _reductions(name)
    for one, then in ((init, a), (a, b), (b, a)):
        assert not one & then, f"{name}: {sorted(then)} are written while {sorted(one)} are read"


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_every_block_reads_the_same_sums_in_any_order_of_events(name):
    """Two blocks, the second run as far ahead of the first as the barriers let it: what the
    first reads for a reduction is what was published for it."""
    init, a, b = _reductions(name)
    steps = [init] + [a, b] * 3
    for slow_reads_last in (True, False):
        memory = {}  # (block, slot) -> reduction
        for n, slots in enumerate(steps):
            memory.update({(blk, s): n for blk in (0, 1) for s in slots})  # then the barrier
            ahead = steps[n + 1] if slow_reads_last and n + 1 < len(steps) else ()
            memory.update({(1, s): n + 1 for s in ahead})  # block 1 has read and goes on
            for s in slots:
                assert (memory[0, s], memory[1, s]) == (n, n), (name, n, s)
