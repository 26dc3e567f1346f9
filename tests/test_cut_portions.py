"""The cut of long prompts' work items into shares (host arithmetic of the tcgen05 prompt attention)."""
import heapq
import os
import random
import subprocess
import sys

import numpy as np
import pytest

from llm_steadyinfer_b200.csrc import ops

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def plain(tiles, copies, blocks, least, most):
    """The rule written down: (limit, schedule) taken, or None."""
    def schedule(limit):
        cost = sorted((-(-t // n) + 2 + (3 if n > 1 else 0) for t in tiles for n in [-(-t // limit)] for _ in range(n)), reverse=True)
        heap = [0] * blocks
        for c in cost:
            for _ in range(copies):
                heapq.heapreplace(heap, heap[0] + c)
        return max(heap)

    longest = max(tiles)
    if longest < 2 * least or len(tiles) * copies > 8 * blocks:
        return None
    whole = schedule(longest)
    if whole * 0.95 <= sum(tiles) * copies / blocks:
        return None
    limits = {max(least, -(-longest // k)) for k in (2, 3, 4, 6, 9, 13, 18) if k <= 6 or len(tiles) * copies * k <= 4 * blocks}
    fits = [(schedule(l), l) for l in limits if l < longest and copies * sum(-(-t // l) for t in tiles if t > l) <= most]
    return min(fits)[1] if fits and min(fits)[0] <= 0.95 * whole else None


def test_a_cut_follows_the_rule_and_covers_every_item_once():
    rng = random.Random(5)
    cuts = 0
    for _ in range(150):
        copies, blocks, per = rng.choice([1, 2, 4, 8]), rng.choice([9, 24, 148]), rng.choice([1, 2, 3])
        start, n = rng.randint(1, 300), rng.randint(1, 60)
        tiles = [start + per * i for i in range(n)] + [rng.randint(1, 40) for _ in range(rng.choice([0, 0, 3]))]
        limit = plain(tiles, copies, blocks, 16, 3 * blocks)
        got = ops.cut_portions(tiles, copies, blocks)
        assert (got is None) == (limit is None), (tiles, copies, blocks)
        if got is None:
            continue
        cuts += 1
        entries, cut, slots = got
        assert entries.dtype == cut.dtype == np.int32 and slots <= ops.cut_slots(copies, blocks)
        want = {i: -(-t // limit) for i, t in enumerate(tiles)}
        assert sorted(map(tuple, entries[:, :3].tolist())) == sorted((i, s, k) for i, k in want.items() for s in range(k))
        lengths = [-(-tiles[i] // k) for i, _, k, _ in entries.tolist()]
        assert lengths == sorted(lengths, reverse=True), "longest first"
        first = {i: f for i, _, f, _ in cut[:, [0, 1, 2, 3]].tolist()}
        assert {i: k for i, k, _, _ in cut.tolist()} == {i: k for i, k in want.items() if k > 1}
        taken = [f + s for i, f in first.items() for s in range(want[i])]
        assert sorted(taken) == list(range(slots)), "every share a slot of its own"
        assert all(f == first.get(i, 0) for i, _, _, f in entries.tolist())
    assert cuts > 20


@pytest.mark.parametrize("tiles,copies,blocks", [([31], 1, 148), ([1], 8, 148), ([400] * 149, 8, 148)])
def test_short_and_many_items_stay_whole(tiles, copies, blocks):
    assert ops.cut_portions(tiles, copies, blocks) is None


def test_no_memory_for_the_search_leaves_items_whole():
    # (a child process, whose address space is limited to little more than what it has)
    code = """
import resource
from llm_steadyinfer_b200.csrc import ops
ops.cut_portions([400] * 20, 8, 148)                     # (loads the library)
pages = int(open("/proc/self/statm").read().split()[0])
resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + (1 << 30),) * 2)
assert ops.cut_portions([400], 1 << 20, 2**31 - 1) is None       # asks for 17 GB
"""
    got = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert got.returncode == 0, got.stderr[-500:]
