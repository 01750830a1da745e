"""The turns that the two query tiles of an attention work item take on the exponential unit,
walked through on the host with the ring of key blocks between them: no pair of key ranges
that takes turns may stop. (Every wait is for a count that only grows, so the order of the
steps does not matter.)"""
import itertools
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "svod_b200" / "csrc" / "attention_parts.cuh").read_text()
STAGES = int(re.search(r"kStages = (\d+);", SOURCE)[1])


def reach():
    """How far apart (in key blocks) the kernels let two ranges that take turns begin."""
    m = re.search(r"kTurnReach = (\d+);", SOURCE)
    return int(m[1]) if m else 1 << 30


def ends(ranges, paired, moved):
    """Whether an item over these key block ranges [lo, hi) ends; its first `paired` blocks take
    turns; `moved`: every block rescales the sum, which waits for the next block's scores."""
    lo, hi = min(r[0] for r in ranges), max(r[1] for r in ranges)
    at = dict(k=lo, v=lo)  # blocks brought so far
    k_free, v_free, scores, weights, products, turns = ([lo, lo], [lo, lo], [0, 0], [0, 0], [0, 0], [0, 0])

    def loader():
        for j in range(lo, hi):
            yield lambda: j - STAGES < min(k_free)
            at["k"] = j + 1
            yield lambda: j - STAGES < min(v_free)
            at["v"] = j + 1

    def issuer(i):
        a, b = ranges[i]
        for t in range(lo - 1, hi + 1):
            jq, jp = t + 1, t - 1
            if lo <= jq < hi:
                yield lambda: at["k"] > jq
            if lo <= jp < hi:
                yield lambda: at["v"] > jp
                if a <= jp < b:
                    yield lambda: weights[i] > jp - a
                    products[i] += 1
            if lo <= jq < hi and a <= jq < b:
                scores[i] += 1
            if lo <= jp < hi:
                v_free[i] = jp + 1
            if lo <= jq < hi:
                k_free[i] = jq + 1

    def softmax(i):
        blocks = ranges[i][1] - ranges[i][0]
        taken = 0
        for n in range(blocks):
            yield lambda: scores[i] > n
            if moved and n > 0:
                yield lambda: scores[i] > n + 1 if n + 1 < blocks else products[i] >= blocks - 1
            if n < paired and (i == 1 or n > 0):
                taken += 1
                yield lambda: turns[i] >= taken
            if n < paired and (i == 0 or n + 1 < paired):
                turns[1 - i] += 1
            if n + 1 == blocks and blocks > 1:
                yield lambda: products[i] >= blocks - 1
            weights[i] += 1

    running = [[g, None] for g in (loader(), issuer(0), issuer(1), softmax(0), softmax(1))]
    while running:
        progress = False
        for r in list(running):
            while r[1] is None or r[1]():
                progress = True
                try:
                    r[1] = next(r[0])
                except StopIteration:
                    running.remove(r)
                    break
        if not progress:
            return False
    return True


def paired_blocks(r0, r1, reach):
    return 0 if abs(r0[0] - r1[0]) > reach else min(r0[1] - r0[0], r1[1] - r1[0])


@pytest.mark.parametrize("moved", [False, True])
def test_no_pair_of_ranges_stops(moved):
    for lo0, lo1, n0, n1 in itertools.product((0, 1, 2, 3, 5, 6, 7, 9, 16), (0, 1, 2, 4, 6, 15), (1, 2, 3, 5, 8, 17),
                                              (1, 2, 3, 4, 9, 17)):
        r0, r1 = (lo0, lo0 + n0), (lo1, lo1 + n1)
        assert ends((r0, r1), paired_blocks(r0, r1, reach()), moved), (r0, r1)


def test_turns_of_ranges_far_apart_are_seen_to_stop():
    """What the walk is for: a chunk border or a segment's start inside an item moves the second
    tile's first block past what the ring can bring before the first tile's next turn."""
    assert not ends(((0, 32), (15, 32)), 17, False)
    assert not ends(((0, 6), (6, 8)), 2, False)
    assert ends(((0, 32), (15, 32)), 0, False) and ends(((0, 4), (2, 6)), 4, True)
