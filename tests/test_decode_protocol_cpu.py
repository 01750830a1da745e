"""The hand-over of blocks inside the decode attention kernel, walked through in every
order its warps can take: the MMA issuer, softmax warps and the barriers between them,
with the barrier and parity expressions read from the kernel's source."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "svod_b200" / "csrc" / "attention_decode.cu").read_text()
WARPS = 2  # of the four softmax warps: two are enough for every order of arrivals


def _expr(text):
    """A C index expression of `j` as a function."""
    code = compile(text, "<kernel>", "eval")
    return lambda j: int(eval(code, {"j": j}))


def _p_full():
    """(barrier, parity) the issuer waits on for block j's weights, and the barrier a warp arrives on."""
    wait = re.search(r"mbar_wait\(&?p_full(?:\[([^\]]*)\])?, ([^,]*), p\.status\)", SOURCE)
    arrive = re.search(r"mbar_arrive\(&?p_full(?:\[([^\]]*)\])?\)", SOURCE)
    return _expr(wait[1] or "0"), _expr(wait[2]), _expr(arrive[1] or "0")


def explore(n, bufs, index, parity, arrive):
    """Every state reachable with `n` blocks and `bufs` buffers of weights. Fails on a state
    nobody can leave, on a block multiplied before its weights are there, and on scores or
    weights written over before they are read."""
    # issuer: (block, step); each warp: (block, step, whether the maximum moved); phases of s_full[2], p_full[2],
    # pv_done[2]; arrivals pending on p_full[2]; scores issued, products issued
    start = ((0, 0), ((0, 0, 0),) * WARPS, (0, 0), (0, 0), (0, 0), (0, 0), 0, 0)
    passed = lambda phases, b, par: (phases[b] & 1) != par
    bump = lambda t, b, by=1: tuple(x + by if i == b else x for i, x in enumerate(t))
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        (ij, istep), warps, s_ph, p_ph, v_ph, pend, scores, products = state
        after = []
        # ---- issuer: scores(0); then per block scores(j + 1), wait for the weights, the product
        if istep == 0:
            want = 1 if ij == 0 and scores == 0 else min(ij + 2, n)
            if scores < want:
                b = scores
                # the score buffer of block b - 2 has been read by every warp
                assert b < 2 or all(w[0] > b - 2 or (w[0] == b - 2 and w[1] == 4) for w in warps), "scores written over"
                after.append(((ij, 0), warps, bump(s_ph, b & 1), p_ph, v_ph, pend, scores + 1, products))
            elif ij < n:
                after.append(((ij, 1), warps, s_ph, p_ph, v_ph, pend, scores, products))
        elif passed(p_ph, index(ij), parity(ij)):
            assert all(w[0] > ij for w in warps), "weights read before they are there"
            after.append(((ij + 1, 0), warps, s_ph, p_ph, bump(v_ph, ij & 1), pend, scores, products + 1))
        # ---- a softmax warp: wait for the scores, meet the others, (rescale,) wait for the buffer, write, arrive
        for k, (j, step, moved) in enumerate(warps):
            put = lambda *w: warps[:k] + (w,) + warps[k + 1:]
            if j == n:
                continue
            if step == 0 and passed(s_ph, j & 1, (j >> 1) & 1):
                assert scores > j, "scores read before they are there"
                after.append(((ij, istep), put(j, 1, 0), s_ph, p_ph, v_ph, pend, scores, products))
            elif step == 1 and all(w[0] == j and w[1] == 1 for w in warps):  # the block's maxima: all meet
                for m in ((0, 1) if j > 0 else (0,)):
                    after.append(((ij, istep), ((j, 2, m),) * WARPS, s_ph, p_ph, v_ph, pend, scores, products))
            elif step == 2 and (not moved or passed(v_ph, (j - 1) & 1, ((j - 1) >> 1) & 1)):
                assert not moved or products >= j, "the sum rescaled before the last product"
                after.append(((ij, istep), put(j, 3, 0), s_ph, p_ph, v_ph, pend, scores, products))
            elif step == 3 and (j < bufs or passed(v_ph, (j - bufs) & 1, ((j - bufs) >> 1) & 1)):
                assert products >= j - bufs + 1, "weights written over"
                after.append(((ij, istep), put(j, 4, 0), s_ph, p_ph, v_ph, pend, scores, products))
            elif step == 4:
                b = arrive(j)
                q, ph = bump(pend, b), p_ph
                if q[b] == WARPS:
                    q, ph = bump(q, b, -WARPS), bump(p_ph, b)
                after.append(((ij, istep), put(j + 1, 0, 0), s_ph, ph, v_ph, q, scores, products))
        done = ij == n and all(w[0] == n for w in warps)
        assert after or done, f"nobody can go on: issuer at block {ij}, warps at {[w[0] for w in warps]}"
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)


@pytest.mark.parametrize("bufs", [1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 7])
def test_no_order_of_the_warps_stops_or_overtakes(n, bufs):
    explore(n, bufs, *_p_full())


def test_one_barrier_for_two_buffers_of_weights_is_seen_to_stop():
    """What the walk is for: with one barrier the warps may complete its next phase before
    the issuer has looked at the one before, which then reads as not complete."""
    one = (lambda j: 0, lambda j: j & 1, lambda j: 0)
    explore(7, 1, *one)
    with pytest.raises(AssertionError, match="nobody can go on"):
        explore(7, 2, *one)
