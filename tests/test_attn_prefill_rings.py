"""The hand-offs of the prompt attention (csrc/attn_prefill.cu) under random interleavings, on the CPU: two buffers of K, of scores and of
probabilities by tile parity, one of V and one of output, waits that know a phase's parity only, MMAs that run in the order of their issue some time after it; and,
byte by byte, the shared memory through which the two soft-max warps of a row exchange its largest score, and hand on its sum at the end."""

import os
import random
import re

import pytest

from interleavings import Barrier, interleave

WARPS, SOFT = 4, 8  # warps that read the output; that make probabilities

with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yule_b200", "csrc", "attn_prefill.cu")) as f:
    SOURCE = f.read()


def exchange_of_the_source():
    """Bytes of a row's largest score, where it lies (b: tile parity), whether the two warps meet again after reading, and how many threads meet before the sums are stored over them."""
    kind, = re.findall(r"(unsigned short|float) \*most_row = ", SOURCE)
    index, = re.findall(r"most_row\[([^\]]*)\] = ", SOURCE)
    read, end, sums = SOURCE.index("const float mx = "), SOURCE.index("mbar_arrive(p_full"), SOURCE.index("sum_row[half * kRows + r] = l;")
    meet = re.findall(r"bar\.sync (?:%0|\d+), (\d+);", SOURCE[end:sums])
    return {"unsigned short": 2, "float": 4}[kind], index, "bar.sync" in SOURCE[read:end], int(meet[-1]) if meet else 0


class Meeting:
    """bar.sync of so many warps."""

    def __init__(self, warps):
        self.warps, self.here, self.over = warps, 0, 0

    def meet(self):
        mine = self.over
        self.here += 1
        if self.here == self.warps:
            self.here, self.over = 0, self.over + 1
        return lambda: self.over > mine


def simulate(seed, n, o_waits=True, alpha_waits=True, exchange=exchange_of_the_source()):
    rng = random.Random(seed)
    size, index, again, last_meeting = exchange
    place = lambda b, half, r: size * eval(index, {"b": b, "half": half, "kRows": 128, "r": r})  # noqa: E731
    memory = [None] * 1024
    pairs = [Meeting(2) for _ in range(4)]
    last = [Meeting(8)] * 4 if last_meeting == 256 else pairs
    assert last_meeting in (0, 64, 256)

    def store(at, width, what):
        memory[at:at + width] = [what] * width

    def check(at, width, what):
        assert memory[at:at + width] == [what] * width, f"{what} read, there is {memory[at:at + width]}"

    pair = lambda c: [Barrier(c), Barrier(c)]  # noqa: E731
    k_full, k_empty, s_full, s_empty, v_full, v_empty = pair(1), pair(1), pair(1), pair(SOFT), [Barrier(1)], [Barrier(1)]
    p_full, p_empty, a_empty, o_full, o_empty, l_full = pair(SOFT), pair(1), pair(WARPS), Barrier(2), Barrier(WARPS), Barrier(SOFT)
    kv = {"k": [[-1], [-1]], "v": [[-1]]}
    used = {"k": {-2, -1}, "v": {-2, -1}}
    scores, score_readers = [-1, -1], [SOFT, SOFT]
    probs, alpha, alpha_read = [[-2] * SOFT, [-1] * SOFT], [[-2] * WARPS, [-1] * WARPS], [[-2] * WARPS, [-1] * WARPS]
    out, out_readers, used_p = -1, WARPS, {-1, -2}
    queue = []

    def load(which):
        full, empty = (k_full, k_empty) if which == "k" else (v_full, v_empty)
        for j in range(n):
            b, ph = (j & 1, j >> 1 & 1) if which == "k" else (0, j & 1)
            yield lambda: empty[b].over(ph ^ 1)
            assert kv[which][b][0] in used[which], "operand overwritten before it was read"
            kv[which][b][0] = j
            yield lambda: True
            full[b].arrive()

    def issue():
        def run_scores(j):
            def go():
                b = j & 1
                assert all(x == j for x in kv["k"][j & 1]), "scores of another tile's K"
                assert score_readers[b] == SOFT, "scores overwritten before they were read"
                scores[b], score_readers[b] = j, 0
                used["k"].add(j)
            return go

        def run_out(j):
            def go():
                nonlocal out, out_readers
                assert all(x == j for x in kv["v"][0]) and all(x == j for x in probs[j & 1]), "output of other operands"
                assert out_readers == WARPS, "output overwritten before it was read"
                out, out_readers = j, 0
                used["v"].add(j)
                used_p.add(j)
            return go

        for j in range(n + 1):
            if j < n:  # scores of tile j before the output of tile j - 1
                b = j & 1
                yield lambda: s_empty[b].over(j >> 1 & 1 ^ 1)
                yield lambda: k_full[j & 1].over(j >> 1 & 1)
                queue.extend([run_scores(j), s_full[b].arrive, k_empty[j & 1].arrive])
            i = j - 1
            if i >= 0:
                yield lambda: v_full[0].over(i & 1)
                if o_waits:
                    yield lambda: o_empty.over(i & 1 ^ 1)
                yield lambda: p_full[i & 1].over(i >> 1 & 1)
                queue.extend([run_out(i), o_full.arrive, v_empty[0].arrive, p_empty[i & 1].arrive])
                o_full.arrive()

    def softmax(w):
        quarter, half = w & 3, w >> 2
        rows = (quarter * 32, quarter * 32 + 17, quarter * 32 + 31)
        for j in range(n):
            b = j & 1
            yield lambda: s_full[b].over(j >> 1 & 1)
            assert scores[b] == j
            for r in rows:
                store(place(b, half, r), size, ("largest", j, half, r))
            yield pairs[quarter].meet()
            yield lambda: True
            for r in rows:
                check(place(b, half ^ 1, r), size, ("largest", j, half ^ 1, r))
            if again:
                yield pairs[quarter].meet()
            yield lambda: p_empty[b].over(j >> 1 & 1 ^ 1)
            if alpha_waits:
                yield lambda: a_empty[b].over(j >> 1 & 1 ^ 1)
            assert probs[b][w] in used_p, "probabilities overwritten before they were used"
            if w < WARPS:
                assert alpha_read[b][w] == j - 2, "alpha overwritten before it was read"
                alpha[b][w] = j
            score_readers[b] += 1
            s_empty[b].arrive()
            yield lambda: True
            probs[b][w] = j
            p_full[b].arrive()
        if last_meeting:
            yield last[quarter].meet()
        for r in rows:
            store(4 * (half * 128 + r), 4, ("sum", half, r))
        l_full.arrive()

    def sums(w):
        nonlocal out_readers
        for j in range(n):
            yield lambda: o_full.over(j & 1)
            assert out == j and alpha[j & 1][w] == j, "output or alpha of another tile"
            alpha_read[j & 1][w] = j
            if alpha_waits:
                a_empty[j & 1].arrive()
            yield lambda: True
            out_readers += 1
            o_empty.arrive()
        yield lambda: l_full.over(0)
        for r in (w * 32, w * 32 + 17, w * 32 + 31):
            for half in (0, 1):
                check(4 * (half * 128 + r), 4, ("sum", half, r))

    roles = [issue()] + [softmax(w) for w in range(SOFT)] + [sums(w) for w in range(WARPS)] + [load(x) for x in "kv"]
    interleave(rng, roles, [queue])


@pytest.mark.parametrize("n", [1, 2, 3, 8, 13])
def test_hand_offs_hold(n):
    for seed in range(60):
        simulate(seed, n)


@pytest.mark.parametrize("missing", ["o_waits", "alpha_waits"])
def test_the_model_catches_a_missing_wait(missing):
    with pytest.raises(AssertionError):
        for seed in range(300):
            simulate(seed, 8, **{missing: False})


@pytest.mark.parametrize("exchange", [
    (2, "(b * 2 + half) * kRows + r", False, 64),  # scores in 16 bits under sums in 32, and only the two warps of a row meet in between
    (4, "half * kRows + r", False, 64),            # a row's own words, stored again before they are read
])
def test_the_model_catches_stores_over_what_is_still_to_be_read(exchange):
    with pytest.raises(AssertionError, match="read, there is"):
        for seed in range(300):
            simulate(seed, 4, exchange=exchange)
