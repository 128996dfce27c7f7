"""The rings of csrc/qgemm_int.cu under random interleavings, on the CPU: as test_gemm_rings.py, with one or two accumulators per stage, the offset's
accumulator behind the last stage of a super-block, and the ring of block scales that the unpacking warps store and the drain warps read."""

import os
import random
import re

import pytest

from interleavings import Barrier, interleave

with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yule_b200", "csrc", "qgemm_int.cu")) as f:
    SOURCE = f.read()
STAGES, SCALES = (int(re.search(rf"{n} = (\d+);", SOURCE).group(1)) for n in ("kStages", "kScaleRing"))
WARPS = 8


def accumulators(bn, w_cols):
    """kMainCols, kAccFit and NBUF of the source."""
    return min(8, (512 - STAGES * w_cols) // (2 * bn if bn <= 64 else bn))


CASES = [(bn, name, accumulators(bn, 64 if name == "q6" else 32)) for bn in (32, 64, 128) for name in ("block32", "q5", "q6")] + [(128, "q4k", accumulators(128, 32))]


def simulate(seed, nbuf, name, blocks, scale_ring=SCALES):
    rng = random.Random(seed)
    n, per = 4 * blocks, 2 if name == "block32" else 1
    closes = lambda i: name in ("q5", "q4k") and i % 4 == 3  # noqa: E731
    span = 2 if name == "q4k" else 1  # stages that share an accumulator
    full, empty = [[Barrier(c) for _ in range(STAGES)] for c in (WARPS + 1, 1)]
    acc_full, acc_empty = [[Barrier(c) for _ in range(nbuf)] for c in (2 if name == "block32" else 1, WARPS)]
    w = [[-1] * (WARPS + 1) for _ in range(STAGES)]
    ran, acc, readers = {-1}, [-1] * nbuf, [WARPS] * nbuf
    scales = [[-1] * WARPS for _ in range(scale_ring)]
    queues = [[], []]

    def producer(p):
        for i in range(n):
            s = i % STAGES
            yield lambda: empty[s].over(i // STAGES & 1 ^ 1)
            assert w[s][p] in ran, "operand overwritten before it was read"
            w[s][p] = i
            if p < WARPS:
                scales[i % scale_ring][p] = i
            full[s].arrive()

    def mma(stages, slot, a, first, frees):
        def go():
            assert all(t == i for i in stages for t in w[i % STAGES]), "MMA on operands of another stage"
            assert readers[slot] == WARPS or (not first and acc[slot] == a), "accumulator overwritten before it was drained"
            acc[slot], readers[slot] = a, 0
            ran.update(frees)
        return go

    def issuer(mine):
        a = 0
        for i in range(0, n, span):
            stages = range(i, i + span)
            uses = per + closes(stages[-1])
            if i // span & 1 == mine:
                for k in range(uses):
                    slot, ph = (a + k) % nbuf, (a + k) // nbuf & 1
                    yield lambda: acc_empty[slot].over(ph ^ 1)
                    if k == 0:
                        for j, t in enumerate(stages):
                            yield lambda: full[t % STAGES].over(t // STAGES & 1)
                            if j + 1 < span:  # the small products of the first stage go out before the second is there
                                queues[mine].append(mma([t], slot, a, True, []))
                    last = k == uses - 1
                    frees = (list(stages) if last else list(stages)[:-1]) if k == 0 else [stages[-1]] if last else []
                    queues[mine] += [mma(list(stages) if k == 0 or span == 1 else [stages[-1]], slot, a + k, k > 0 or span == 1, frees)]
                    queues[mine] += [empty[t % STAGES].arrive for t in frees] + [acc_full[slot].arrive]
                    if name == "block32":
                        acc_full[slot].arrive()
            a += uses

    def drain():
        a = 0
        for i in range(0, n, span):
            for k in range(per + closes(i + span - 1)):
                slot = a % nbuf
                yield lambda: acc_full[slot].over(a // nbuf & 1)
                assert acc[slot] == a, "drained another step's sums"
                assert name != "block32" or all(t == i for t in scales[i % scale_ring]), "scales of another stage"
                readers[slot] += 1
                acc_empty[slot].arrive()
                a += 1

    roles = [producer(p) for p in range(WARPS + 1)] + [issuer(0), issuer(1)] + [drain() for _ in range(WARPS)]
    interleave(rng, roles, queues)


@pytest.mark.parametrize("bn,name,nbuf", CASES)
def test_rings_hold(bn, name, nbuf):
    for seed in range(50):
        simulate(seed, nbuf, name, 1 + seed % 7)


def test_the_model_catches_rings_that_are_too_short():
    for nbuf, name, ring in ((2, "block32", SCALES), (2, "q5", SCALES), (2, "q4k", SCALES), (3, "block32", 4)):
        with pytest.raises(AssertionError):
            for seed in range(400):
                simulate(seed, nbuf, name, 6, ring)
