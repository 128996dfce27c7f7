"""The rings of the GEMM with W in tensor memory (csrc/qgemm_tc.cu) under random interleavings, on the CPU: four operand stages, an accumulator ring in
which the min term of a super-block takes a turn of its own, two issuing warps that alternate stages, waits that know a phase's parity only."""

import random

import pytest

from interleavings import Barrier, interleave
from test_gemm_pipeline_model import RINGS

STAGES, WARPS = RINGS["q4k-128"].stages, 8


def simulate(seed, nbuf, per_block, with_min, blocks):
    rng = random.Random(seed)
    n = blocks * per_block
    full, empty = [[Barrier(c) for _ in range(STAGES)] for c in (WARPS + 1, 1)]
    acc_full, acc_empty = [[Barrier(c) for _ in range(nbuf)] for c in (1, WARPS)]
    w = [[-1] * (WARPS + 1) for _ in range(STAGES)]  # stage whose bytes each producer (and the loader) has put there
    ran = {-1}                                       # stages whose MMAs have run
    acc, readers = [-1] * nbuf, [WARPS] * nbuf       # step an accumulator holds, warps that have drained it
    queues = [[], []]                                # issued and not yet run, per issuing warp

    def producer(p):
        for i in range(n):
            s = i % STAGES
            yield lambda: empty[s].over(i // STAGES & 1 ^ 1)
            assert w[s][p] in ran, "operand overwritten before it was read"
            w[s][p] = i
            full[s].arrive()

    def run_mma(s, i, slot, a, last):
        def go():
            assert all(t == i for t in w[s]), "MMA on operands of another stage"
            assert readers[slot] == WARPS, "accumulator overwritten before it was drained"
            acc[slot], readers[slot] = a, 0
            if last:
                ran.add(i)
        return go

    def issuer(mine):
        a = 0
        for i in range(n):
            s, closes = i % STAGES, with_min and i % per_block == per_block - 1
            if i & 1 == mine:
                for k in range(2 if closes else 1):
                    slot, ph = (a + k) % nbuf, (a + k) // nbuf & 1
                    yield lambda: acc_empty[slot].over(ph ^ 1)
                    if k == 0:
                        yield lambda: full[s].over(i // STAGES & 1)
                    last = not closes or k == 1
                    queues[mine] += [run_mma(s, i, slot, a + k, last), acc_full[slot].arrive]
                    if last:
                        queues[mine].append(empty[s].arrive)
            a += 2 if closes else 1

    def drain():
        steps = n + (blocks if with_min else 0)
        for a in range(steps):
            slot = a % nbuf
            yield lambda: acc_full[slot].over(a // nbuf & 1)
            assert acc[slot] == a, "drained another step's sums"
            readers[slot] += 1
            acc_empty[slot].arrive()

    roles = [producer(p) for p in range(WARPS + 1)] + [issuer(0), issuer(1)] + [drain() for _ in range(WARPS)]
    interleave(rng, roles, queues)


# accumulators, stages per super-block, min term of every instantiation, as the source has them
@pytest.mark.parametrize("nbuf,per_block,with_min", sorted({(c.nbuf, c.stages_per_unit, c.min_term) for c in RINGS.values()}))
def test_rings_hold(nbuf, per_block, with_min):
    for seed in range(60):
        simulate(seed, nbuf, per_block, with_min, 1 + seed % 7)


def test_the_model_catches_a_ring_that_is_too_short():
    """With one accumulator fewer than the parities need, a warp takes the phase before last for the last."""
    with pytest.raises(AssertionError):
        for seed in range(400):
            simulate(seed, 2, 4, True, 6)
