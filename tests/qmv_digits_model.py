"""A model of the hand-offs inside the one-vector matvec kernel (yule_b200/csrc/qmv_digits.cu), for checking the protocol on the
CPU under many interleavings.  It models the barriers and the buffers they guard, nothing of the arithmetic:

* weight stages (ring of ``slots``): filled by the copying warp, read by every multiplying warp, which then arrives on the
  stage's ``empty`` barrier;
* sums of a unit (``finish`` buffers in turn): written by every multiplying warp, added up by one of them (unit k: warp
  k mod warps), which waits for all the others.

Every wait on a stage is bounded.  ``fail_at`` makes it run out: from that scheduler step on the context's status word is
set and no copy lands any more; a warp that finds its stage missing gives up waiting for stages and goes on through its units.
The sums of a unit meet at a named barrier: an arrival count that starts over when it is full, whoever arrived, and
waits that have no bound; ``more_barriers`` than buffers, because a warp may give up one unit further on than the ring would
let it come.  ``dead_waits``: a warp that gave up waits for the others at every unit (as the kernel has it), or
(False) arrives and goes on, as a healthy one that does not finish the unit.  ``dead_keeps``: a warp that gave
up releases no stage; where it does, the copying warp asks for a stage again whose last copy may still be on its way.

Checks: sums are complete when they are added up and not overwritten before (runs without a failure), no barrier gets more
arrivals than its phase takes, and everybody gets to the end."""

from __future__ import annotations

import random
from dataclasses import dataclass

from gemm_pipeline_model import Barrier, ProtocolViolation


@dataclass
class Config:
    warps: int = 16
    slots: int = 4
    finish: int = 3
    units: int = 12
    stages_per_unit: int = 1
    dead_waits: bool = True
    dead_keeps: bool = True
    more_barriers: int = 1
    fail_at: int | None = None


def finish_buffers(slots: int, stages_per_unit: int) -> int:
    """As the host picks it: a warp may be a whole ring ahead of the one that finishes a unit."""
    return 2 + (slots - 1 + stages_per_unit - 1) // stages_per_unit


class NamedBarrier:
    def __init__(self, count: int):
        self.count, self.arrived, self.phase = count, 0, 0

    def arrive(self):
        self.arrived += 1
        if self.arrived == self.count:
            self.arrived = 0
            self.phase += 1


class State:
    def __init__(self, cfg: Config):
        self.cfg = cfg
        self.full = [Barrier(f"full[{s}]", 1) for s in range(cfg.slots)]
        self.empty = [Barrier(f"empty[{s}]", cfg.warps) for s in range(cfg.slots)]
        self.sums = [NamedBarrier(cfg.warps) for _ in range(cfg.finish + cfg.more_barriers)]
        self.written = [set() for _ in range(cfg.units)]  # warps whose sums of unit k are parked
        self.added = [False] * cfg.units
        self.in_flight = []
        self.failed = False   # the status word


# What an agent yields is (condition, bounded): it goes on once the condition holds (sent True), or, if the wait is bounded
# and the status word is set, it may give up (sent False).
def copier(st: State):
    c = st.cfg
    for j in range(c.units * c.stages_per_unit):
        s, ph = j % c.slots, (j // c.slots) & 1
        if not (yield (lambda: st.empty[s].test(ph ^ 1)), True):
            return
        st.full[s].arrive_expect_tx()
        st.in_flight.append(s)
        yield (lambda: True), False


def engine(st: State, done):
    """Lands copies until the failure, then none."""
    while not done() and not st.failed:
        yield (lambda: bool(st.in_flight) or done() or st.failed), False
        if st.in_flight and not st.failed:
            st.full[st.in_flight.pop(st.rng.randrange(len(st.in_flight)))].complete_tx()


def warp(st: State, w: int):
    c = st.cfg
    dead, j = False, 0
    for k in range(c.units):
        for _ in range(c.stages_per_unit):
            s, ph = j % c.slots, (j // c.slots) & 1
            j += 1
            if not dead:
                dead = not (yield (lambda: st.full[s].test(ph)), True)
            if not (dead and c.dead_keeps):
                st.empty[s].arrive()
            yield (lambda: True), False
        if not st.failed:
            if k >= c.finish and not st.added[k - c.finish]:
                raise ProtocolViolation(f"warp {w}: sums of unit {k} over those of unit {k - c.finish}, not added up yet")
            st.written[k].add(w)
        bar = st.sums[k % len(st.sums)]
        phase = bar.phase
        bar.arrive()
        if k % c.warps == w or (dead and c.dead_waits):
            yield (lambda: bar.phase > phase), False
        if k % c.warps == w:
            if not st.failed and len(st.written[k]) != c.warps:
                raise ProtocolViolation(f"warp {w}: unit {k} added up with sums missing")
            st.added[k] = True
        yield (lambda: True), False


def run(cfg: Config, seed: int, max_steps: int = 100000) -> None:
    """One random interleaving to its end.  Raises ProtocolViolation on a broken invariant or a deadlock."""
    st = State(cfg)
    st.rng = rng = random.Random(seed)
    workers = {f"warp{w}": warp(st, w) for w in range(cfg.warps)}
    workers["copier"] = copier(st)
    agents = dict(workers)
    agents["engine"] = engine(st, lambda: not any(n in agents for n in workers))
    speed = {n: rng.choice((1, 1, 2, 4, 16)) for n in agents}
    want = {n: next(a) for n, a in agents.items()}
    for step in range(max_steps):
        if not any(n in agents for n in workers):
            return
        if cfg.fail_at is not None and step >= cfg.fail_at:
            st.failed = True
        ready = [n for n in agents if want[n][0]()]
        quits = [n for n in agents if n not in ready and want[n][1] and st.failed]
        pool = [n for n in ready + quits for _ in range(speed[n])]
        if not pool:
            raise ProtocolViolation(f"deadlock: {sorted(agents)} wait")
        n = rng.choice(pool)
        try:
            want[n] = agents[n].send(n in ready)
        except StopIteration:
            del agents[n]
    raise ProtocolViolation("no end in sight")
