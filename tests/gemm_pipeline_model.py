"""A model of the hand-offs inside the tcgen05 GEMM kernel (yule_b200/csrc/qgemm_tc.cu), for checking the protocol on the
CPU under many interleavings.  It models what the kernel's roles do to the mbarriers and to the buffers they guard,
nothing of the arithmetic:

* operand stages (ring of ``stages``): filled by the unpacking warps (W, in tensor memory) and by the loader's bulk copy (x
  slabs), read by the MMAs of that stage, released by ``tcgen05.commit`` on the stage's ``empty`` barrier;
* raw boxes (ring of ``raw_slots``): filled by the tiled TMA load of one super-block, read by every unpacking warp;
* accumulators (ring of ``nbuf``): written by the MMAs of a stage, read by every drain warp.  With ``min_term`` (the Q4_K
  kernel) the stage that ends a super-block is followed by its min term, which reads the same stage and takes the next accumulator;
* two issuing warps on alternate stages, each committing only its own MMAs;
* without ``min_term`` (the kernel for the other formats) there are no raw boxes: the unpacking warps copy the bytes of a super-block
  themselves and meet at a named barrier before and after they unpack it, a wait that has no bound.

An mbarrier here is what the hardware gives: an arrival count per phase, an optional transaction count, and a wait
that knows only the PARITY of the phase it wants, so it cannot tell phase k from phase k - 2.  The checks: no arrival
beyond a phase's count, no buffer written before its last reader is done, no buffer read before its writers are
done, and no deadlock.  The scheduler resumes one runnable agent at a time, chosen at random with per-agent speeds
drawn per run, so slow and fast roles of every kind occur.

Every wait on an mbarrier is bounded.  ``fail_at`` makes them run out: from that scheduler step on no copy lands any more, and a wait whose
condition does not hold may give up (the kernel's abort flag).  Then nothing is checked but that everybody gets to the end.

Variants: ``teams`` lets two teams of unpacking warps take alternate stages (each waits on every other phase of a
stage's ``empty`` barrier), ``producers_leave`` lets an unpacking warp that gave up leave the named barriers to the others.
Both are broken, as is an accumulator ring that is too short for the parities; the tests show that the model finds it."""

from __future__ import annotations

import random
from dataclasses import dataclass


class ProtocolViolation(AssertionError):
    pass


class Barrier:
    """Phase k is in progress; phases 0 .. k-1 are complete.  ``test(parity)`` is mbarrier.try_wait.parity: true when
    the phase with that parity is not the one in progress."""

    def __init__(self, name: str, count: int):
        self.name, self.count = name, count
        self.pending, self.tx, self.phase = count, 0, 0

    def _maybe_complete(self):
        if self.pending == 0 and self.tx == 0:
            self.phase += 1
            self.pending = self.count

    def arrive(self):
        if self.pending == 0:
            raise ProtocolViolation(f"{self.name}: arrival beyond the count of phase {self.phase}")
        self.pending -= 1
        self._maybe_complete()

    def arrive_expect_tx(self):
        self.tx += 1
        self.arrive()

    def complete_tx(self):
        if self.tx == 0:
            raise ProtocolViolation(f"{self.name}: transaction bytes nobody announced")
        self.tx -= 1
        self._maybe_complete()

    def test(self, parity: int) -> bool:
        return (self.phase & 1) != parity


@dataclass
class Config:
    stages: int = 4
    nbuf: int = 3
    raw_slots: int = 3
    stages_per_unit: int = 4      # stages per super-block
    units: int = 9                # super-blocks this CTA walks through
    producer_warps: int = 4
    drain_warps: int = 2
    min_term: bool = True
    teams: bool = False
    producers_leave: bool = False
    fail_at: int | None = None


class State:
    def __init__(self, cfg: Config, rng: random.Random):
        c = self.cfg = cfg
        self.rng, self.failed, self.finished_issuers = rng, False, False
        writers = c.producer_warps // 2 if c.teams else c.producer_warps
        self.full = [Barrier(f"full[{s}]", writers + 1) for s in range(c.stages)]
        self.empty = [Barrier(f"empty[{s}]", 1) for s in range(c.stages)]
        self.acc_full = [Barrier(f"acc_full[{b}]", 1) for b in range(c.nbuf)]
        self.acc_empty = [Barrier(f"acc_empty[{b}]", c.drain_warps) for b in range(c.nbuf)]
        self.raw_full = [Barrier(f"raw_full[{r}]", 1) for r in range(c.raw_slots)]
        self.raw_empty = [Barrier(f"raw_empty[{r}]", c.producer_warps) for r in range(c.raw_slots)]
        n = self.n_stages = c.units * c.stages_per_unit
        self.n_steps = n + (c.units if c.min_term else 0)  # uses of accumulators
        self.w_written = [set() for _ in range(n)]    # per stage use j: the warps that wrote its W operand
        self.x_landed = [False] * n
        self.stage_read = [False] * n                 # its MMAs, the min term among them, have run
        self.computed = [False] * self.n_steps
        self.drained = [set() for _ in range(self.n_steps)]
        self.raw_landed = [False] * c.units
        self.raw_read = [set() for _ in range(c.units)]
        self.pipe = [[], []]                          # per issuing warp: issued, not yet executed
        self.copies = []                              # bulk copies in flight: callables that land them
        self.met, self.meetings = 0, 0                # the named barrier of the unpacking warps

    def check(self, holds: bool, what: str):
        if not holds and not self.failed:
            raise ProtocolViolation(what)

    def closes(self, j: int) -> bool:
        return self.cfg.min_term and j % self.cfg.stages_per_unit == self.cfg.stages_per_unit - 1

    def writers_of(self, j: int) -> set:
        c = self.cfg
        half = c.producer_warps // 2
        return set(range(j % 2 * half, j % 2 * half + half)) if c.teams else set(range(c.producer_warps))


# What an agent yields is (condition, bounded): it goes on once the condition holds (sent True), or, if the wait is bounded and the
# copies have stopped, it may give up (sent False).
def wait(bar: Barrier, parity: int):
    return (lambda: bar.test(parity)), True


GO_ON = (lambda: True), False


def loader(st: State):
    """One thread: the x slabs of every stage (waits for the stage to be free, announces the bytes, issues the copy)."""
    c = st.cfg
    for j in range(st.n_stages):
        s, ph = j % c.stages, (j // c.stages) & 1
        if not (yield wait(st.empty[s], ph ^ 1)):
            return
        st.check(j < c.stages or st.stage_read[j - c.stages], f"loader: x slab of stage {j} asked for before the MMAs of the stage in slot {s}")
        st.full[s].arrive_expect_tx()

        def land(j=j, s=s):
            st.x_landed[j] = True
            st.full[s].complete_tx()
        st.copies.append(land)
        yield GO_ON


def raw_loader(st: State):
    c = st.cfg
    for u in range(c.units):
        r, ph = u % c.raw_slots, (u // c.raw_slots) & 1
        if not (yield wait(st.raw_empty[r], ph ^ 1)):
            return
        st.check(u < c.raw_slots or len(st.raw_read[u - c.raw_slots]) == c.producer_warps, f"raw loader: box {r} refilled for unit {u} before every warp read it")
        st.raw_full[r].arrive_expect_tx()

        def land(u=u, r=r):
            st.raw_landed[u] = True
            st.raw_full[r].complete_tx()
        st.copies.append(land)
        yield GO_ON


def copy_engine(st: State):
    """Lands the bulk copies in flight, in any order; after the failure, none."""
    while True:
        yield (lambda: bool(st.copies) or st.finished_issuers or st.failed), False
        if st.failed or not st.copies:
            return
        st.copies.pop(st.rng.randrange(len(st.copies)))()
        yield GO_ON


def meet(st: State):
    """bar.sync of the unpacking warps: ends when as many have arrived as there are."""
    meeting = st.meetings
    st.met += 1
    if st.met == st.cfg.producer_warps:
        st.met, st.meetings = 0, meeting + 1
    return (lambda: st.meetings > meeting), False


def producer(st: State, warp: int):
    c = st.cfg
    half = c.producer_warps // 2
    team = warp // half if c.teams else 0
    dead = False
    for u in range(c.units):
        r, ph = u % c.raw_slots, (u // c.raw_slots) & 1
        if c.min_term:
            if not (yield wait(st.raw_full[r], ph)):
                return
            st.check(st.raw_landed[u], f"warp {warp}: read raw box {r} for unit {u} before it landed")
            st.raw_read[u].add(warp)
            yield GO_ON
        else:
            if dead and c.producers_leave:
                return
            yield meet(st)
        for g in range(c.stages_per_unit):
            if dead or (c.teams and g % 2 != team):
                continue
            j = u * c.stages_per_unit + g
            s, sph = j % c.stages, (j // c.stages) & 1
            if not (yield wait(st.empty[s], sph ^ 1)):
                dead = True
                continue
            st.check(j < c.stages or st.stage_read[j - c.stages], f"warp {warp}: W of stage {j} written while an MMA has not read slot {s}")
            st.w_written[j].add(warp)
            yield GO_ON
            st.full[s].arrive()
            yield GO_ON
        if c.min_term:
            if dead:
                return
            st.raw_empty[r].arrive()
            yield GO_ON
        else:
            yield meet(st)


def issuer(st: State, t: int):
    c = st.cfg
    a = 0  # the next use of an accumulator
    for j in range(st.n_stages):
        if j % 2 == t:
            s, ph = j % c.stages, (j // c.stages) & 1
            if not (yield wait(st.acc_empty[a % c.nbuf], (a // c.nbuf & 1) ^ 1)) or not (yield wait(st.full[s], ph)):
                return
            st.pipe[t] += [("mma", j, a), ("commit", [st.acc_full[a % c.nbuf]] + ([] if st.closes(j) else [st.empty[s]]))]
            yield GO_ON
            if st.closes(j):
                m = a + 1
                if not (yield wait(st.acc_empty[m % c.nbuf], (m // c.nbuf & 1) ^ 1)):
                    return
                st.pipe[t] += [("min", j, m), ("commit", [st.acc_full[m % c.nbuf], st.empty[s]])]
                yield GO_ON
        a += 2 if st.closes(j) else 1


def tensor_pipe(st: State):
    """Executes each warp's MMAs in its issue order, the two warps' in any order; a commit arrives when the MMAs its warp
    issued before it are done."""
    c = st.cfg
    while True:
        yield (lambda: any(st.pipe) or st.finished_issuers), False
        ready = [t for t in (0, 1) if st.pipe[t]]
        if not ready:
            return
        what = st.pipe[st.rng.choice(ready)].pop(0)
        if what[0] == "commit":
            for bar in what[1]:
                bar.arrive()
        else:
            kind, j, a = what
            st.check(st.w_written[j] == st.writers_of(j) and st.x_landed[j], f"MMA of stage {j} ran before its operands were complete")
            st.check(a < c.nbuf or len(st.drained[a - c.nbuf]) == c.drain_warps, f"accumulator {a % c.nbuf} overwritten before it was drained")
            st.computed[a] = True
            st.stage_read[j] = kind == "min" or not st.closes(j)
        yield GO_ON


def drain(st: State, warp: int):
    c = st.cfg
    for a in range(st.n_steps):
        if not (yield wait(st.acc_full[a % c.nbuf], a // c.nbuf & 1)):
            return
        st.check(st.computed[a] and (a + c.nbuf >= st.n_steps or not st.computed[a + c.nbuf]), f"drain warp {warp}: read accumulator {a % c.nbuf} at another use than {a}")
        st.drained[a].add(warp)
        yield GO_ON
        st.acc_empty[a % c.nbuf].arrive()
        yield GO_ON


def run(cfg: Config, seed: int, max_steps: int = 200000) -> None:
    """One random interleaving to completion.  Raises ProtocolViolation on a broken invariant or a deadlock."""
    rng = random.Random(seed)
    st = State(cfg, rng)
    issuers = {"loader": loader(st), "mma0": issuer(st, 0), "mma1": issuer(st, 1)}
    if cfg.min_term:
        issuers["raw"] = raw_loader(st)
    for w in range(cfg.producer_warps):
        issuers[f"prod{w}"] = producer(st, w)
    for w in range(cfg.drain_warps):
        issuers[f"drain{w}"] = drain(st, w)
    agents = {**issuers, "copy": copy_engine(st), "pipe": tensor_pipe(st)}
    speed = {name: rng.choice((1, 1, 2, 4, 16)) for name in agents}  # some roles much slower than others, per run
    want = {name: next(agent) for name, agent in agents.items()}
    for step in range(max_steps):
        st.failed = st.failed or (cfg.fail_at is not None and step >= cfg.fail_at)
        st.finished_issuers = all(name not in agents for name in issuers)
        ready = [n for n in agents if want[n][0]()]
        quits = [n for n in agents if st.failed and want[n][1] and n not in ready]
        if not agents:
            return
        if not ready and not quits:
            raise ProtocolViolation(f"deadlock: {sorted(agents)} wait forever")
        name = rng.choices(ready + quits, weights=[1.0 / speed[n] for n in ready + quits])[0]
        try:
            want[name] = agents[name].send(name in ready)
        except StopIteration:
            del agents[name], want[name]
    raise ProtocolViolation("no completion within the step budget")
