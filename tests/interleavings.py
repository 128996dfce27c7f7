"""What the models of the kernels' hand-offs share: barriers that tell a phase's parity only, and roles that go on in random order at random speeds beside queues of
work (MMAs, commits) that runs some time after its issue, in order."""


class Barrier:
    def __init__(self, count):
        self.count, self.pending, self.done = count, count, 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0, "more arrivals than a phase has"
        if self.pending == 0:
            self.pending, self.done = self.count, self.done + 1

    def over(self, parity):  # what mbarrier.try_wait.parity can tell
        return (self.done - 1) & 1 == parity


def interleave(rng, roles, queues):
    """Runs generators that yield what they wait for, and pops calls off the queues, until nothing is left."""
    waits = {r: next(r, None) for r in roles}
    speed = {r: rng.choice([1, 1, 3, 20]) for r in roles}
    waits = {r: c for r, c in waits.items() if c is not None}
    while waits or any(queues):
        ready = [r for r, c in waits.items() if c()]
        pipe = [q for q in queues if q]
        assert ready or pipe, "nothing can go on"
        if pipe and (not ready or rng.random() < 0.3):
            rng.choice(pipe).pop(0)()
            continue
        r = rng.choices(ready, [1 / speed[x] for x in ready])[0]
        waits[r] = next(r, None)
        if waits[r] is None:
            del waits[r]
