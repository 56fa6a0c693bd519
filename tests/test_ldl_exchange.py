"""CPU model of the exchange of the cluster LDL^T solve (k_ldl_factor_solve in
thesis-emx-bach_gb300/csrc/xb_ldl.cu).

Every CTA runs the same phases, apart from each other by the split barrier of the
cluster (arrive, then wait).  Factorisation of panel p: read Tg, the gathered
diagonal block; write the own rows of Yg in global memory; barrier; read all rows of
Yg into Y; push the next panel's diagonal rows into every CTA's Tg; barrier, under
which the update still reads Y.  Then the inverses through Yg and three triangular
passes, each with one barrier per panel and a pair of buffers (SB, FB) by the
panel's parity.

The model runs the CTAs' phases interleaved step by step (random schedules) and
checks that the barrier is never arrived at twice without a wait, that nobody
writes a buffer that another CTA is reading, that every read finds the values of
its own panel from every CTA, and that all CTAs end.  No GPU is involved."""
import random

import pytest


class Cluster:
    def __init__(self, cl):
        self.cl = cl
        self.gen = self.arrived = 0
        self.mine = [0] * cl
        self.waited = [True] * cl
        self.data = {}      # (buffer, owner, writer) -> value
        self.reading = {}   # (buffer, owner) -> CTAs that read it now

    def arrive(self, r):
        assert self.waited[r], "two arrivals without a wait"
        self.waited[r] = False
        self.mine[r] += 1
        self.arrived += 1
        if self.arrived == self.cl:
            self.arrived = 0
            self.gen += 1

    def wait(self, r):
        while self.gen < self.mine[r]:
            yield "wait"
        self.waited[r] = True

    def sync(self, r):
        self.arrive(r)
        yield from self.wait(r)

    def write(self, buf, owner, r, value):
        others = self.reading.get((buf, owner), set()) - {r}
        assert not others, f"CTA {r} writes {buf} of {owner}, which {others} read"
        self.data[buf, owner, r] = value

    def read(self, buf, owner, r, value, writers):
        """Reads the parts of all writers, one step each."""
        self.reading.setdefault((buf, owner), set()).add(r)
        for q in writers:
            assert self.data.get((buf, owner, q)) == value, (buf, owner, q, value)
            yield "step"
        self.reading[buf, owner].discard(r)


def cta(c, r, n_panels, flagged):
    everyone = list(range(c.cl))

    def push(buf, value):
        for d in random.sample(everyone, c.cl):
            c.write(buf, d, r, value)
            yield "step"

    yield from c.sync(r)
    yield from push("Tg", 0)
    yield from c.sync(r)
    for p in range(n_panels):
        yield from c.read("Tg", r, r, p, everyone)
        c.write("Yg", "all", r, p)
        yield "step"
        if p + 1 == n_panels:
            break
        c.arrive(r)
        if p:  # the rest of the update of the panel before
            yield from c.read("Y", r, r, p - 1, [r])
        yield from c.wait(r)
        yield from c.read("Yg", "all", r, p, everyone)
        c.write("Y", r, r, p)
        yield from push("Tg", p + 1)
        c.arrive(r)
        yield from c.read("Y", r, r, p, [r])
        yield from c.wait(r)
    if flagged:
        yield from c.sync(r)
        return
    c.write("Yg", "all", r, "inverses")
    yield from c.sync(r)
    yield from c.read("Yg", "all", r, "inverses", everyone)
    c.write("Y", r, r, "inverses")

    def triangular(name, buf, panels):
        for p in panels:
            yield from push((buf, p & 1), (name, p))
            c.arrive(r)
            yield "step"  # what was known already is added under the barrier
            yield from c.wait(r)
            yield from c.read((buf, p & 1), r, r, (name, p), everyone)
            yield from c.read("Y", r, r, "inverses", [r])

    yield from triangular("backward 1", "SB", reversed(range(n_panels)))
    yield from triangular("forward", "FB", range(n_panels))
    yield from triangular("backward 2", "SB", reversed(range(n_panels)))
    yield from c.sync(r)


@pytest.mark.parametrize("cl", [16, 8])
@pytest.mark.parametrize("n_panels", [1, 2, 3, 4, 7, 10])
def test_exchange(cl, n_panels):
    for seed in range(12):
        rng = random.Random(seed)
        random.seed(seed)
        c = Cluster(cl)
        runs = {r: cta(c, r, n_panels, seed % 4 == 3) for r in range(cl)}
        slow = rng.randrange(cl) if seed % 2 else None  # one CTA far behind
        idle = 0
        while runs:
            r = rng.choice(list(runs))
            if r == slow and rng.random() < 0.9:
                continue
            try:
                idle = idle + 1 if next(runs[r]) == "wait" else 0
            except StopIteration:
                del runs[r]
                idle = 0
            assert idle < 400 * cl, "no CTA can go on"
        assert c.arrived == 0 and all(c.waited)
