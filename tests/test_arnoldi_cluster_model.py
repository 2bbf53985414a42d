"""CPU model of the one-launch Arnoldi step's protocol (csrc/arnoldi_cluster.cu): copy warp, compute
warps and cluster meetings as coroutines under random interleavings, with mbarrier phases, arrival
counts and copies that land late.  Every wait ends, no barrier gets more arrivals than a phase holds,
every slot read holds the vectors meant, and sums are read only when complete."""

import random

import pytest

WARPS = 8


class Barrier:
    def __init__(self, count):
        self.count, self.pending, self.tx, self.phase = count, count, 0, 0

    def arrive(self, tx=0):
        assert self.pending > 0, "more arrivals than the phase holds"
        self.pending -= 1
        self.tx += tx
        self._turn()

    def complete(self, tx):
        self.tx -= tx
        self._turn()

    def _turn(self):
        if self.pending == 0 and self.tx == 0:
            self.pending = self.count
            self.phase += 1

    def done(self, parity):  # mbarrier.test_wait.parity
        return (self.phase & 1) != parity


class Cta:
    def __init__(self, wr, slots, S):
        self.wc = WARPS // wr
        self.full = [[Barrier(1) for _ in range(slots)] for _ in range(self.wc)]
        self.empty = [[Barrier(wr) for _ in range(slots)] for _ in range(self.wc)]
        self.wq_full, self.wq_empty = Barrier(1), Barrier(WARPS)
        self.meet = [Barrier(S), Barrier(S)]
        self.data = [[None] * slots for _ in range(self.wc)]
        self.wq = None
        self.part = self.npart = None
        self.sync_n, self.sync_gen = 0, 0


def simulate(wr, slots, S, ns, probes, seed, keep_bug=False):
    rng = random.Random(seed)
    ctas = [Cta(wr, slots, S) for _ in range(S)]
    wc = WARPS // wr
    flying = []  # copies under way: callables that land them

    def of(g):
        return (ns - g + wc - 1) // wc if g < ns else 0

    def kept(g):
        return min(of(g), slots)

    def copier(c):
        fills, pos, par = [0] * wc, [0] * wc, [0] * wc
        for t in range(probes):
            if t > 1:
                while not c.wq_empty.done((t - 2) & 1):
                    yield
            if t > 0:  # the first probe's vectors are loaded directly
                c.wq_full.arrive(1)
                flying.append(lambda t=t: (setattr(c, "wq", t), c.wq_full.complete(1)))
            for again in range(2):
                for s in range(ns):
                    g = s % wc
                    if again and s // wc >= of(g) - kept(g):
                        continue
                    if fills[g] >= slots:
                        while not c.empty[g][pos[g]].done(par[g] ^ 1):
                            yield
                    c.full[g][pos[g]].arrive(1)

                    def land(g=g, at=pos[g], what=(t, s)):
                        c.data[g][at] = what
                        c.full[g][at].complete(1)

                    flying.append(land)
                    fills[g] += 1
                    pos[g] += 1
                    if pos[g] == slots:
                        pos[g], par[g] = 0, par[g] ^ 1
                    yield

    def cta_sync(c):
        gen = c.sync_gen
        c.sync_n += 1
        if c.sync_n == WARPS:
            c.sync_n, c.sync_gen = 0, gen + 1
        while c.sync_gen == gen:
            yield

    def compute(c, warp):
        group = warp // wr
        full, empty, data = c.full[group], c.empty[group], c.data[group]
        gs, gk = of(group), kept(group)
        pos = sp = par = 0

        def advance(pos, sp):
            return (0, sp ^ 1) if pos + 1 == slots else (pos + 1, sp)

        for t in range(probes):
            if t > 0:
                while not c.wq_full.done((t - 1) & 1):
                    yield
                assert c.wq == t
                yield
                assert c.wq == t
                c.wq_empty.arrive()
            kept_at = (pos, sp)
            for u in range(gs):
                if u == gs - gk:
                    kept_at = (pos, sp)
                while not full[pos].done(sp):
                    yield
                assert data[pos] == (t, u * wc + group)
                yield
                assert data[pos] == (t, u * wc + group)
                if u < gs - gk or keep_bug:
                    empty[pos].arrive()
                pos, sp = advance(pos, sp)
            yield from cta_sync(c)
            if warp == 0:
                c.part = t
            yield from cta_sync(c)
            if S > 1:
                if warp == 0:
                    for other in ctas:
                        other.meet[0].arrive()
                        yield
                while not c.meet[0].done(par):
                    yield
                for other in ctas:
                    assert other.part == t
                    yield
                yield from cta_sync(c)
            after = (pos, sp)
            pos, sp = kept_at
            for i in range(gs):
                if i == gk:
                    pos, sp = after
                u = gs - gk + i if i < gk else i - gk
                while not full[pos].done(sp):
                    yield
                assert data[pos] == (t, u * wc + group)
                yield
                assert data[pos] == (t, u * wc + group)
                empty[pos].arrive()
                pos, sp = advance(pos, sp)
            if gs == gk:
                pos, sp = after
            if wc > 1:
                yield from cta_sync(c)
            yield from cta_sync(c)
            if warp == 0:
                c.npart = t
                if S > 1:
                    for other in ctas:
                        other.meet[1].arrive()
                        yield
                    while not c.meet[1].done(par):
                        yield
                    for other in ctas:
                        assert other.npart == t
                        yield
            yield from cta_sync(c)
            par ^= 1

    agents = [copier(c) for c in ctas] + [compute(c, w) for c in ctas for w in range(WARPS)]
    idle = 0
    while agents:
        if flying and rng.random() < 0.3:
            flying.pop(rng.randrange(len(flying)))()  # copies land in any order
        a = rng.choice(agents)
        try:
            next(a)
        except StopIteration:
            agents.remove(a)
        idle += 1
        assert idle < 4_000_000, "a wait that does not end"
    assert not flying


@pytest.mark.parametrize("wr,slots,S", [(8, 5, 2), (8, 2, 1), (4, 3, 2), (2, 2, 4), (1, 2, 1), (1, 3, 2)])
@pytest.mark.parametrize("ns", [0, 1, 3, 9, 17])
def test_every_interleaving_ends_with_the_right_data(wr, slots, S, ns):
    for seed in range(3):
        simulate(wr, slots, S, ns, probes=4, seed=seed)


def test_the_model_sees_a_slot_released_too_early():
    with pytest.raises(AssertionError):
        simulate(8, 3, 1, 9, probes=3, seed=0, keep_bug=True)


def simulate_passes(wr, slots, S, ns, nsx, passes, norm, probes, seed):
    """The Gram-Schmidt / adjoint kernel (csrc/gs_cluster.cu): nsx slots read once, then `passes` passes over
    ns slots in rotated orders, a meeting of the cluster after every other pass (and after the norm)."""
    rng = random.Random(seed)
    ctas = [Cta(wr, slots, S) for _ in range(S)]
    for c in ctas:
        c.meet = [Barrier(S) for _ in range(3)]
        c.part = {}
    wc = WARPS // wr
    flying = []

    def of(g, n=ns):
        return (n - g + wc - 1) // wc if g < n else 0

    def copier(c):
        fills, pos, par = [0] * wc, [0] * wc, [0] * wc

        def fill(g, what):
            if fills[g] >= slots:
                while not c.empty[g][pos[g]].done(par[g] ^ 1):
                    yield
            c.full[g][pos[g]].arrive(1)

            def land(at=pos[g]):
                c.data[g][at] = what
                c.full[g][at].complete(1)

            flying.append(land)
            fills[g] += 1
            pos[g] += 1
            if pos[g] == slots:
                pos[g], par[g] = 0, par[g] ^ 1
            yield

        for b in range(probes):
            for s in range(nsx):
                yield from fill(s % wc, (b, "x", s))
            for t in range(1, passes + 1):
                for i in range(of(0)):
                    for g in range(wc):
                        gs = of(g)
                        gk = min(gs, slots)
                        if i >= gs or (t > 1 and i < gk):
                            continue
                        yield from fill(g, (b, "q", (i + (t - 1) * (gs - gk)) % gs * wc + g))

    def cta_sync(c):
        gen = c.sync_gen
        c.sync_n += 1
        if c.sync_n == WARPS:
            c.sync_n, c.sync_gen = 0, gen + 1
        while c.sync_gen == gen:
            yield

    def meet(c, warp, which, b):
        yield from cta_sync(c)
        if warp == 0:
            c.part[which, b & 1] = b
        yield from cta_sync(c)
        if S > 1:
            if warp == 0:
                for other in ctas:
                    other.meet[which].arrive()
                    yield
            while not c.meet[which].done(b & 1):
                yield
            for other in ctas:
                assert other.part[which, b & 1] == b
                yield
            yield from cta_sync(c)

    def compute(c, warp):
        group = warp // wr
        full, empty, data = c.full[group], c.empty[group], c.data[group]
        gs = of(group)
        gk = min(gs, slots)
        pos = sp = 0

        def advance():
            nonlocal pos, sp
            pos, sp = (0, sp ^ 1) if pos + 1 == slots else (pos + 1, sp)

        def use(what, release):
            while not full[pos].done(sp):
                yield
            assert data[pos] == what
            yield
            assert data[pos] == what
            if release:
                empty[pos].arrive()
            advance()

        for b in range(probes):
            for u in range(of(group, nsx)):
                yield from use((b, "x", u * wc + group), True)
            for t in range(1, passes + 1):
                u = (t - 1) * (gs - gk) % gs if gs else 0
                kept = (pos, sp)
                for i in range(gs):
                    if i == gs - gk:
                        kept = (pos, sp)
                    yield from use((b, "q", u * wc + group), t == passes or i < gs - gk)
                    u = 0 if u + 1 == gs else u + 1
                if t < passes:
                    pos, sp = kept
                if t % 2:
                    yield from meet(c, warp, t // 2, b)
                elif wc > 1:
                    yield from cta_sync(c)
            if norm:
                yield from meet(c, warp, 2, b)

    agents = [copier(c) for c in ctas] + [compute(c, w) for c in ctas for w in range(WARPS)]
    steps = 0
    while agents:
        if flying and rng.random() < 0.3:
            flying.pop(rng.randrange(len(flying)))()
        a = rng.choice(agents)
        try:
            next(a)
        except StopIteration:
            agents.remove(a)
        steps += 1
        assert steps < 4_000_000, "a wait that does not end"
    assert not flying


@pytest.mark.parametrize("wr,slots,S", [(8, 5, 2), (8, 2, 1), (4, 3, 2), (2, 2, 4), (1, 2, 1)])
@pytest.mark.parametrize("ns,nsx,passes,norm", [(0, 0, 4, True), (1, 0, 4, True), (7, 0, 2, True), (13, 0, 4, True),
                                                (1, 9, 2, False), (6, 4, 4, False), (17, 2, 4, False)])
def test_rotated_passes_end_with_the_right_data(wr, slots, S, ns, nsx, passes, norm):
    for seed in range(2):
        simulate_passes(wr, slots, S, ns, nsx, passes, norm, probes=3, seed=seed)
