"""The asynchronous kernel's credit and idle reports, restated on the CPU.

`k_sssp_async` (medusa_b200/csrc/sssp_async.cuh) ends when two sums of counters
are equal and raises its threshold when every CTA is idle at once:

  * a warp holds credit, the bits it may set: taken from its `p` slot (added, the
    add awaited) before it sets one, spent by a bit newly set, earned by a claim
    finished, and given back to its `d` slot by an add that nothing waits for when
    a pass finds no work.  Every `d` read, then every `p`: equal sums end the run;
  * a warp that finds nothing below the threshold reports itself idle in its
    CTA's word (phase, warps); the CTA's last one adds the CTA to the phase's
    count, and whoever makes that count full and claims the phase in `open`
    raises the threshold.  With idle_back a warp that finds work again takes its
    report back, and its next report waits for that.

Warps are generators that yield at every memory operation, operations that
nothing waits for are performed later, and a seeded scheduler interleaves them
all.  The run must end, with the exact distances, and at the moment the check
passes no bit is set, no claim held and no credit out.  A warp that gives its
credit back before its claims are finished must be caught."""
import numpy as np
import pytest

SLOTS = 4
INF = float("inf")


def bellman_ford(V, src, dst, w):
    d = np.full(V, INF)
    d[0] = 0.0
    while True:
        nd = d.copy()
        np.minimum.at(nd, dst, d[src] + w)
        if (nd == d).all():
            return d
        d = nd


class Machine:
    def __init__(self, rng, V, src, dst, w, ctas, warps, delta, idle_back, credit_extra, broken):
        order = np.argsort(src, kind="stable")
        self.src, self.dst, self.w = src[order], dst[order], w[order]
        self.row = np.searchsorted(self.src, np.arange(V + 1))
        self.V, self.ctas, self.per, self.delta = V, ctas, warps, delta
        self.idle_back, self.extra, self.broken, self.rng = idle_back, credit_extra, broken, rng
        self.dist = np.full(V, INF)
        self.dist[0] = 0.0
        self.dirty = np.zeros(V, bool)
        self.dirty[0] = True
        self.p, self.d = [1] + [0] * (SLOTS - 1), [0] * SLOTS
        self.pt = (0, delta)  # phase, threshold
        self.idle, self.mn, self.open = [0, 0], [INF, INF], 0
        self.cta = [[0, 0] for _ in range(ctas)]  # phase, idle warps
        self.posted = []  # operations on their way
        self.credit, self.holding = [0] * (ctas * warps), 0
        self.done, self.ended = False, None

    def post(self, op):
        ticket = {"done": False}
        self.posted.append((op, ticket))
        return ticket

    def perform(self, i):
        op, ticket = self.posted.pop(i)
        op()
        ticket["done"] = True

    def add(self, counter, slot, x):
        counter[slot] += x

    def relax(self, g, v, T, local):
        slot, e0, e1 = g % SLOTS, self.row[v], self.row[v + 1]
        yield
        du = self.dist[v]
        if self.credit[g] < e1 - e0:
            more = e1 - e0 - self.credit[g] + self.extra
            yield
            self.p[slot] += more
            self.credit[g] += more
        if self.broken:  # the credit goes back before its bits are set
            self.post(lambda c=self.credit[g]: self.add(self.d, slot, c))
            self.credit[g] = 0
        for e in range(e0, e1):
            x, nd = self.dst[e], du + self.w[e]
            yield
            if nd < self.dist[x]:
                self.dist[x] = nd
                yield
                if not self.dirty[x]:
                    self.dirty[x] = True
                    self.credit[g] -= 1
                    if nd < T:
                        local.append(x)
        self.credit[g] += 1
        self.holding -= 1

    def warp(self, g):
        slot, c = g % SLOTS, g // self.per
        reported, back = None, None
        while not self.done:
            yield
            ph, T = self.pt
            found, above, local = False, INF, []
            for v in range(g, self.V, self.ctas * self.per):
                yield
                if not self.dirty[v]:
                    continue
                if not self.dist[v] < T:
                    above = min(above, self.dist[v])
                    continue
                yield
                if not self.dirty[v]:
                    continue
                self.dirty[v] = False  # the claim
                self.holding += 1
                if self.idle_back and not found and reported == ph:
                    if self.cta[c][0] == ph and self.cta[c][1] > 0:
                        self.cta[c][1] -= 1
                        if self.cta[c][1] + 1 == self.per:
                            back = self.post(lambda q=ph & 1: self.add(self.idle, q, -1))
                    reported = None
                found = True
                yield from self.relax(g, v, T, local)
                while local:  # what this warp made dirty below T, claimed back
                    x = local.pop()
                    yield
                    if self.dirty[x]:
                        self.dirty[x] = False
                        self.holding += 1
                        yield from self.relax(g, x, T, local)
            if found:
                continue
            if self.credit[g]:
                self.post(lambda k=self.credit[g]: self.add(self.d, slot, k))
                self.credit[g] = 0
            if reported == ph or T == INF:
                continue
            yield
            self.mn[ph & 1] = min(self.mn[ph & 1], above)
            while back and not back["done"]:
                yield
            yield
            if self.cta[c][0] > ph:
                continue
            self.cta[c] = [ph, (self.cta[c][1] if self.cta[c][0] == ph else 0) + 1]
            reported = ph
            if self.cta[c][1] != self.per:
                continue
            yield
            self.idle[ph & 1] += 1
            if self.idle[ph & 1] != self.ctas:
                continue
            yield
            if self.open != ph:
                continue
            self.open = ph + 1
            yield
            m, self.mn[ph & 1] = self.mn[ph & 1], INF
            yield
            self.idle[(ph + 1) & 1] = 0
            yield
            self.pt = (ph + 1, max(T + self.delta, m + self.delta if m < INF else 0.0))

    def checker(self):
        while not self.done:
            d = p = 0
            for i in range(SLOTS):
                yield
                d += self.d[i]
            for i in range(SLOTS):
                yield
                p += self.p[i]
            if d == p:
                self.ended = (bool(self.dirty.any()), self.holding, sum(self.credit))
                self.done = True


def run(seed, idle_back, threshold=True, broken=False):
    rng = np.random.default_rng(seed)
    V = int(rng.integers(4, 20))
    E = int(rng.integers(V, 4 * V))
    src, dst, w = rng.integers(0, V, E), rng.integers(0, V, E), rng.integers(0, 9, E).astype(float)
    ctas, warps = int(rng.integers(1, 4)), int(rng.integers(1, 4))
    m = Machine(rng, V, src, dst, w, ctas, warps, float(rng.integers(1, 6)) if threshold else INF, idle_back,
                int(rng.integers(0, 6)), broken)
    gens = [m.warp(g) for g in range(ctas * warps)] + [m.checker()]
    live = list(range(len(gens)))
    steps = 0
    while live and not m.done and steps < 400000:
        steps += 1
        k = int(rng.integers(len(live) + min(len(m.posted), 2)))
        if k >= len(live):  # one on its way arrives, in any order
            m.perform(int(rng.integers(len(m.posted))))
            continue
        try:
            next(gens[live[k]])
        except StopIteration:
            live.pop(k)
    return m, bellman_ford(V, src, dst, w)


@pytest.mark.parametrize("idle_back", [True, False])
@pytest.mark.parametrize("seed", range(60))
def test_the_run_ends_with_nothing_left(seed, idle_back):
    m, want = run(seed, idle_back)
    assert m.done, "a phase that never opened, or sums that never met"
    assert m.ended == (False, 0, 0)
    np.testing.assert_array_equal(m.dist, want)


@pytest.mark.parametrize("seed", range(20))
def test_without_a_threshold(seed):
    m, want = run(1000 + seed, True, threshold=False)
    assert m.done and m.ended == (False, 0, 0)
    assert m.pt[0] == 0
    np.testing.assert_array_equal(m.dist, want)


def test_credit_given_back_too_early_is_caught():
    bad = 0
    for seed in range(300):
        m, want = run(seed, True, broken=True)
        if not m.done or m.ended[0] or m.ended[1] or not (m.dist == want).all():
            bad += 1
    assert bad > 0
