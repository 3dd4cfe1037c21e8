"""The annealer's step kernels against a restatement of the step in Python:
proposal draws, acceptance and the applied swaps, move by move.

All quantities are integers (the acceptance of a worse graph compares exp() with
a 53-bit draw; a last-bit difference of exp() would have to fall on the draw), so
states are compared for equality."""
import math

import numpy as np
import pytest

import graphgolf_b200 as gg
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu
M = (1 << 64) - 1


def _mix(z):
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M
    return z ^ (z >> 31)


def _draw(seed, a, b, c):
    x = _mix((a + 0x9E3779B97F4A7C15) & M) ^ _mix((b * 0xD1B54A32D192ED03 + c + 1) & M)
    return _mix((seed + 0x9E3779B97F4A7C15 * x) & M)


def _below(h, n):
    return ((h & M) >> 32) * n >> 32


def _distances(n, d, edges):
    """(diameter, total over ordered pairs) by bit-parallel search; None if disconnected."""
    adj = graphs.create_adj(n, d, edges)
    rows = np.packbits(np.eye(n, dtype=bool), axis=1)
    reached, diam, total = n, 0, 0
    while reached < n * n:
        rows = rows | np.bitwise_or.reduce(rows[adj], axis=1)
        now = int(np.unpackbits(rows, axis=1, count=n).sum())
        if now == reached:
            return None
        diam += 1
        total += diam * (now - reached)
        reached = now
    return diam, total


class _Plain:
    def __init__(self, g, seed, temp, cooling, hill):
        self.n, self.d, self.seed = g.nodes, g.degree, seed
        self.edges = np.array(g.edges).reshape(-1, 2).copy()
        self.temp, self.cooling, self.hill = temp, cooling, hill
        self.cur = self.best = _distances(self.n, self.d, self.edges)
        self.best_edges = self.edges.copy()
        self.step = self.accepts = 0

    def propose(self):
        E = self.edges
        have = {frozenset(map(int, e)) for e in E}
        for attempt in range(64):
            h = _draw(self.seed, self.step, 0, attempt)
            i, j = _below(h, len(E)), _below((h << 32) & M, len(E))
            if i == j:
                continue
            a, b, c, e = int(E[i][0]), int(E[i][1]), int(E[j][0]), int(E[j][1])
            if _mix(h) & 1:
                c, e = e, c
            if a == c or b == e or frozenset((a, c)) in have or frozenset((b, e)) in have:
                continue
            return i, j, (a, c), (b, e)
        return None

    def run(self, steps):
        for _ in range(steps):
            mv, cand = self.propose(), None
            if mv:
                edges = self.edges.copy()
                edges[mv[0]], edges[mv[1]] = mv[2], mv[3]
                cand = _distances(self.n, self.d, edges)
            acc = False
            if cand and cand[0] <= self.cur[0]:
                acc = cand <= self.cur
                if not acc and not self.hill:
                    u = ((_draw(self.seed ^ 0x5BD1E995, self.step, 0xDEC1DE, 7) >> 11) + 1.0) / (2.0**53 + 2.0)
                    acc = math.exp((self.cur[1] - cand[1]) / self.temp) > u
            if acc:
                self.edges, self.cur = edges, cand
                self.accepts += 1
                if cand < self.best:
                    self.best, self.best_edges = cand, edges.copy()
            self.temp *= self.cooling
            self.step += 1


def _same(an, st, p):
    assert (st.step, st.accepts) == (p.step, p.accepts)
    assert (st.cur_diam, st.cur_total) == p.cur
    assert (st.best_diam, st.best_total) == p.best
    assert np.array_equal(np.array(an.edges()).reshape(-1, 2), p.edges)
    assert np.array_equal(np.array(an.edges(best=True)).reshape(-1, 2), p.best_edges)


# one window and several, odd sizes, odd degrees (the last entry of a row has no
# pair), 64-source windows, more lines than the two-launch step takes
@pytest.mark.parametrize("n,d,steps,hill", [(10, 3, 40, True), (65, 4, 60, False), (301, 4, 40, False),
                                            (512, 7, 30, True), (1024, 8, 20, False), (4200, 8, 4, True)])
def test_plain_steps(gpu, n, d, steps, hill):
    g = graphs.random_regular(n, d, n + 3 * d)
    temp = 40.0 if not hill else 0.0
    with gg.Annealer(g, seed=9) as an:
        an.schedule(temp, 0.99, hill)
        p = _Plain(g, 9, temp, 0.99, hill)
        for part in (1, steps // 2, steps - steps // 2 - 1):
            p.run(part)
            _same(an, an.run(part), p)
        ckpt = an.save()
        an.autotune()   # may change the plan: the same steps follow
        p.run(steps // 2)
        st = an.run(steps // 2)
        _same(an, st, p)
    with gg.Annealer(gg.checkpoint_graph(ckpt), seed=9) as an:
        an.restore(ckpt)
        assert an.run(steps // 2) == st


def test_target_stops_the_plain_steps(gpu):
    g = graphs.random_regular(128, 5, 4)
    p = _Plain(g, 2, 0.0, 1.0, True)
    gains = 0
    while gains < 5:   # stop where the state is first reached
        before = p.cur
        p.run(1)
        gains += p.cur < before
    with gg.Annealer(g, seed=2) as an:
        an.target(*p.cur)
        st = an.run(p.step + 50)
        _same(an, st, p)
        _same(an, an.run(3), p)


def test_candidates_patched_in_place(gpu):
    """Several candidates without the delta evaluation (degree > 32), small graphs."""
    g = graphs.random_regular(220, 34, 8)
    with gg.Annealer(g, candidates=4, compose=4, seed=5) as an:
        for _ in range(3):
            st = an.run(6)
            assert not st.delta
            assert _distances(220, 34, np.array(an.edges()).reshape(-1, 2)) == (st.cur_diam, st.cur_total)


# proposals that fill the ranking's power of two and that do not
@pytest.mark.parametrize("K,G", [(16, 32), (16, 48), (32, 256), (64, 1008)])
def test_ranking(gpu, K, G):
    g = graphs.random_regular(700, 6, 21)
    with gg.Annealer(g, candidates=K, proposals=G, compose=4, seed=4) as an:
        for _ in range(4):
            st = an.run(2)
            predicted, _ = an.last_step()
            top = K - max(1, K // 4)
            assert np.all(np.diff(predicted[:top]) >= 0)
            assert np.all(predicted[top:] >= predicted[top - 1])
            assert _distances(700, 6, np.array(an.edges()).reshape(-1, 2)) == (st.cur_diam, st.cur_total)
