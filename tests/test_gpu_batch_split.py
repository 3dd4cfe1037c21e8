"""The automatic plan of a batch: shared-memory windows, level-by-level teams
and window teams in one batch, against the oracle, with the graphs that the
level-by-level kernel leaves to the windows, and errors in every part."""
import numpy as np
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs
from _cases import union_graph

pytestmark = pytest.mark.gpu


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


def _asymmetric(n, d, seed):
    a = graphs.random_regular(n, d, seed).adj.copy()
    a[n // 2, 1] = (a[n // 2, 1] + 1) % n
    return a


def _mix():
    out = [(graphs.random_regular(n, d, n).adj, 1) for n, d in
           [(33, 4), (700, 5), (1024, 8), (2000, 14), (3000, 9), (2800, 11), (4400, 12), (4502, 7), (4608, 12),
            (5001, 6), (6000, 16), (7000, 5), (8192, 12), (9000, 8)]]
    out += [(graphs.symmetric_regular(2048, 8, 16, 1).adj, 16), (graphs.symmetric_regular(9216, 6, 4, 2).adj, 4),
            (_asymmetric(6002, 6, 3), 1), (_asymmetric(1500, 6, 4), 1)]
    return out


def _batch(m):
    return gg.Batch([a.shape[0] for a, _ in m], [a.shape[1] for a, _ in m], [g for _, g in m])


def test_every_part_matches_oracle(gpu):
    m = _mix()
    want = [oracle.general(a, groups=g) for a, g in m]
    # a disconnected graph per part: the reference's answer without its N levels
    for n in (600, 6000):
        m.append((union_graph(n // 2, 6, n), 1))
        want.append((False, 2**31 - 1, np.finfo(np.float64).max, 0))
    with _batch(m) as b:
        for _ in range(2):
            res = b.evaluate([a for a, _ in m])
            assert [_got(r) for r in res] == want
        bits = [r.window_bits for r in res]
        assert bits[0] == 64 and bits[7] == 4608 and bits[13] == 9216 and bits[15] % 128 == 0
        b.set_plan(4096, 8)
        assert [_got(r) for r in b.evaluate([a for a, _ in m])] == want
        b.set_plan()
        assert [_got(r) for r in b.evaluate([a for a, _ in m])] == want


@pytest.mark.parametrize("n", [700, 4400, 9000])
def test_errors_in_every_part(gpu, n):
    m = _mix()
    i = [a.shape[0] for a, _ in m].index(n)
    with _batch(m) as b:
        bad = [a for a, _ in m]
        bad[i] = bad[i].copy()
        bad[i][n - 1, 2] = n
        with pytest.raises(gg.EvaluationError) as e:
            b.evaluate(bad)
        assert e.value.code == -3 and f"graph {i}:" in str(e.value)
        res = b.evaluate([a for a, _ in m])
        assert _got(res[i]) == oracle.general(m[i][0])


@pytest.mark.parametrize("n,d,bits", [(1024, 8, 32), (9000, 6, 9216), (6000, 8, 4096)])
def test_one_graph(gpu, n, d, bits):
    """A batch of one takes the single graph's lines (one step of an annealer)."""
    a = graphs.random_regular(n, d, 5).adj
    with gg.Batch([n], d) as b:
        r = b.evaluate([a])[0]
        assert _got(r) == oracle.general(a) and r.window_bits == bits
