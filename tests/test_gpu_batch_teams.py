"""Level-by-level teams (graphgolf_b200/csrc/apsp_levels.cuh) whose graphs
follow one another without a barrier: several asymmetric ones in a row, and an
id out of range behind them."""
import numpy as np
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


def _asymmetric(n, d, seed):
    a = graphs.random_regular(n, d, seed).adj.copy()
    a[n // 2, 1] = (a[n // 2, 1] + 1) % n
    return a


# 20 graphs on teams of a few each: the first 14 in the teams' order of size are asymmetric
_ASYM = [(n, d) for n, d in zip(range(9000, 6200, -200), [4, 6, 8, 5, 12, 7, 6] * 2)]
_SYM = [(6001 - 200 * i + (i % 2) * (4 + i), 6) for i in range(6)]


def _mixed():
    out = [_asymmetric(n, d, n) for n, d in _ASYM]
    return out + [graphs.random_regular(n + n % 2, d, n).adj for n, d in _SYM]


def test_asymmetric_graphs_in_a_row(gpu):
    m = _mixed()
    want = [oracle.general(a) for a in m]
    with gg.Batch([a.shape[0] for a in m], [a.shape[1] for a in m]) as b:
        for _ in range(5):
            assert [_got(r) for r in b.evaluate(m)] == want


@pytest.mark.parametrize("i", [0, 5, 13, 16, 19])
def test_error_behind_asymmetric_graphs(gpu, i):
    """The error names the graph that has it, not one that was left to the windows."""
    m = _mixed()
    good = m[i]
    m[i] = good.copy()
    m[i][good.shape[0] // 3, 2] = good.shape[0]
    with gg.Batch([a.shape[0] for a in m], [a.shape[1] for a in m]) as b:
        for _ in range(2):
            with pytest.raises(gg.EvaluationError) as e:
                b.evaluate(m)
            assert e.value.code == -3 and f"graph {i}:" in str(e.value)
        m[i] = good
        assert _got(b.evaluate(m)[i]) == oracle.general(good)
