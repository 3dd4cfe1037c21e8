"""Half sweeps of large symmetric graphs (graphgolf_b200/csrc/apsp_sym.cuh)
against the oracle, bit-exact: whole and partial last windows, both vector
widths, few and many levels, and every way back to the persistent kernel."""
import numpy as np
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs
from _cases import union_graph

pytestmark = pytest.mark.gpu


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


@pytest.mark.parametrize("n,d", [(11000, 12), (11001, 6), (16384, 8), (16386, 7), (16640, 12), (20002, 4), (20001, 16),
                                 (24580, 9), (24576, 24)])
def test_random_graphs(gpu, n, d):
    adj = graphs.random_regular(n, d, n + d).adj
    r = gg.evaluate(adj)
    assert _got(r) == oracle.general(adj)
    assert r.window_bits == 8192


def _multi_edges():
    """Repeated entries and self entries, symmetric."""
    a = graphs.random_regular(12000, 5, 1).adj
    return np.concatenate([a, a[:, :2], np.arange(12000, dtype=np.int32)[:, None]], axis=1)


def _unmatched():
    """One row's entry does not hold the row in return."""
    a = graphs.random_regular(12002, 6, 2).adj.copy()
    a[7000, 3] = (a[7000, 3] + 1) % 12002
    return a


def _circulant():
    """More levels than any random graph has."""
    v = np.arange(12000, dtype=np.int32)[:, None]
    return (v + np.array([1, -1, 40, -40, 1700, -1700], dtype=np.int32)) % 12000


def _tail():
    """A random core whose every vertex carries a leaf: the first window is
    reached early, the leaves among themselves are not (a list too long)."""
    n = 8192
    core = graphs.random_regular(n, 6, 3).adj
    adj = np.empty((2 * n, 7), dtype=np.int32)
    i = np.arange(n, dtype=np.int32)
    adj[:n, :6], adj[:n, 6] = core, i + n
    adj[n:] = (i + n)[:, None]
    adj[n:, 0] = i
    return adj


@pytest.mark.parametrize("make", [_multi_edges, _unmatched, _circulant, _tail])
def test_other_adjacencies(gpu, make):
    adj = np.ascontiguousarray(make(), dtype=np.int32)
    assert _got(gg.evaluate(adj)) == oracle.general(adj)


def test_stalls_and_errors(gpu):
    """Two components, a component too small to show in the first window's
    counts, an entry out of range; then a good graph again."""
    r = gg.evaluate(union_graph(6000, 6, 5))
    assert (r.connected, r.diameter) == (False, 2**31 - 1)
    a = graphs.random_regular(12000, 6, 6).adj
    k4 = np.array([[j for j in range(4) if j != i] * 2 for i in range(4)], dtype=np.int32) + 12000
    r = gg.evaluate(np.concatenate([a, k4]))
    assert (r.connected, r.diameter) == (False, 2**31 - 1)
    bad = a.copy()
    bad[11999, 5] = 12000
    with pytest.raises(gg.EvaluationError) as e:
        gg.evaluate(bad)
    assert e.value.code == -3
    assert _got(gg.evaluate(a)) == oracle.general(a)


def test_nonregular(gpu):
    _, adj, deg = graphs.nonregular(graphs.random_regular(14000, 7, 8), 3000, 9)
    r = gg.evaluate_nonregular(adj, deg)
    assert _got(r) == oracle.general_nr(adj, deg)
