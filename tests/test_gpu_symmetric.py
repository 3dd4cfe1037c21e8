"""Symmetric graphs past 8192 vertices (graphgolf_b200/csrc/apsp_levels.cuh and
apsp_sym.cuh) against the oracle, bit-exact: whole and partial last windows, both vector
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


@pytest.mark.parametrize("n,d,bits", [(8194, 5, 8448), (8448, 8, 8448), (9001, 6, 9216), (12288, 12, 12288),
                                      (12290, 4, 12544), (16386, 7, 16640), (9000, 32, 9216), (21999, 16, 22016),
                                      (18002, 7, 8192), (20002, 4, 8192), (22001, 16, 8192), (24576, 9, 8192),
                                      (24580, 8, 8192), (24576, 24, 8192)])
def test_random_graphs(gpu, n, d, bits):
    """Level by level over all sources (one window of at least n), and half
    sweeps of windows of 8192."""
    adj = graphs.random_regular(n, d, n + d).adj
    r = gg.evaluate(adj)
    assert _got(r) == oracle.general(adj)
    assert r.window_bits == bits


def _multi_edges(n):
    """Repeated entries and self entries, symmetric."""
    a = graphs.random_regular(n, 6, 1).adj
    return np.concatenate([a, a[:, :2], np.arange(n, dtype=np.int32)[:, None]], axis=1)


def _unmatched(n):
    """One row's entry does not hold the row in return."""
    a = graphs.random_regular(n + 2, 6, 2).adj.copy()
    a[7000, 3] = (a[7000, 3] + 1) % (n + 2)
    return a


def _circulant(n):
    """More levels than any random graph has."""
    v = np.arange(n, dtype=np.int32)[:, None]
    return (v + np.array([1, -1, 40, -40, 1700, -1700], dtype=np.int32)) % n


def _tail(n):
    """A random core whose every vertex carries a leaf: the first window is
    reached early, the leaves among themselves are not (a list too long)."""
    n = n * 2 // 3
    core = graphs.random_regular(n, 6, 3).adj
    adj = np.empty((2 * n, 7), dtype=np.int32)
    i = np.arange(n, dtype=np.int32)
    adj[:n, :6], adj[:n, 6] = core, i + n
    adj[n:] = (i + n)[:, None]
    adj[n:, 0] = i
    return adj


@pytest.mark.parametrize("n", [12000, 20400])
@pytest.mark.parametrize("make", [_multi_edges, _unmatched, _circulant, _tail])
def test_other_adjacencies(gpu, make, n):
    adj = np.ascontiguousarray(make(n), dtype=np.int32)
    assert _got(gg.evaluate(adj)) == oracle.general(adj)


@pytest.mark.parametrize("n", [12000, 24000])
def test_stalls_and_errors(gpu, n):
    """Two components, a component too small to show in the first window's
    counts, an entry out of range; then a good graph again."""
    r = gg.evaluate(union_graph(n // 2, 6, 5))
    assert (r.connected, r.diameter) == (False, 2**31 - 1)
    a = graphs.random_regular(n, 6, 6).adj
    k4 = np.array([[j for j in range(4) if j != i] * 2 for i in range(4)], dtype=np.int32) + n
    r = gg.evaluate(np.concatenate([a, k4]))
    assert (r.connected, r.diameter) == (False, 2**31 - 1)
    bad = a.copy()
    bad[n - 1, 5] = n
    with pytest.raises(gg.EvaluationError) as e:
        gg.evaluate(bad)
    assert e.value.code == -3
    assert _got(gg.evaluate(a)) == oracle.general(a)


def test_nonregular(gpu):
    _, adj, deg = graphs.nonregular(graphs.random_regular(14000, 7, 8), 3000, 9)
    r = gg.evaluate_nonregular(adj, deg)
    assert _got(r) == oracle.general_nr(adj, deg)
