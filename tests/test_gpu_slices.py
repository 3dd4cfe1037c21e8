"""Evaluation on shared-memory windows (graphgolf_b200/csrc/apsp_slice.cuh)
against the oracle, bit-exact, at the edges of its windows, row widths and
routes: window_bits 32 or 64 says that a slice kernel ran."""
import numpy as np
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs
from _cases import union_graph

pytestmark = pytest.mark.gpu


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


@pytest.mark.parametrize("n,d,g,ac,bits", [(2, 1, 1, 0, 32), (31, 4, 1, 0, 32), (32, 5, 1, 0, 32), (33, 4, 1, 0, 32),
                                           (1024, 3, 1, 0, 32), (1056, 8, 33, 0, 32), (610, 5, 2, 10, 32),
                                           (1000, 6, 1, 999, 32), (4736, 8, 1, 0, 32), (4738, 7, 1, 0, 64),
                                           (9400, 4, 1, 0, 64), (9472, 3, 1, 0, 64), (9474, 3, 1, 0, 0)])
def test_general(gpu, n, d, g, ac, bits):
    adj = graphs.random_regular(n, d, n + d).adj
    bn = (n - ac) // g
    r = gg.evaluate(adj, based_nodes=bn, groups=g, added_centers=ac)
    assert _got(r) == oracle.general(adj, based_nodes=bn, groups=g, added_centers=ac)
    assert r.window_bits == bits if bits else r.window_bits > 64


@pytest.mark.parametrize("n,d", [(500, 3), (3601, 4)])
def test_any_adjacency(gpu, n, d):
    """Rows need not be symmetric, simple or free of self entries (a directed
    cycle in the first column keeps the graph connected)."""
    adj = np.random.default_rng(n).integers(0, n, (n, d)).astype(np.int32)
    adj[:, 0] = (np.arange(n) + 1) % n
    assert _got(gg.evaluate(adj)) == oracle.general(adj)
    rh = np.arange(n, dtype=np.int32)
    assert _got(gg.evaluate_grid(adj, rh)) == oracle.grid(adj, rh)


@pytest.mark.parametrize("w,h,d,length,g,shuffle", [(2, 2, 2, 2, 1, False), (70, 50, 4, 3, 1, False),
                                                    (50, 70, 6, 3, 1, False), (64, 64, 4, 4, 2, False),
                                                    (60, 60, 4, 3, 4, False), (70, 61, 4, 3, 1, True),
                                                    (118, 122, 4, 9, 1, False), (120, 122, 4, 9, 1, False)])
def test_lattices(gpu, w, h, d, length, g, shuffle):
    """Rings on lattices of several shapes, with symmetry groups, with a
    numbering that hides the lattice, and past the largest that fits."""
    gr = graphs.grid_regular(w, h, d, length, w + h)
    adj, n = gr.adj, gr.nodes
    if shuffle:
        p = np.random.default_rng(1).permutation(n).astype(np.int32)
        out = np.empty_like(adj)
        out[p] = p[adj]
        adj = out
    rh = graphs.rotate_hash(n, h, w, g)
    r, want = gg.evaluate_grid(adj, rh, groups=g), oracle.grid(adj, rh, groups=g)
    assert (r.connected, r.diameter) == want[:2] and (not r.connected or (r.aspl, r.total) == want[2:])
    assert (r.window_bits == 32) == (n * 16 <= 231424)


def test_routes_in_turn(gpu):
    """Errors, stalls and other kernels between slices leave nothing behind."""
    big = graphs.random_regular(12000, 6, 1).adj
    small = graphs.random_regular(700, 5, 2).adj
    gr = graphs.grid_regular(70, 60, 4, 3, 3)
    two = union_graph(2100, 4, 4)
    want = [oracle.general(big), oracle.general(small), oracle.grid(gr.adj, gr.rotate_hash)]
    for _ in range(2):
        bad = gr.adj.copy()
        bad[4000, 1] = 4200
        with pytest.raises(gg.EvaluationError) as e:
            gg.evaluate_grid(bad, gr.rotate_hash)
        assert e.value.code == -3
        rh = gr.rotate_hash.copy()
        rh[17] = rh[18]
        with pytest.raises(gg.EvaluationError) as e:
            gg.evaluate_grid(gr.adj, rh)
        assert e.value.code == -5
        r = gg.evaluate_grid(two, np.arange(4200, dtype=np.int32))
        assert (r.connected, r.diameter) == (False, 4201)
        got = [_got(gg.evaluate(big)), _got(gg.evaluate(small)), _got(gg.evaluate_grid(gr.adj, gr.rotate_hash))]
        assert got == want
