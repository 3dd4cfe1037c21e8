"""Grid evaluations whose edges are long against the lattice: the windows in
shared memory (window_bits 32) push thick rings then, and another kernel
serves the graph."""
import numpy as np
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,d,length,rings", [(100, 100, 4, 3, True), (128, 112, 8, 5, True), (80, 80, 6, 5, True),
                                                (64, 100, 6, 6, True), (100, 100, 8, 60, False),
                                                (120, 120, 6, 25, False), (120, 100, 12, 40, False),
                                                (80, 80, 12, 60, False), (60, 60, 12, 60, True)])
@pytest.mark.parametrize("g", [1, 2])
def test_long_edges(gpu, w, h, d, length, rings, g):
    gr = graphs.grid_regular(w, h, d, length, w + length)
    rh = graphs.rotate_hash(gr.nodes, h, w, g)
    r, want = gg.evaluate_grid(gr.adj, rh, groups=g), oracle.grid(gr.adj, rh, groups=g)
    assert (r.connected, r.diameter, r.aspl, r.total) == want
    assert (r.window_bits == 32) == rings


@pytest.mark.parametrize("length", [3, 60])
def test_errors_on_both_routes(gpu, length):
    gr = graphs.grid_regular(100, 100, 6, length, 1)
    n = gr.nodes
    for row in (0, 1, n // 2, n - 1):     # sampled rows and others
        for bad in (n, -1, 70000):
            adj = gr.adj.copy()
            adj[row, 0] = bad
            with pytest.raises(gg.EvaluationError) as e:
                gg.evaluate_grid(adj, gr.rotate_hash)
            assert e.value.code == -3
            rh = gr.rotate_hash.copy()
            rh[row] = bad
            with pytest.raises(gg.EvaluationError) as e:
                gg.evaluate_grid(gr.adj, rh)
            assert e.value.code == -5
    deg = np.full(n, 6, dtype=np.int32)
    deg[5] = 0
    r, want = gg.evaluate_grid_nonregular(gr.adj, deg, gr.rotate_hash), oracle.grid_nr(gr.adj, deg, gr.rotate_hash)
    assert (r.connected, r.diameter) == want[:2] and (not r.connected or (r.aspl, r.total) == want[2:])
