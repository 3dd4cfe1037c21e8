"""The annealing step that reaches the target: every move of the accepted
composite is applied, also by the warps that come late to the decision."""
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,K,G,comp", [(2048, 8, 256, 256, 256), (1024, 6, 128, 128, 128), (4096, 10, 64, 1024, 64)])
def test_last_step_applies_a_whole_composite(gpu, n, d, K, G, comp):
    largest = 0
    for seed in range(1, 9):
        g = graphs.random_regular(n, d, seed)

        def make():
            an = gg.Annealer(g, candidates=K, proposals=G, compose=comp, seed=seed)
            if G > K:
                an.predicted(2, 256)
            return an

        with make() as an:
            first = an.run(1)
        with make() as an:
            start = an.run(0)
            if (first.cur_diam, first.cur_total) >= (start.cur_diam, start.cur_total):
                continue
            an.target(first.cur_diam, first.cur_total)
            st = an.run(3)
            assert st.done and st.step == 1 and st.moved_swaps == first.moved_swaps
            largest = max(largest, st.moved_swaps)
            for best in (False, True):
                edges = an.edges(best=best)
                adj = graphs.create_adj(n, d, edges)
                assert graphs.verify(graphs.Graph(n, d, edges, adj)) == 0
                assert oracle.general(adj)[1::2] == (st.cur_diam, st.cur_total)
    assert largest > 32
