"""Which graphs just past 8192 vertices are evaluated level by level over all
sources (one window of at least n) and which as windows, on both sides of
every line, against the oracle."""
import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,levels", [(8900, 5, True), (8902, 5, False), (11472, 5, False), (11474, 5, True),
                                        (12300, 6, True), (12302, 6, False), (15002, 5, True), (8598, 7, False),
                                        (8600, 7, True), (8200, 6, True)])
def test_regular(gpu, n, d, levels):
    adj = graphs.random_regular(n, d, n).adj
    r = gg.evaluate(adj)
    assert (r.connected, r.diameter, r.aspl, r.total) == oracle.general(adj)
    assert (r.window_bits >= n) == levels


@pytest.mark.parametrize("n,d,levels", [(8200, 5, False), (9000, 5, False), (11472, 5, False), (11474, 5, True),
                                        (10144, 6, False), (10146, 6, True), (12290, 6, False), (15002, 6, True),
                                        (9000, 8, True)])
def test_nonregular(gpu, n, d, levels):
    _, adj, deg = graphs.nonregular(graphs.random_regular(n, d, n), n // 20, 1)
    r = gg.evaluate_nonregular(adj, deg)
    assert (r.connected, r.diameter, r.aspl, r.total) == oracle.general_nr(adj, deg)
    assert (r.window_bits >= n) == levels
