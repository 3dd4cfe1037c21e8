"""A batch evaluated from the host while a launch of it on another stream has
not been collected: the two share workspaces and control blocks."""
import pytest
import torch

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu

_SHAPES = [(500, 4, 1), (1024, 8, 1), (3000, 8, 1), (9000, 6, 1), (10000, 5, 1), (9216, 6, 4), (6001, 6, 1)]


def test_evaluate_behind_an_uncollected_launch(gpu):
    adjs = [[(graphs.symmetric_regular(n, d, g, n + s) if g > 1 else graphs.random_regular(n + n * d % 2, d, n + s)).adj
             for n, d, g in _SHAPES] for s in range(2)]
    want = [[oracle.general(a, groups=s[2]) for a, s in zip(set_, _SHAPES)] for set_ in adjs]
    stream = torch.cuda.Stream()
    with gg.Batch([a.shape[0] for a in adjs[0]], [s[1] for s in _SHAPES], [s[2] for s in _SHAPES]) as b:
        for i in range(6):
            b.launch(stream.cuda_stream)
            res = b.evaluate(adjs[i % 2])
            assert [(r.connected, r.diameter, r.aspl, r.total) for r in res] == want[i % 2]
        b.launch(stream.cuda_stream)
        res = b.collect(stream.cuda_stream)
        assert [(r.connected, r.diameter, r.aspl, r.total) for r in res] == want[1]
