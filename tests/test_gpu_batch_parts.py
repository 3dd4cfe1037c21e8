"""evaluate() sends a batch kernel by kernel, each launch beside the next one's
upload: the same answers as upload, launch and collect, whatever the order of
the graphs, and errors of every part leave the batch usable."""
import random

import pytest

import graphgolf_b200 as gg
import oracle
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu

# shared-memory windows, window teams (small ones of groups > 1 or degree 3
# among them), level by level; N * d odd and even
SHAPES = [(40, 3), (511, 6), (1500, 9), (2048, 12), (3000, 11), (4100, 12), (9001, 4), (10, 4), (4501, 8),
          (5003, 6), (6002, 5), (6500, 16), (7100, 4), (8000, 12), (5200, 7), (4900, 6), (5600, 9), (9500, 3)]


def _graphs(seed):
    return [graphs.random_regular(n, d, n + seed).adj for n, d in SHAPES]


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


@pytest.mark.parametrize("order", ["up", "down", "mixed"])
def test_parts_match_one_launch(gpu, order):
    perm = sorted(range(len(SHAPES)), key=lambda i: SHAPES[i][0])
    if order == "down":
        perm.reverse()
    if order == "mixed":
        random.Random(5).shuffle(perm)
    first, second = ([gs[i] for i in perm] for gs in (_graphs(0), _graphs(1)))
    with gg.Batch([a.shape[0] for a in first], [a.shape[1] for a in first]) as b:
        for adjs in (first, second, first):
            got = [_got(r) for r in b.evaluate(adjs)]
            assert b.kernel_ms() > 0
            b.upload(adjs)
            b.launch()
            assert [_got(r) for r in b.collect()] == got
            if adjs is second:
                assert got == [oracle.general(a) for a in adjs]


@pytest.mark.parametrize("n", [511, 9001, 6002])
@pytest.mark.parametrize("value", [-1, 70000])
def test_ids_that_do_not_fit(gpu, n, value):
    """Ids outside 16 bits: the part is sent again as ints, and refused."""
    adjs = _graphs(0)
    i = [s[0] for s in SHAPES].index(n)
    bad = [a.copy() for a in adjs]
    bad[i][n // 2, 1] = value
    with gg.Batch([a.shape[0] for a in adjs], [a.shape[1] for a in adjs]) as b:
        good = [_got(r) for r in b.evaluate(adjs)]
        with pytest.raises(gg.EvaluationError) as e:
            b.evaluate(bad)
        assert e.value.code == -3 and f"graph {i}:" in str(e.value)
        assert [_got(r) for r in b.evaluate(adjs)] == good
        assert good[i] == oracle.general(adjs[i])
