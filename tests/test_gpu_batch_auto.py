"""Which kernels the automatic plan takes for batches of equal graphs, on both
sides of its lines (window_bits: 64 in shared memory, at least n level by level,
128 to 4096 on window teams), against the single-graph evaluator."""
import pytest

import graphgolf_b200 as gg
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


def _kind(r, n):
    return "levels" if r.window_bits >= n and r.window_bits > 4096 else "slices" if r.window_bits <= 64 else "windows"


def _run(n, d, k):
    adjs = [graphs.random_regular(n, d, s).adj for s in (1, 2)]
    want = [_got(gg.evaluate(a)) for a in adjs]
    with gg.Batch([n] * k, d) as b:
        res = b.evaluate([adjs[i % 2] for i in range(k)])
        assert [_got(r) for r in res] == [want[i % 2] for i in range(k)]
        kinds = {_kind(r, n) for r in res}
        assert len(kinds) == 1
        return kinds.pop(), b.plan


@pytest.mark.parametrize("n,d,k,kind", [(500, 8, 256, "slices"), (2000, 8, 8, "slices"), (2000, 8, 64, "windows"),
                                        (2000, 5, 64, "windows"), (1000, 16, 64, "windows"), (4000, 5, 32, "windows"),
                                        (4600, 5, 64, "slices"), (200, 12, 64, "slices"), (64, 2, 40, "slices")])
def test_small_graphs(gpu, n, d, k, kind):
    """Windows of 2048 and 4096 sources fit some sizes so well that teams beat
    one window a CTA."""
    assert _run(n, d, k)[0] == kind


@pytest.mark.parametrize("n,d,k,kind", [(7000, 4, 16, "windows"), (8000, 4, 16, "windows"), (10000, 4, 16, "windows"),
                                        (8600, 4, 16, "levels"), (11000, 4, 16, "levels"), (10000, 4, 4, "levels"),
                                        (6000, 6, 16, "levels"), (7000, 5, 16, "levels")])
def test_mid_size_graphs(gpu, n, d, k, kind):
    assert _run(n, d, k)[0] == kind


@pytest.mark.parametrize("n,k", [(10000, 32), (20000, 8)])
def test_window_teams_stay_near_l2(gpu, n, k):
    """The teams' matrices of graphs that only windows serve (degree 3)."""
    kind, (bits, _, teams) = _run(n, 3, k)
    assert kind == "windows" and teams * n * (12 + 32 * bits // 128) < 160e6
