"""ggb_kernel_launches counts every kernel of a batch evaluation and of an
annealing step."""
import pytest

import graphgolf_b200 as gg
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu

# (nodes, degree, groups), kernels of one evaluation: shared-memory windows in
# one launch per size class, level by level with the windows behind it, window teams
_CASES = [([(1024, 8, 1)], 1), ([(9000, 6, 1)], 2), ([(9216, 6, 4)], 1), ([(1024, 8, 1), (9000, 6, 1)], 3),
          ([(1024, 8, 1), (9000, 6, 1), (9216, 6, 4)], 4),
          ([(500, 4, 1), (2400, 11, 1), (4200, 6, 1), (9000, 6, 1), (9216, 6, 4)], 6)]


def _adj(n, d, g):
    return (graphs.symmetric_regular(n, d, g, n) if g > 1 else graphs.random_regular(n, d, n)).adj


@pytest.mark.parametrize("shapes,kernels", _CASES)
def test_batch(gpu, shapes, kernels):
    adjs = [_adj(*s) for s in shapes]
    with gg.Batch([s[0] for s in shapes], [s[1] for s in shapes], [s[2] for s in shapes]) as b:
        b.upload(adjs)
        for plan, want in (((0, 0), kernels), ((1024, 8), 1), ((0, 0), kernels)):
            b.set_plan(*plan)
            before = gg.kernel_launches()
            b.launch()
            b.collect()
            assert gg.kernel_launches() - before == want
            before = gg.kernel_launches()
            b.evaluate(adjs)
            uploads = gg.kernel_launches() - before - want   # the widening of 16-bit ids, once per part
            assert 1 <= uploads <= (3 if want > 1 else 1)


def test_captured_step(gpu):
    """The plain step: the batch's kernel and one more."""
    with gg.Annealer(graphs.random_regular(1024, 8, 1), seed=1) as an:
        before = gg.kernel_launches()
        an.run(1)
        assert gg.kernel_launches() - before == 1 + 2     # the first proposal, the step
