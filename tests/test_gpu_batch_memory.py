"""Plans whose workspace does not fit the device: the automatic plan falls back
to window teams, and a plan that could not be had launches nothing."""
import pytest
import torch

import graphgolf_b200 as gg
from graphgolf_b200 import graphs

pytestmark = pytest.mark.gpu


def _got(r):
    return (r.connected, r.diameter, r.aspl, r.total)


def _leave(mib):
    """A tensor that leaves about `mib` MiB of the device free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - (mib << 20), dtype=torch.uint8, device="cuda")


def test_level_by_level_workspace_does_not_fit(gpu):
    adjs = [graphs.random_regular(n, 16, n).adj for n in (21800, 21900, 1000)]
    want = [_got(gg.evaluate(a)) for a in adjs]
    hog = _leave(150)        # a level-by-level team of 21 900 vertices takes 115 MiB, a window team 22
    try:
        with gg.Batch([a.shape[0] for a in adjs], 16) as b:
            res = b.evaluate(adjs)
            assert [_got(r) for r in res] == want
            assert len({r.window_bits for r in res}) == 1      # one windows plan
    finally:
        del hog
        torch.cuda.empty_cache()


def test_plan_that_does_not_fit_launches_nothing(gpu):
    n, k = 30000, 64
    adj = graphs.random_regular(n, 4, 1).adj
    want = _got(gg.evaluate(adj))
    with gg.Batch([n] * k, 4) as b:
        assert {_got(r) for r in b.evaluate([adj] * k)} == {want}
        hog = _leave(200)
        try:
            with pytest.raises(gg.EvaluationError) as e:
                b.set_plan(4096, 1)                            # 64 teams of 29 MiB
            assert e.value.code == -6          # GGB_ENOMEM
            before = gg.kernel_launches()
            b.launch()
            with pytest.raises(gg.EvaluationError) as e:
                b.collect()
            assert "not evaluated" in str(e.value) and gg.kernel_launches() == before
        finally:
            del hog
            torch.cuda.empty_cache()
        b.set_plan()
        assert {_got(r) for r in b.evaluate([adj] * k)} == {want}
