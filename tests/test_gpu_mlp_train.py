"""The training step's two kernels at the edges of their tiles (16 rows a CTA,
at most 256) against the network's oracle, and Adam against its formula.

Tolerances: gradients as in test_gpu_mlp.py (2 % in relative L2 norm per block:
BF16 rounding boundaries).  One Adam step is a handful of FP32 operations, each
within 2^-24 relative, and two powf and one sqrtf within a few units in the last
place; three steps stay within 1e-5 of the parameter's change plus one FP32
rounding of the parameter (at most 2^-23 of it) per step."""
import numpy as np
import pytest

import graphgolf_b200 as gg
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu

BLOCKS = [(mo.OFF_W1, mo.OFF_B1), (mo.OFF_B1, mo.OFF_W2), (mo.OFF_W2, mo.OFF_B2), (mo.OFF_B2, mo.OFF_W3),
          (mo.OFF_W3, mo.OFF_B3), (mo.OFF_B3, mo.N_PARAMS)]


def _data(rows):
    rng = np.random.default_rng(rows)
    return (mo.init(rows), rng.uniform(-1, 1, (rows, 32)).astype(np.float32),
            rng.uniform(-2, 2, rows).astype(np.float32))


@pytest.mark.parametrize("rows", [16, 32, 48, 240, 256])
def test_gradients(gpu, rows):
    p, x, t = _data(rows)
    net = gg.FilterNet(rows)
    net.params = p
    loss, g = net.grads(x, t)
    loss_ref, g_ref = mo.grads(p, x, t)
    net.close()
    assert abs(loss - loss_ref) <= 0.02 * loss_ref
    for a, b in BLOCKS:
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) < 0.02 * (np.linalg.norm(g_ref[a:b]) + 1e-12), (a, b)


@pytest.mark.parametrize("rows", [16, 256])
def test_adam_steps(gpu, rows):
    """Three steps equal Adam in float64 on the gradients the kernels report
    (read from a second network that holds the same parameters)."""
    p, x, t = _data(rows)
    net, probe = gg.FilterNet(rows), gg.FilterNet(rows)
    net.params = p
    m1, m2 = np.zeros(mo.N_PARAMS), np.zeros(mo.N_PARAMS)
    for k in range(1, 4):
        before = net.params
        probe.params = before
        g = probe.grads(x, t)[1].astype(np.float64)
        net.train(x, t, 1)
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        want = -1e-3 * (m1 / (1 - 0.9 ** k)) / (np.sqrt(m2 / (1 - 0.999 ** k)) + 1e-8)
        got = net.params.astype(np.float64) - before
        assert np.all(np.abs(got - want) <= 1e-5 * np.abs(want) + 2.0 ** -23 * np.abs(before) + 1e-9)
    net.close()
    probe.close()
