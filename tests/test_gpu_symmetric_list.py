"""Half sweeps (graphgolf_b200/csrc/apsp_sym.cuh) of a graph whose unreached
pairs at the listing level number just over 2^32: a 32-bit counter of them
wraps round to a number that looks like a list that fits."""
import numpy as np
import pytest

import graphgolf_b200 as gg
from graphgolf_b200 import graphs

CORE, DEGREE, LEAVES, FEWER, ROW, LIST = 9728, 18, 13, 3192, 32, 1 << 22


def _core_levels(adj, leaves, top):
    """For k = 0 .. top, over the ordered pairs (u, v) of the core at a distance
    above k: their number, the sum of leaves[v], and that of leaves[u] * leaves[v]."""
    n = adj.shape[0]
    row = np.zeros((n, n // 64), dtype=np.uint64)
    i = np.arange(n)
    row[i, i // 64] = np.uint64(1) << (i % 64).astype(np.uint64)
    out = []
    for k in range(top + 1):
        a = b = c = 0
        for u in range(0, n, 2048):
            far = np.unpackbits(row[u:u + 2048].view(np.uint8), axis=1, bitorder="little") == 0
            a += int(np.count_nonzero(far))
            hit = far.astype(np.float32) @ leaves.astype(np.float32)    # at most 13 n: exact
            b += int(hit.astype(np.int64).sum())
            c += int((hit.astype(np.int64) * leaves[u:u + 2048]).sum())
        out.append((a, b, c))
        if k < top:
            new = row.copy()
            for j in range(adj.shape[1]):
                new |= row[adj[:, j]]
            row = new
    return out


def _unreached(lv, n, edges, k):
    """Ordered pairs of the whole graph at a distance above k."""
    if k < 2:
        return n * n - n - 2 * edges * k
    return lv[k][0] + 2 * lv[k - 1][1] + lv[k - 2][2]


def _graph():
    """A random core, 13 leaves to a vertex less one for the first FEWER of
    them: the rows, and the ordered pairs at a distance above k = 0, 1, ..."""
    core = graphs.random_regular(CORE, DEGREE, 5).adj
    leaves = np.full(CORE, LEAVES, dtype=np.int64)
    leaves[:FEWER] -= 1
    n = CORE + int(leaves.sum())
    adj = np.repeat(np.arange(n, dtype=np.int32)[:, None], ROW, axis=1)
    adj[:CORE, :DEGREE] = core
    owner = np.repeat(np.arange(CORE), leaves)
    slot = np.concatenate([np.arange(x) for x in leaves])
    leaf = CORE + np.arange(n - CORE)
    adj[owner, DEGREE + slot] = leaf
    adj[leaf, 0] = owner
    lv = _core_levels(core, leaves, 7)
    un = [_unreached(lv, n, CORE * DEGREE // 2 + n - CORE, k) for k in range(8)]
    # level 5 is the one at which the pairs are listed
    assert 1 << 32 <= un[5] // 2 < (1 << 32) + LIST and un[7] == 0
    return adj, un


@pytest.mark.gpu
def test_more_than_2_32_unreached_pairs(gpu):
    adj, un = _graph()
    r = gg.evaluate(adj)
    assert (r.connected, r.diameter, r.total) == (True, un.index(0), sum(un))
