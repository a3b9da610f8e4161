"""The same call on the same graphs gives the same bits: no sum depends on the
order in which blocks or atomics come."""
import numpy as np
import pytest

import lgbc
from lgbc import generators as G

pytestmark = pytest.mark.gpu


def same(a, b):
    return all(np.array_equal(np.asarray(x).view(np.uint64), np.asarray(y).view(np.uint64)) for x, y in zip(a, b))


@pytest.mark.parametrize("endpoints", [False, True])
def test_many_graphs_repeat_bit_for_bit(endpoints):
    graphs = [G.barabasi_albert(n, 3, seed=n) for n in (40, 700, 3000, 5000, 9000, 12500)]
    graphs += [G.rmat(11, 16, seed=1), G.erdos_renyi_nm(6000, 20000, seed=2)]  # warp-walked rows, ragged ends
    want = lgbc.betweenness_centrality_many(graphs, endpoints=endpoints)
    for _ in range(3):
        assert same(lgbc.betweenness_centrality_many(graphs, endpoints=endpoints), want)


@pytest.mark.parametrize("directed", [False, True])
def test_handles_of_one_graph_agree_bit_for_bit(directed):
    g = G.rmat(11, 16, seed=3, directed=directed)
    src = np.random.default_rng(1).choice(g.nv(), 900, replace=False) + 1
    build = lgbc.SimpleDiGraph if directed else lgbc.SimpleGraph
    want = None
    for _ in range(4):
        h = build.from_csr(*g.csr(), *(g.in_csr() if directed else ()))
        got = lgbc.betweenness_centrality(h, src)
        assert want is None or same([got], [want])
        want = got
