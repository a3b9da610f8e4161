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


def test_one_graph_with_repeated_entries_leaves_the_others_where_they_are():
    # a row longer than n is left to the unions; the others' results are those
    # of a call without that graph, bit for bit
    graphs = [G.barabasi_albert(n, 3, seed=n) for n in (5000, 1200, 60)]
    odd = lgbc.SimpleGraph.from_csr([0, 4, 7, 8], [1, 1, 1, 1, 0, 0, 2, 1])
    want = lgbc.betweenness_centrality_many(graphs)
    got = lgbc.betweenness_centrality_many([graphs[0], odd, graphs[1], odd, graphs[2]])
    assert same([got[0], got[2], got[4]], want)
    alone = lgbc.betweenness_centrality_many([odd])[0]
    assert same([got[1], got[3]], [alone, alone])
