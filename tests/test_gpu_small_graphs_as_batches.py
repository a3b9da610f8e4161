"""The batch paths on graphs that the shared-memory kernels take by default: a
direction threshold next to the default one (alpha 13 for 14) keeps the handle on
batches, so that the option under test is what differs, and the level counts of
the statistics, which the shared-memory kernels leave at zero, say that it did."""
import numpy as np
import pytest

import lgbc
import lgbc.generators as gen
from conftest import csr_args
from lgbc.learned import betweenness_raw_weighted
from oracle import oracle
from test_gpu_bfs_bins import GRAPHS as BFS_GRAPHS
from test_gpu_parity import assert_bc_close, oracle_bc

pytestmark = pytest.mark.gpu


def graph(kind):
    if kind == "rmat":
        return gen.rmat(13, 16, seed=5)
    if kind == "rmat_dir":
        return gen.rmat(13, 8, seed=6, directed=True)
    if kind == "ba":
        return gen.barabasi_albert(4000, 3, seed=7)
    e = np.random.default_rng(11).integers(0, 3000, (2, 2500))
    return lgbc.SimpleGraph.from_edge_arrays(3000, e[0], e[1])


def batches(g, **tuning):
    h = g.device_handle()
    h.set_tuning(alpha=13.0, **tuning)
    return h


@pytest.mark.parametrize("kind", ["rmat", "rmat_dir", "ba", "sparse"])
def test_level_loops(kind):
    g = graph(kind)
    src = np.random.default_rng(11).choice(g.nv(), 300, replace=False)
    want = oracle_bc(g, src, endpoints=True)
    levels = []
    for loop in (0, 1):
        h = batches(g, graph_loop=loop)
        assert_bc_close(lgbc.betweenness_centrality(g, src + 1, endpoints=True), want)
        levels.append(h.stats()["levels"])
    assert levels[0] > 0 and levels[1] > 0


@pytest.mark.parametrize("kind", ["rmat", "rmat_dir", "ba", "sparse"])
def test_distances_in_level_loops(kind):
    g = graph(kind)
    rp, ci, kw = csr_args(g)
    src = np.random.default_rng(12).choice(g.nv(), 70, replace=False).astype(np.int32)
    want = oracle.gdistances_many(rp, ci, src, nthreads=8).astype(np.int64)
    far = want == oracle.UNREACHED32
    for loop in (0, 1):
        h = batches(g, graph_loop=loop)
        got = lgbc.multi_gdistances(g, src + 1)
        assert np.array_equal(got, np.where(far, np.iinfo(g.eltype).max, want))
        assert h.stats()["batches"] == 2 and h.stats()["levels"] > 0
        reached, dsum, dmax = lgbc.distance.distance_stats(g, src)
        assert h.stats()["levels"] > 0
        assert np.array_equal(reached, (~far).sum(1))
        assert np.array_equal(dsum, np.where(far, 0, want).sum(1))
        assert np.array_equal(dmax, np.where(far, 0, want).max(1))
    assert np.array_equal(lgbc.stress_centrality(g, src + 1), oracle.stress(rp, ci, src, **kw))
    assert h.stats()["levels"] > 0


@pytest.mark.parametrize("directed,endpoints", [(False, False), (True, True)])
def test_stacked_unions(directed, endpoints):
    g = gen.erdos_renyi_nm(2000, 7000, seed=9, directed=directed)
    src = np.random.default_rng(4).choice(g.nv(), 900, replace=False)
    want = oracle_bc(g, src, endpoints=endpoints)
    levels = {}
    for stack in (0, 1 << 21):
        h = batches(g, stack_vertices=stack)
        assert_bc_close(lgbc.betweenness_centrality(g, src + 1, endpoints=endpoints), want)
        levels[stack] = h.stats()["levels"]
    assert 0 < levels[1 << 21] < levels[0] / 4  # eight batches in one union


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("loop", [0, 1])
@pytest.mark.parametrize("stack", [0, 1 << 21])
def test_weighted_batches(directed, loop, stack):
    g = gen.erdos_renyi_nm(3000, 12000, seed=21, directed=directed)
    rng = np.random.default_rng(8)
    src = rng.integers(0, g.nv(), 700).astype(np.int32)
    w = rng.uniform(0.2, 3.0, len(src))
    h = batches(g, graph_loop=loop, stack_vertices=stack)
    rp, ci, kw = csr_args(g)
    _, want = oracle.dependency(rp, ci, src, w, **kw)
    np.testing.assert_allclose(betweenness_raw_weighted(g, src, w), want, rtol=1e-9, atol=1e-9)
    assert h.stats()["levels"] > 0


@pytest.mark.parametrize("name", sorted(BFS_GRAPHS))
def test_single_searches_over_the_grid(name):
    g = BFS_GRAPHS[name]()
    rp, ci, _ = csr_args(g)
    h = batches(g)
    hubs = np.flatnonzero(np.diff(rp) > 1024)
    for srcs in ([0], [int(hubs[0])], [1, 2, 3], np.random.default_rng(3).choice(g.nv(), 25).tolist()):
        got = lgbc.gdistances(g, [s + 1 for s in srcs]).astype(np.int64)
        want = oracle.gdistances(rp, ci, srcs).astype(np.int64)
        want[want == oracle.UNREACHED32] = np.iinfo(g.eltype).max
        assert np.array_equal(got, want)
        assert h.stats()["topdown_levels"] + h.stats()["bottomup_levels"] > 0


@pytest.mark.parametrize("endpoints", [False, True])
def test_unions_of_graphs_that_the_kernel_refuses(endpoints):
    # too deep, too many paths, too many vertices, repeated entries
    def line(n):
        return lgbc.SimpleGraph.from_edge_arrays(n, np.arange(n - 1), np.arange(1, n))
    layers = [(l * 4 + i, l * 4 + 4 + j) for l in range(25) for i in range(4) for j in range(4)]
    graphs = [line(400), lgbc.SimpleGraph.from_edge_arrays(104, *np.asarray(layers).T), line(300),
              gen.erdos_renyi_nm(24000, 12000, seed=1), gen.erdos_renyi_nm(23000, 9000, seed=2)]
    for g, z in zip(graphs, lgbc.betweenness_centrality_many(graphs, normalize=False, endpoints=endpoints)):
        assert_bc_close(z, oracle_bc(g, normalize=False, endpoints=endpoints, nthreads=16))


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("n,k", [(1, 1), (33, 70), (1000, 3), (1024, 8), (1025, 8), (2048, 8), (2049, 8), (127, 129)])
def test_short_distance_tables(n, k, dtype):
    # tables up to the 64 KB that leave through pinned memory, in both types
    e = np.random.default_rng(n).integers(0, n, (2, 2 * n))
    g = lgbc.SimpleGraph.from_edge_arrays(n, e[0], e[1], eltype=dtype)
    rp, ci, _ = csr_args(g)
    batches(g)
    src = np.random.default_rng(k).integers(0, n, k).astype(np.int32)
    want = oracle.gdistances_many(rp, ci, src).astype(np.int64)
    want[want == oracle.UNREACHED32] = np.iinfo(dtype).max
    for _ in range(2):
        got = lgbc.multi_gdistances(g, src + 1)
        assert got.dtype == dtype and np.array_equal(got, want)
