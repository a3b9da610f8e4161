"""The shared-memory betweenness and distance kernels of small graphs (small.cu)
against the oracle where it can go wrong: chunk and warp edges of the vertex count, rows
at the lengths where threads hand over to warps, every row long, levels at the
depth cap, path counts around 2^16, 2^32 and 2^48, sources nothing enters,
repeats, weights, and the sizes on both sides of the shared-memory limit."""
import numpy as np
import pytest

import lgbc
from lgbc import generators as G
from lgbc.learned import betweenness_raw_weighted
from conftest import csr_args
from oracle import oracle
from test_gpu_parity import assert_bc_close, oracle_bc

pytestmark = pytest.mark.gpu


def random_graph(n, m, seed, directed=False):
    e = np.random.default_rng(seed).integers(0, n, (2, m))
    return (lgbc.SimpleDiGraph if directed else lgbc.SimpleGraph).from_edge_arrays(n, e[0], e[1])


def path(n):
    return lgbc.SimpleGraph.from_edge_arrays(n, np.arange(n - 1), np.arange(1, n))


def layers(count, width):
    """Complete bipartite steps between consecutive layers: width^L paths to layer L + 1."""
    e = [(l * width + i, (l + 1) * width + j) for l in range(count - 1) for i in range(width)
         for j in range(width)]
    return lgbc.SimpleGraph.from_edge_arrays(count * width, *np.asarray(e).T)


def fan(n, degree):
    """A vertex of the given degree among short rows."""
    ring = np.arange(n)
    return lgbc.SimpleGraph.from_edge_arrays(
        n, np.concatenate([ring, np.zeros(degree, int)]),
        np.concatenate([(ring + 1) % n, 1 + np.arange(degree)]))


def check(g, sources=None, endpoints=False):
    vs = None if sources is None else np.asarray(sources) + 1
    got = lgbc.betweenness_centrality(g, vs, normalize=False, endpoints=endpoints)
    assert_bc_close(got, oracle_bc(g, sources, normalize=False, endpoints=endpoints, nthreads=8))


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65, 300, 1023, 1025])
@pytest.mark.parametrize("degree", [1, 5, 80])
def test_vertex_counts(n, degree, directed):
    # degree 80: every row is walked by a warp and the last chunk is ragged
    check(random_graph(n, n * degree // (1 if directed else 2) + 1, n + degree, directed),
          endpoints=n % 2 == 0)


@pytest.mark.parametrize("degree", [60, 61, 62, 63, 64, 65, 128, 129, 1500])
def test_row_lengths(degree):
    # with its two ring edges the first vertex's row crosses 64 entries at 62
    check(fan(2000, degree), np.arange(0, 2000, 13))


@pytest.mark.parametrize("n", [126, 127, 128, 129, 130, 131, 400])
def test_depths(n):
    check(path(n))


@pytest.mark.parametrize("count,width", [(10, 4), (17, 4), (18, 4), (12, 8), (13, 8), (24, 4), (26, 4)])
def test_path_counts(count, width):
    # 2^16, 2^32 and 2^48 paths lie between these depths
    check(layers(count, width), np.arange(0, count * width, 3))


def test_sources_nothing_enters_and_other_components():
    n = 500
    e = np.random.default_rng(5).integers(50, 400, (2, 900))
    src = np.concatenate([e[0], np.arange(50)])
    dst = np.concatenate([e[1], np.random.default_rng(6).integers(50, 400, 50)])
    g = lgbc.SimpleDiGraph.from_edge_arrays(n, src, dst)
    check(g)
    check(g, [0, 0, 49, 60, 60, 450, 499])


@pytest.mark.parametrize("n", [10000, 22000, 24000])
def test_shared_memory_limit(n):
    check(random_graph(n, 3 * n, n), np.arange(0, n, n // 40))
    check(G.barabasi_albert(n, 3, seed=n), np.arange(0, n, n // 40))


def test_weights_and_repeats():
    g = G.rmat(10, 8, seed=2)
    rp, ci, _ = csr_args(g)
    rng = np.random.default_rng(3)
    src = rng.integers(0, g.nv(), 700).astype(np.int32)
    w = rng.random(700) * np.where(rng.random(700) < 0.1, 0.0, 10.0)
    _, want = oracle.dependency(rp, ci, src, w)
    np.testing.assert_allclose(betweenness_raw_weighted(g, src, w), want, rtol=1e-9)


@pytest.mark.parametrize("endpoints", [False, True])
def test_many_mixed(endpoints):
    # size classes, a refused depth, refused counts, isolated vertices, and a
    # graph beyond the limit in one call
    graphs = [G.barabasi_albert(n, 3, seed=n) for n in (30, 1500, 3000, 5000, 12000)]
    graphs += [path(400), layers(26, 4), lgbc.SimpleGraph(0), lgbc.SimpleGraph(7),
               random_graph(2000, 900, 8), random_graph(300, 12000, 9), path(2)]
    small = [g for g in graphs if g.nv() <= 5000]
    for g, z in zip(small, lgbc.betweenness_centrality_many(small, normalize=False, endpoints=endpoints)):
        assert_bc_close(z, oracle_bc(g, normalize=False, endpoints=endpoints, nthreads=8))
    big = [graphs[4], G.erdos_renyi_nm(24000, 12000, seed=1)]
    for g, z in zip(big, lgbc.betweenness_centrality_many(big, normalize=False, endpoints=endpoints)):
        assert_bc_close(z, lgbc.betweenness_centrality(g, normalize=False, endpoints=endpoints))


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n", [1, 2, 32, 33, 300, 1025, 18800, 19200])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 70])
def test_distances(n, k, directed):
    # lanes at the edges of a block's 32, both sides of the size limit, long rows at n = 300
    g = random_graph(n, n * (80 if n == 300 else 2), n + k, directed)
    rp, ci, _ = csr_args(g)
    src = np.random.default_rng(k).integers(0, n, k).astype(np.int32)
    want = np.stack([oracle.gdistances(rp, ci, [s]) for s in src]).astype(np.int64)
    far = want == oracle.UNREACHED32
    top = np.iinfo(g.eltype).max
    assert np.array_equal(lgbc.multi_gdistances(g, src + 1), np.where(far, top, want))
    reached, dsum, dmax = lgbc.distance.distance_stats(g, src)
    assert np.array_equal(reached, (~far).sum(1))
    assert np.array_equal(dsum, np.where(far, 0, want).sum(1))
    assert np.array_equal(dmax, np.where(far, 0, want).max(1))
    nearest = np.where(far, top, want).min(0)
    assert np.array_equal(lgbc.gdistances(g, src + 1), nearest)


def test_distances_along_a_path():
    g = path(3000)
    d = lgbc.multi_gdistances(g, [1, 1500, 3000])
    i = np.arange(3000)
    assert np.array_equal(d, np.stack([i, abs(i - 1499), 2999 - i]))


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("n,degree", [(1, 1), (2, 1), (33, 5), (300, 80), (1025, 3), (16384, 6), (18900, 2), (19200, 2)])
def test_stress(n, degree, directed):
    # odd and even vertex counts (two counts share a word), long rows, both
    # sides of the size limit; whole numbers, compared exactly
    g = random_graph(n, n * degree // (1 if directed else 2) + 1, n, directed)
    rp, ci, kw = csr_args(g)
    src = np.random.default_rng(n).integers(0, n, min(n, 60)).astype(np.int32)
    want = oracle.stress(rp, ci, src, **kw)
    assert np.array_equal(lgbc.stress_centrality(g, src + 1), want)


def test_stress_wraps_and_depths():
    for g in (layers(40, 4), path(126), path(400), fan(2000, 1500)):
        rp, ci, kw = csr_args(g)
        src = np.arange(0, g.nv(), 3, dtype=np.int32)
        assert np.array_equal(lgbc.stress_centrality(g, src + 1), oracle.stress(rp, ci, src, **kw))


def test_many_rejects_what_it_did():
    good = path(5)
    bad = lgbc.SimpleGraph.from_csr([0, 1, 2, 2], [1, 3])
    with pytest.raises(lgbc.ArgumentError, match="column index"):
        lgbc.betweenness_centrality_many([good, bad])
    drop = lgbc.SimpleGraph.from_csr([0, 2, 1, 2], [1, 2])
    with pytest.raises(lgbc.ArgumentError, match="rowptr"):
        lgbc.betweenness_centrality_many([good, drop])


def test_repeated_entries_take_the_batches():
    # a row longer than n (repeated entries): accepted as before
    g = lgbc.SimpleGraph.from_csr([0, 4, 7, 8], [1, 1, 1, 1, 0, 0, 2, 1])
    h = lgbc.SimpleGraph.from_csr([0, 4, 7, 8], [1, 1, 1, 1, 0, 0, 2, 1])
    h.device_handle().set_tuning(stack_vertices=0)
    a, b = (lgbc.betweenness_centrality(x, normalize=False) for x in (g, h))
    np.testing.assert_allclose(a, b, rtol=1e-12)
    np.testing.assert_allclose(lgbc.betweenness_centrality_many([g], normalize=False)[0], b, rtol=1e-12)


@pytest.mark.parametrize("n", [8191, 8192, 8193])
@pytest.mark.parametrize("k", [8, 9, 256, 257])
def test_results_and_sources_at_the_sizes_of_the_pinned_areas(n, k):
    # n 8-byte results fill the pinned 64 KB at 8192; 8 sources travel with a
    # search's launch, 256 sources are read where the host wrote them
    g = random_graph(n, 2 * n, n + k)
    src = np.random.default_rng(k).choice(n, k, replace=False)
    for _ in range(2):  # the second call finds the first one's counters and areas
        check(g, src)
    rp, ci, _ = csr_args(g)
    want = oracle.gdistances(rp, ci, src.astype(np.int32)).astype(np.int64)
    want[want == oracle.UNREACHED32] = np.iinfo(g.eltype).max
    assert np.array_equal(lgbc.gdistances(g, src + 1), want)


def deep_and_shallow():
    """A digraph of a path of 300 and a random part: sources near the path's head
    are deeper than a per-source search may be, all others are shallow."""
    e = np.random.default_rng(7).integers(300, 2000, (2, 8000))
    i = np.arange(299)
    return lgbc.SimpleDiGraph.from_edge_arrays(2000, np.concatenate([i, e[0]]), np.concatenate([i + 1, e[1]]))


@pytest.mark.parametrize("kind", ["betweenness", "stress"])
def test_deep_sources_leave_the_others_as_they_are(kind):
    g = deep_and_shallow()
    rp, ci, kw = csr_args(g)
    h = g.device_handle()
    shallow = np.concatenate([np.arange(290, 299), np.arange(300, 2000, 9)])
    deep = np.asarray([3, 100, 171])

    def call(src):
        if kind == "stress":
            got = lgbc.stress_centrality(g, src + 1)
            assert np.array_equal(got, oracle.stress(rp, ci, src.astype(np.int32), **kw))
        else:
            got = lgbc.betweenness_centrality(g, src + 1, normalize=False)
            assert_bc_close(got, oracle_bc(g, src, normalize=False))
        return got, h.stats()["levels"], h.stats()["kernel_launches"]

    first, levels, _ = call(shallow)
    assert levels == 0  # the per-source kernel counts none
    attempt = call(deep)
    assert attempt[1] > 127
    again = call(deep)
    assert again[2] < attempt[2]  # not tried twice
    assert np.array_equal(again[0], attempt[0])
    last, levels, _ = call(shallow)
    assert levels == 0 and np.array_equal(first, last)
    assert call(np.concatenate([shallow, deep]))[1] > 127


def test_graphs_of_deep_sources_are_left_to_batches():
    # one attempt, then the launches of a handle that never tries (a hub order
    # other than the default, which a graph without hubs does not notice)
    g, never = path(2000), path(2000)
    never.device_handle().set_tuning(hub_order=1)
    more = []
    for s in (0, 5, 9):
        for x in (g, never):
            check(x, np.arange(s, 2000, 10))
        more.append(g.device_handle().stats()["kernel_launches"] - never.device_handle().stats()["kernel_launches"])
    assert more[0] > 0 and more[1:] == [0, 0]


@pytest.mark.parametrize("n", [127, 128, 129, 130])
def test_where_the_depth_limit_lies(n):
    # distances up to 127 (a call counts levels only when batches run)
    g = path(n)
    check(g, [0])
    levels = g.device_handle().stats()["levels"]
    assert levels == 0 if n <= 128 else levels >= 128


@pytest.mark.parametrize("endpoints", [False, True])
def test_many_in_the_large_size_classes(endpoints):
    # one call's launches for graphs of 8,193 to 11,000 and of more vertices
    graphs = [G.barabasi_albert(n, 2, seed=n) for n in (8200, 10900, 11100, 12500)]
    for g, z in zip(graphs, lgbc.betweenness_centrality_many(graphs, normalize=False, endpoints=endpoints)):
        assert_bc_close(z, oracle_bc(g, normalize=False, endpoints=endpoints, nthreads=16))


@pytest.mark.parametrize("n,degree,k,rows_small,stats_small", [
    (1500, 100, 3, True, True), (2400, 40, 64, True, True), (3000, 80, 5, False, True),
    (4000, 90, 64, False, False), (4000, 90, 65, True, True), (7000, 90, 96, False, False), (7000, 90, 97, True, True)])
def test_distances_over_long_rows(n, degree, k, rows_small, stats_small):
    # few searches of a graph of many rows of more than 64 entries run over the
    # whole grid (and count levels), rows on both sides written by every lane
    g = random_graph(n, n * degree // 2, n + degree)
    rp, ci, _ = csr_args(g)
    h = g.device_handle()
    src = np.random.default_rng(k).choice(n, k, replace=False).astype(np.int32)
    want = oracle.gdistances_many(rp, ci, src, nthreads=8).astype(np.int64)
    far = want == oracle.UNREACHED32
    assert np.array_equal(lgbc.multi_gdistances(g, src + 1), np.where(far, np.iinfo(g.eltype).max, want))
    assert (h.stats()["levels"] == 0) == rows_small
    reached, dsum, dmax = lgbc.distance.distance_stats(g, src)
    assert (h.stats()["levels"] == 0) == stats_small
    assert np.array_equal(reached, (~far).sum(1))
    assert np.array_equal(dsum, np.where(far, 0, want).sum(1))
    assert np.array_equal(dmax, np.where(far, 0, want).max(1))


def dense(n, share):
    a, b = np.triu_indices(n, 1)
    keep = np.random.default_rng(n).random(len(a)) < share
    return lgbc.SimpleGraph.from_edge_arrays(n, a[keep], b[keep])


@pytest.mark.parametrize("make,k,small", [
    (lambda: G.barabasi_albert(11500, 1, seed=1), 4800, True), (lambda: G.barabasi_albert(11500, 1, seed=1), 5000, False),
    (lambda: G.barabasi_albert(10900, 1, seed=2), 5000, True), (lambda: G.barabasi_albert(11500, 2, seed=3), 5000, True),
    (lambda: lgbc.SimpleGraph.from_edge_arrays(11500, np.zeros(11499, int), np.arange(1, 11500)), 5000, True),
    (lambda: random_graph(20000, 9000, 4), 5000, True),
    (lambda: dense(800, 0.98), 600, True), (lambda: dense(800, 0.98), 700, False), (lambda: dense(800, 1.0), 700, True),
    (lambda: dense(790, 0.98), 700, True), (lambda: dense(800, 0.93), 700, True)])
def test_graphs_of_many_sources_that_batches_take(make, k, small):
    # trees past one block per SM, nearly complete graphs, and what lies next to them
    g = make()
    src = np.random.default_rng(k).choice(g.nv(), k, replace=False)
    check(g, src)
    assert (g.device_handle().stats()["levels"] == 0) == small
