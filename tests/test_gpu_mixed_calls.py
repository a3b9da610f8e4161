"""Calls of different kinds in turn on one handle: each keeps a workspace there,
and growing one must leave the others as they were.  Int64 graphs (distances in
64 bits pass through a buffer of their own) of more than 2^17 stored entries,
below and above the vertex count up to which searches run in shared memory."""
import numpy as np
import pytest

import lgbc
from conftest import csr_args
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(3000, 80000), (19500, 75000)])
def test_distance_statistics_between_distance_calls(n, m):
    e = np.random.default_rng(n).integers(0, n, (2, m))
    g = lgbc.SimpleGraph.from_edge_arrays(n, e[0], e[1])
    rp, ci, _ = csr_args(g)
    assert g.eltype == np.int64 and rp[n] > 1 << 17
    src = np.arange(0, n, n // 90, dtype=np.int32)
    want = oracle.gdistances_many(rp, ci, src, nthreads=8).astype(np.int64)
    far = want == oracle.UNREACHED32
    top = np.iinfo(np.int64).max

    def statistics():
        reached, dsum, dmax = lgbc.distance.distance_stats(g, src)
        assert np.array_equal(reached, (~far).sum(1))
        assert np.array_equal(dsum, np.where(far, 0, want).sum(1))
        assert np.array_equal(dmax, np.where(far, 0, want).max(1))

    statistics()
    assert np.array_equal(lgbc.gdistances(g, int(src[0]) + 1), np.where(far, top, want)[0])
    statistics()
    assert np.array_equal(lgbc.multi_gdistances(g, src + 1), np.where(far, top, want))
    statistics()
    few = src[:3]
    assert np.array_equal(lgbc.eccentricity(g, list(few + 1)), np.where(far.any(1), top, want.max(1))[:3])


def test_closeness_between_distance_calls():
    n = 3000
    e = np.random.default_rng(5).integers(0, n, (2, 80000))
    g = lgbc.SimpleGraph.from_edge_arrays(n, e[0], e[1])
    rp, ci, _ = csr_args(g)
    want = oracle.closeness(rp, ci, np.diff(rp))
    for call in (lambda: lgbc.gdistances(g, 1), lambda: lgbc.multi_gdistances(g, range(1, 200)), lambda: None):
        assert np.array_equal(lgbc.closeness_centrality(g), want)
        call()


def test_wide_distances_take_a_bounded_buffer():
    # 64 rows of 2^20 vertices: the 64-bit table may cost the device at most
    # 2^25 entries (256 MB) more than the 32-bit one, and more than one piece
    # of it is widened
    torch = pytest.importorskip("torch")
    n = 1 << 20
    e = np.random.default_rng(3).integers(0, n, (2, 3 * n // 2))
    used, rows = {}, {}
    for dtype in (np.int32, np.int64):
        g = lgbc.SimpleGraph.from_edge_arrays(n, e[0], e[1], eltype=dtype)
        g.device_handle()
        free = torch.cuda.mem_get_info()[0]
        rows[dtype] = lgbc.multi_gdistances(g, range(1, 65))
        used[dtype] = free - torch.cuda.mem_get_info()[0]
        del g
    assert used[np.int64] - used[np.int32] <= (1 << 28) + (1 << 23)
    narrow, wide = rows[np.int32], rows[np.int64]
    far = narrow == np.iinfo(np.int32).max
    assert far.any() and np.array_equal(far, wide == np.iinfo(np.int64).max)
    assert np.array_equal(narrow[~far], wide[~far])


@pytest.mark.parametrize("n,k", [(20000, 64), (20000, 65), (20000, 150), (200000, 200)])
def test_wide_tables_of_several_batches(n, k):
    # 64-bit rows wait on the device until 2^25 of them (or the last) are copied:
    # one batch, several in one copy, two copies
    e = np.random.default_rng(n).integers(0, n, (2, 2 * n))
    src = np.random.default_rng(k).choice(n, k, replace=False) + 1
    narrow, wide = (lgbc.multi_gdistances(lgbc.SimpleGraph.from_edge_arrays(n, e[0], e[1], eltype=t), src)
                    for t in (np.int32, np.int64))
    far = narrow == np.iinfo(np.int32).max
    assert wide.dtype == np.int64 and np.array_equal(far, wide == np.iinfo(np.int64).max)
    assert np.array_equal(narrow[~far], wide[~far])
