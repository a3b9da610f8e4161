"""The one-launch BFS (k_bfs_run) against the oracle's gdistances! bit for bit:
rows around the lengths that one claim of a warp covers (128 entries), vertex
counts around the 32-vertex words of its bitmaps, both directions forced and
the default choice between them.  A tuning other than the default keeps these
small graphs on this kernel."""
import numpy as np
import pytest

import lgbc
from conftest import csr_args
from oracle import oracle

pytestmark = pytest.mark.gpu

TUNINGS = {"topdown": (1e-12, 1e12), "bottomup": (1e12, 1e12), "auto": (13.0, 23.0)}


def bfs(g, srcs, tuning):
    rp, ci, _ = csr_args(g)
    alpha, beta = TUNINGS[tuning]
    g.device_handle().set_tuning(alpha=alpha, beta=beta)
    want = oracle.gdistances(rp, ci, np.asarray(srcs, np.int32)).astype(np.int64)
    want[want == oracle.UNREACHED32] = np.iinfo(g.eltype).max
    for _ in range(2):  # the second search finds the first one's state
        assert np.array_equal(lgbc.gdistances(g, np.asarray(srcs) + 1), want), (tuning, srcs)


@pytest.mark.parametrize("tuning", sorted(TUNINGS))
@pytest.mark.parametrize("degree", [31, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1500])
def test_row_lengths(degree, tuning):
    # a hub, its leaves, and a second hub of one more entry two levels on
    n = 2 * degree + 40
    hub2 = degree + 1
    e = [(0, i) for i in range(1, degree + 1)] + [(degree, hub2)]
    e += [(hub2, i) for i in range(hub2 + 1, hub2 + 1 + degree)]
    a = np.asarray(e)
    bfs(lgbc.SimpleGraph.from_edge_arrays(n, a[:, 0], a[:, 1]), [0], tuning)
    bfs(lgbc.SimpleDiGraph.from_edge_arrays(n, a[:, 0], a[:, 1]), [1, 0, degree], tuning)


@pytest.mark.parametrize("tuning", sorted(TUNINGS))
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 40001])
def test_vertex_counts(n, tuning):
    rng = np.random.default_rng(n)
    e = rng.integers(0, n, (2, 3 * n))
    for kind in (lgbc.SimpleGraph, lgbc.SimpleDiGraph):
        bfs(kind.from_edge_arrays(n, e[0], e[1]), [n - 1], tuning)
        bfs(kind.from_edge_arrays(n, e[0], e[1]), rng.integers(0, n, 9).tolist(), tuning)


@pytest.mark.parametrize("tuning", ["bottomup", "auto"])
@pytest.mark.parametrize("length", [4095, 4096, 4097, 8192, 8193, 20000])
def test_long_in_lists_without_a_hit(length, tuning):
    # one thread walks the in-list of a vertex that a bottom-up level does not
    # reach, in stretches of 4,096 entries; its last entry is reached late or never
    tail = 6
    n = length + tail + 2
    hub = n - 1
    chain = length + np.arange(tail + 1)  # vertices after the list's own
    src = np.concatenate([np.arange(length), chain[:-1], [chain[-1]]])
    dst = np.concatenate([np.full(length, hub), chain[1:], [hub]])
    g = lgbc.SimpleDiGraph.from_edge_arrays(n, src, dst)
    bfs(g, [int(chain[0])], tuning)       # the hub's last entry, six levels on
    bfs(g, [length - 1], tuning)          # the last of the list itself
    g = lgbc.SimpleDiGraph.from_edge_arrays(n, src[:-1], dst[:-1])
    bfs(g, [int(chain[0])], tuning)       # never
