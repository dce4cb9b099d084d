"""Joins of wide rows (d > 8): members in column blocks of 32, the list's lower
bounds, and the scan that gives a query a whole block when there are few.

Sizes sit at the edges: one row more or less than a block, rows with one float
in their last chunk, every top-k variant, few queries (a block each) and many
(a warp each).
"""
import numpy as np
import pytest

from knn_sweet_b200 import knnjoin
from tests.parity import assert_matches

pytestmark = pytest.mark.gpu


def _mix(rng, n, d, centres):
    return (centres[rng.integers(0, len(centres), n)] +
            0.5 * rng.standard_normal((n, d))).astype(np.float32)


@pytest.mark.parametrize("d,k", [(9, 10), (16, 1), (17, 24), (17, 25), (31, 64), (33, 128),
                                 (64, 200), (100, 300), (130, 600), (257, 5)])
@pytest.mark.parametrize("m", [40, 3000])
def test_wide_rows(cuda_device, oracle, d, k, m):
    rng = np.random.default_rng(d * 1000 + k)
    centres = rng.uniform(-3, 3, (12, d))
    r, q = _mix(rng, 2001, d, centres), _mix(rng, m, d, centres)
    idx, dist = knnjoin(q, r, k, sreps=90)
    rows = rng.permutation(m)[:400]
    oi, od = oracle.bruteforce_f64(q[rows], r, k)
    assert_matches(idx[rows], dist[rows], oi, od)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 65])
@pytest.mark.parametrize("precision", ["fp32", "bf16_refine"])
def test_column_block_edges(cuda_device, oracle, n, precision):
    rng = np.random.default_rng(n)
    r = rng.standard_normal((n, 36)).astype(np.float32)
    q = rng.standard_normal((200, 36)).astype(np.float32)
    idx, dist = knnjoin(q, r, 7, sreps=min(n, 3), precision=precision)
    oi, od = oracle.bruteforce_f64(q, r, 7)
    assert_matches(idx, dist, oi, od)


def test_few_queries_ties(cuda_device, oracle):
    # a block per query: equal distances in several warps' shares
    rng = np.random.default_rng(3)
    r = rng.integers(0, 2, (4000, 12)).astype(np.float32)
    q = rng.integers(0, 2, (33, 12)).astype(np.float32)
    for k in (3, 20, 100):
        idx, dist = knnjoin(q, r, k, sreps=64)
        oi, od = oracle.bruteforce_f64(q, r, k)
        assert_matches(idx, dist, oi, od, exact=True)


def test_tile_that_reaches_too_far(cuda_device, oracle):
    # one query cluster over two distant groups and every member a candidate:
    # the tile goes back to the FP32 scan, with the same result
    rng = np.random.default_rng(9)
    r = np.concatenate([rng.standard_normal((20_000, 16)),
                        rng.standard_normal((20_000, 16)) + 40.0]).astype(np.float32)
    q = np.concatenate([rng.standard_normal((64, 16)),
                        rng.standard_normal((64, 16)) + 40.0]).astype(np.float32)
    idx, dist, st = knnjoin(q, r, 20, qreps=1, sreps=40, precision="bf16_refine", stats=True)
    oi, od = oracle.bruteforce_f64(q, r, 20)
    assert_matches(idx, dist, oi, od)
    assert st.refine_fallbacks > 0


def test_most_tiles_reach_too_far(cuda_device, oracle):
    # more such tiles than may be handed back: the others are streamed
    rng = np.random.default_rng(10)
    r = rng.standard_normal((40_000, 16)).astype(np.float32)
    q = rng.standard_normal((6000, 16)).astype(np.float32)
    idx, dist, st = knnjoin(q, r, 20, qreps=40, sreps=3, precision="bf16_refine", stats=True)
    rows = rng.permutation(6000)[:400]
    oi, od = oracle.bruteforce_f64(q[rows], r, 20)
    assert_matches(idx[rows], dist[rows], oi, od)
    assert 0 < st.refine_fallbacks < 6000


@pytest.mark.parametrize("m", [1500, 5000])
def test_queries_left_to_a_block(cuda_device, oracle, m):
    # four clusters of 15,000 rows: every query passes the step limit of a warp
    # (and, with 5,000, more of them than the list of such queries holds)
    rng = np.random.default_rng(m)
    r = rng.standard_normal((60_000, 16)).astype(np.float32)
    q = rng.standard_normal((m, 16)).astype(np.float32)
    idx, dist = knnjoin(q, r, 40, sreps=4, qreps=8)
    rows = rng.permutation(m)[:200]
    oi, od = oracle.bruteforce_f64(q[rows], r, 40)
    assert_matches(idx[rows], dist[rows], oi, od)
    assert (idx >= 0).all()


@pytest.mark.parametrize("m", [3000, 5000])
def test_statistics_of_queries_left_to_a_block(cuda_device, m):
    # no cluster is out of reach and every query passes the step limit: each of
    # its distances and list entries counts once
    rng = np.random.default_rng(m)
    n, reps = 60_000, 4
    r = rng.standard_normal((n, 16)).astype(np.float32)
    q = (3 * rng.standard_normal((m, 16))).astype(np.float32)
    st = knnjoin(q, r, 40, sreps=reps, qreps=8, stats=True)[2]
    assert 0 < st.dist_evals <= st.pairs_total == m * n
    assert st.pairs_pruned == st.pairs_total - st.dist_evals
    assert st.clusters_visited + st.clusters_pruned <= m * reps


@pytest.mark.parametrize("k", [1, 8, 24, 25, 64, 200, 256, 257, 700])
@pytest.mark.parametrize("sreps", [1, 2, 31, 33])
def test_few_queries_few_clusters(cuda_device, oracle, k, sreps):
    # a block per query, its warps sharing every cluster (lists of fewer than 32)
    # or dealt whole clusters; two distant groups, clusters of every remainder
    rng = np.random.default_rng(100 * sreps + k)
    n = 2049 + 31 * sreps
    side = rng.integers(0, 2, (n, 1)) * 50.0
    r = (rng.standard_normal((n, 16)) + side).astype(np.float32)
    q = (rng.standard_normal((45, 16)) + 50.0 * rng.integers(0, 2, (45, 1))).astype(np.float32)
    idx, dist, st = knnjoin(q, r, k, sreps=sreps, stats=True)
    oi, od = oracle.bruteforce_f64(q, r, k)
    assert_matches(idx, dist, oi, od)
    assert 0 < st.dist_evals <= st.pairs_total
    assert st.clusters_visited + st.clusters_pruned <= 45 * sreps


@pytest.mark.parametrize("sreps", [1, 5])
def test_few_clusters_ties(cuda_device, oracle, sreps):
    # the k-th of the warps' shared words among crowds of equal distances
    rng = np.random.default_rng(sreps)
    r = rng.integers(0, 2, (3000, 10)).astype(np.float32)
    q = rng.integers(0, 2, (20, 10)).astype(np.float32)
    for k in (2, 24, 60):
        idx, dist = knnjoin(q, r, k, sreps=sreps)
        oi, od = oracle.bruteforce_f64(q, r, k)
        assert_matches(idx, dist, oi, od, exact=True)


def _few_far_queries(k):
    # 100 queries in the middle of 60,000 rows reach all of their hundred clusters
    # and more; 4,900 in small groups far away are done at once, and leave the
    # warps idle in which the others are given up
    rng = np.random.default_rng(k)
    groups = 1000.0 * rng.standard_normal((40, 16)) + 5000.0
    r = np.concatenate([rng.standard_normal((60_000, 16)),
                        groups[rng.integers(0, 40, 2000)] + 0.01 * rng.standard_normal((2000, 16))])
    q = np.concatenate([2 * rng.standard_normal((100, 16)),
                        groups[rng.integers(0, 40, 4900)] + 0.01 * rng.standard_normal((4900, 16))])
    return r.astype(np.float32), q[rng.permutation(5000)].astype(np.float32)


@pytest.mark.parametrize("k", [10, 40])
def test_long_lists_left_to_a_block(cuda_device, oracle, k):
    r, q = _few_far_queries(k)
    idx, dist, st = knnjoin(q, r, k, sreps=150, qreps=60, stats=True)
    far = np.flatnonzero(np.abs(q).max(1) < 100)
    rows = np.concatenate([far, np.random.default_rng(1).permutation(5000)[:200]])
    oi, od = oracle.bruteforce_f64(q[rows], r, k)
    assert_matches(idx[rows], dist[rows], oi, od)
    assert (idx >= 0).all() and len(far) == 100
    assert 0 < st.dist_evals <= st.pairs_total


def test_chunked_host_join_orders_no_clusters(cuda_device):
    # 8,192 queries by 256 results go back in eight chunks of rows: three launches
    # each, three to make them, and no order of the clusters, which only a scan of
    # all slots follows; one query less is one scan
    rng = np.random.default_rng(2)
    r = rng.standard_normal((9000, 9)).astype(np.float32)
    q = rng.standard_normal((8192, 9)).astype(np.float32)
    launches = {m: knnjoin(q[:m], r, 256, sreps=100, qreps=100, stats=True)[2].kernels_launched
                for m in (8191, 8192)}
    assert launches[8192] - launches[8191] == 3 + 8 * 3 - 3
