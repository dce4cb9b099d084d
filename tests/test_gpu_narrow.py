"""Joins of narrow rows (d <= 8): the block order of the clusters, the group
scan (k <= 32 and enough queries) and the warp scan over blocks.

Sizes sit where they can go wrong: clusters of a few members, blocks of 32 and
runs of 1,024 positions with one row more or less, the smallest and largest k
of every list length, and crowds of equal distances that overflow a lane's
candidate column.  Group-scan cases pass at least 38,000 queries.
"""
import numpy as np
import pytest

from knn_sweet_b200 import knnjoin
from tests.parity import assert_matches

pytestmark = pytest.mark.gpu

MANY = 38_401  # queries: the group scan, with a remainder of one


def _check(oracle, q, r, k, exact=False, sample=600, **kw):
    idx, dist = knnjoin(q, r, k, **kw)
    rows = np.random.default_rng(1).permutation(q.shape[0])[:sample]
    oi, od = oracle.bruteforce_f64(q[rows], r, k)
    assert_matches(idx[rows], dist[rows], oi, od, exact=exact)


@pytest.mark.parametrize("d,k", [(1, 1), (2, 4), (3, 1), (3, 2), (3, 5), (3, 8), (3, 9), (3, 16),
                                 (3, 17), (3, 32), (4, 8), (4, 32), (5, 16), (8, 1), (8, 20)])
def test_group_scan_float_rows(cuda_device, oracle, d, k):
    rng = np.random.default_rng(10 * d + k)
    r = rng.standard_normal((2049, d)).astype(np.float32)
    q = rng.standard_normal((MANY, d)).astype(np.float32)
    _check(oracle, q, r, k)


@pytest.mark.parametrize("d,k", [(5, 8), (6, 8), (6, 9), (7, 4), (7, 5), (8, 4), (8, 5)])
def test_group_scan_limit_of_k(cuda_device, oracle, d, k):
    rng = np.random.default_rng(10 * d + k)
    r = rng.standard_normal((2049, d)).astype(np.float32)
    q = rng.standard_normal((MANY, d)).astype(np.float32)
    _check(oracle, q, r, k)


@pytest.mark.parametrize("n", [1, 3, 31, 32, 33, 1023, 1024, 1025])
def test_group_scan_reference_sizes(cuda_device, oracle, n):
    rng = np.random.default_rng(n)
    r = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    q = rng.uniform(-1, 1, (MANY, 3)).astype(np.float32)
    _check(oracle, q, r, 16, sreps=min(n, 7))


@pytest.mark.parametrize("k", [1, 4, 16, 31])
def test_group_scan_crowds_of_equal_distances(cuda_device, oracle, k):
    # 64 distinct integer points, 600 copies of each: every list overflows with ties
    rng = np.random.default_rng(k)
    base = rng.integers(0, 4, (64, 3)).astype(np.float32)
    x = base[rng.integers(0, 64, MANY)]
    _check(oracle, x, x, k, exact=True, sample=200)
    # the same shifted off the integers: the boundary is decided in FP64
    y = x + np.float32(0.1)
    _check(oracle, y, y, k, sample=200)


@pytest.mark.parametrize("d,k,sreps", [(1, 40, 3), (3, 33, 1), (3, 64, 50), (3, 200, 9),
                                       (4, 100, 4), (6, 300, 20), (8, 1000, 5), (3, 24, 2)])
def test_warp_scan_over_blocks(cuda_device, oracle, d, k, sreps):
    rng = np.random.default_rng(100 * d + k)
    r = rng.standard_normal((3000, d)).astype(np.float32)
    q = rng.standard_normal((257, d)).astype(np.float32)
    _check(oracle, q, r, k, sample=257, sreps=sreps)


def test_tiny_clusters_and_far_outliers(cuda_device, oracle):
    # as many representatives as points, and one point that stretches a cluster
    rng = np.random.default_rng(5)
    r = rng.standard_normal((500, 3)).astype(np.float32)
    r[17] = 1e6
    q = rng.standard_normal((MANY, 3)).astype(np.float32)
    _check(oracle, q, r, 8, sreps=500)
    _check(oracle, q, r, 8, sreps=1, qreps=1)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1024, 1025, 4095, 4096, 4097])
@pytest.mark.parametrize("d,k", [(1, 5), (3, 16), (3, 200), (4, 1), (5, 33), (8, 24)])
def test_small_joins(cuda_device, oracle, n, d, k):
    # up to 4,096 reference rows and no representatives asked for: one cluster
    rng = np.random.default_rng(1000 * d + n)
    r = rng.standard_normal((n, d)).astype(np.float32)
    q = (2 * rng.standard_normal((123, d))).astype(np.float32)
    _check(oracle, q, r, k, sample=123)
    _check(oracle, r, r, k, sample=200)
    ints = rng.integers(0, 6, (n, d)).astype(np.float32)
    _check(oracle, ints, ints, k, exact=True, sample=100)


def test_small_join_self_and_missing_slots(cuda_device):
    import torch
    x = torch.tensor([[0.0, 0, 0], [1, 0, 0], [float("nan"), 0, 0], [3, 0, 0]], device="cuda")
    idx, dist = knnjoin(x, None, 6)
    assert idx[0].tolist() == [0, 1, 3, -1, -1, -1]
    assert dist[0, :3].tolist() == [0.0, 1.0, 3.0] and bool(torch.isinf(dist[0, 3:]).all())
    assert idx[2].tolist() == [-1] * 6  # no distance from a NaN query is a number


@pytest.mark.parametrize("d,n,m", [(3, 2 * MANY, MANY), (3, 2 * MANY + 1, MANY), (4, 60_000, 76_000),
                                   (4, 60_000, 75_000), (6, 9000, MANY), (6, 10_000, MANY),
                                   (8, 9600, MANY)])
def test_group_scan_limit_of_density(cuda_device, oracle, d, n, m):
    # enough queries for groups of 32, but as many reference rows on both sides of
    # the limit from which they lie too far apart
    rng = np.random.default_rng(n + d)
    r = rng.uniform(-1, 1, (n, d)).astype(np.float32)
    q = rng.uniform(-1, 1, (m, d)).astype(np.float32)
    _check(oracle, q, r, 4, sample=150)


@pytest.mark.parametrize("d", [5, 6, 7, 8])
@pytest.mark.parametrize("n", [8191, 8192, 8193, 9985])
def test_thread_scan_selfjoin(cuda_device, oracle, d, n):
    # k = 1 of a set with itself: copies of a point (the lowest row wins), rows on
    # and off the integers, more than 128 points a cluster (not this kernel's)
    rng = np.random.default_rng(100 * d + n)
    x = rng.standard_normal((n, d)).astype(np.float32)
    x[n // 2:] = x[rng.integers(0, n // 2, n - n // 2)]
    ints = rng.integers(0, 3, (n, d)).astype(np.float32)
    for kw in ({}, {"sreps": n // 128 + 1, "qreps": n // 128 + 1}, {"sreps": 20, "qreps": 20}):
        _check(oracle, x, x, 1, sample=200, **kw)
        _check(oracle, ints, ints, 1, exact=True, sample=200, **kw)


@pytest.mark.parametrize("d,k", [(1, 32), (2, 2), (2, 8), (2, 17), (2, 32), (3, 32), (6, 4)])
def test_group_scan_cut_columns(cuda_device, oracle, d, k):
    # every list and column overflows with equal distances again and again, within
    # a cluster and between clusters; both in whole numbers and off them
    rng = np.random.default_rng(10 * d + k)
    r = rng.integers(0, 3, (9000, d)).astype(np.float32)
    q = rng.integers(0, 3, (MANY, d)).astype(np.float32)
    for sreps in (0, 9):
        _check(oracle, q, r, k, exact=True, sample=150, sreps=sreps, qreps=sreps)
    r[::2] += np.float32(1e-3)
    _check(oracle, q + np.float32(0.3), r, k, sample=150)


@pytest.mark.parametrize("m,k,small", [(2049, 512, True), (2048, 513, True), (2049, 513, False),
                                       (4096, 1000, False)])
def test_small_join_limit_of_k(cuda_device, oracle, m, k, small):
    # many results of few rows: one cluster, or the clustered join
    rng = np.random.default_rng(k)
    r = (rng.standard_normal((4096, 5)) + 30.0 * rng.integers(0, 5, (4096, 1))).astype(np.float32)
    q = (rng.standard_normal((m, 5)) + 30.0 * rng.integers(0, 5, (m, 1))).astype(np.float32)
    idx, dist, st = knnjoin(q, r, k, stats=True)
    rows = rng.permutation(m)[:100]
    oi, od = oracle.bruteforce_f64(q[rows], r, k)
    assert_matches(idx[rows], dist[rows], oi, od)
    assert (st.sreps_used == 1) == small
