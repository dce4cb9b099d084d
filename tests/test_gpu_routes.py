"""Ways into the scans of narrow rows that the sizes of the other tests do not
take: the group scan over a list of slots and over a range of them, joins without
allocation (with and without room for the blocks' boxes), and rows that are not
numbers among many queries.
"""
import ctypes

import numpy as np
import pytest

from knn_sweet_b200 import _lib, knnjoin
from knn_sweet_b200.join import knnjoin_partition, knnjoin_sharded
from tests.parity import assert_matches

pytestmark = pytest.mark.gpu

MANY = 38_401  # queries: the group scan, with a remainder of one


def _check(oracle, q, r, k, idx, dist, sample=400):
    rows = np.random.default_rng(1).permutation(q.shape[0])[:sample]
    oi, od = oracle.bruteforce_f64(q[rows], r, k)
    assert_matches(idx[rows], dist[rows], oi, od)


@pytest.mark.parametrize("d,k", [(3, 16), (2, 9), (3, 32), (8, 4)])
def test_group_scan_in_chunks_of_rows(cuda_device, oracle, d, k):
    # host arrays: eight chunks, the first of 4,736 queries (a warp each), the
    # others of 38,000 and more (groups over a list of slots)
    rng = np.random.default_rng(d + k)
    m = 4736 + 7 * 38_000 if k > 8 else 4736 + 7 * 75_000
    r = rng.standard_normal((4999, d)).astype(np.float32)
    q = rng.standard_normal((m, d)).astype(np.float32)
    idx, dist = knnjoin(q, r, k)
    _check(oracle, q, r, k, idx, dist)


@pytest.mark.parametrize("d,k", [(3, 1), (3, 16), (6, 4)])
def test_group_scan_of_a_range(cuda_device, oracle, d, k):
    import torch
    rng = np.random.default_rng(d * k)
    r = rng.standard_normal((7001, d)).astype(np.float32)
    q = rng.standard_normal((3 * MANY, d)).astype(np.float32)
    tq, tr = torch.from_numpy(q).to(cuda_device), torch.from_numpy(r).to(cuda_device)
    seen = np.zeros(q.shape[0], int)
    for part in range(3):
        idx, dist, rows = knnjoin_partition(tq, tr, k, part=part, nparts=3)
        rows = rows.cpu().numpy()
        seen[rows] += 1
        _check(oracle, q[rows], r, k, idx.cpu().numpy()[rows], dist.cpu().numpy()[rows], 200)
    assert (seen == 1).all()
    idx, dist = knnjoin_sharded(q, r, k, devices=(0, 0, 0))
    _check(oracle, q, r, k, idx, dist)


@pytest.mark.parametrize("reps", [60, 500])
@pytest.mark.parametrize("d,k,m", [(3, 16, MANY), (3, 1, MANY), (3, 40, 900), (4, 1, MANY),
                                   (6, 4, MANY), (8, 70, 900), (12, 9, 900)])
def test_join_without_allocation(cuda_device, oracle, d, k, m, reps):
    # 500 clusters of 2,000 rows leave no room for the boxes
    import torch
    rng = np.random.default_rng(d * k + reps)
    r = rng.standard_normal((2000, d)).astype(np.float32)
    q = rng.standard_normal((m, d)).astype(np.float32)
    tq, tr = torch.from_numpy(q).to(cuda_device), torch.from_numpy(r).to(cuda_device)
    idx = torch.empty((m, k), dtype=torch.int32, device=cuda_device)
    dist = torch.empty((m, k), dtype=torch.float32, device=cuda_device)
    opt = _lib.default_options()
    opt.qreps = opt.sreps = reps
    lib = _lib.load()
    rc = lib.knn_join_device_noalloc(
        ctypes.c_void_p(tq.data_ptr()), m, ctypes.c_void_p(tr.data_ptr()), 2000, d, k,
        ctypes.c_void_p(idx.data_ptr()), ctypes.c_void_p(dist.data_ptr()), ctypes.byref(opt),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _lib.KNN_OK, lib.knn_last_error()
    _check(oracle, q, r, k, idx.cpu().numpy(), dist.cpu().numpy())


@pytest.mark.parametrize("d,k", [(3, 1), (3, 8), (4, 16), (6, 4), (8, 1)])
@pytest.mark.parametrize("m", [900, MANY])
def test_rows_that_are_not_numbers(cuda_device, oracle, d, k, m):
    # NaN and infinite rows on both sides, a hundred copies of one NaN row (blocks
    # without a number): the finite queries' neighbours are the finite rows'
    rng = np.random.default_rng(d + k)
    r = rng.standard_normal((6000, d)).astype(np.float32)
    q = rng.standard_normal((m, d)).astype(np.float32)
    bad_r = rng.permutation(6000)[:400]
    r[bad_r[:100]] = np.nan
    r[bad_r[100:200], 0] = np.nan
    r[bad_r[200:300], d - 1] = np.inf
    r[bad_r[300:]] = -np.inf
    bad_q = rng.permutation(m)[:60]
    q[bad_q[:20]] = np.nan
    q[bad_q[20:40], d - 1] = np.nan
    q[bad_q[40:], 0] = np.inf
    fin_r = np.flatnonzero(np.isfinite(r).all(1))
    fin_q = np.flatnonzero(np.isfinite(q).all(1))
    idx, dist = knnjoin(q, r, k, sreps=70, qreps=70)
    rows = fin_q[np.random.default_rng(1).permutation(fin_q.size)[:400]]
    oi, od = oracle.bruteforce_f64(q[rows], r[fin_r], k)
    assert_matches(idx[rows], dist[rows], fin_r[oi].astype(np.int32), od)
    assert (idx[bad_q[:40]] == -1).all() and np.isinf(dist[bad_q[:40]]).all()
