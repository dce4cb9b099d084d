"""What steers the search and shows in the statistics only: the k-th bound of a
query cluster, and the order of a cluster's members in the refinement steps.

The representatives of these cases are drawn with the C library's rand(), as the
library draws them, from seeds that pick one row of every group.
"""
import ctypes

import numpy as np
import pytest

from knn_sweet_b200 import knnjoin

pytestmark = pytest.mark.gpu


def _seed(group_of_row, groups):
    libc = ctypes.CDLL("libc.so.6")
    n = len(group_of_row)
    for seed in range(1, 100_000):
        libc.srand(seed)
        if sorted(group_of_row[libc.rand() % n] for _ in range(groups)) == list(range(groups)):
            return seed
    raise AssertionError("no seed found")


@pytest.mark.parametrize("d", [6, 9])
@pytest.mark.parametrize("gap", [1e-5, 1e-4])
def test_kth_bound_is_exact(cuda_device, d, gap):
    # three clusters of one point each, the query at 1, 1 + gap and 1 + 2e-4 of
    # them: the second bounds the second distance and puts the third out of reach
    # (the bound is widened by 1e-5 of itself, the test by half as much again; from
    # d = 16 on the assignment is approximate and the clusters not these)
    r = np.zeros((3, d), np.float32)
    r[:, 0] = 1.0, 1.0 + gap, 1.0 + 2e-4 + gap
    q = np.zeros((1, d), np.float32)
    idx, _, st = knnjoin(q, r, 2, sreps=3, qreps=1, rep_trials=1, seed=_seed([0, 1, 2], 3),
                         stats=True)
    assert idx.tolist() == [[0, 1]]
    assert st.clusters_visited + st.clusters_pruned == 2


@pytest.mark.parametrize("swap", [False, True])
def test_refinement_moves_to_the_farthest_member(cuda_device, swap):
    # four groups of 20, 20, 10 and 20 points; the last has two outliers on opposite
    # sides, at 103 and 97.  One refinement step moves the representative of the
    # small group (whose points then join the first, 50 away) onto the farther one:
    # a query 50 beyond it is left with that cluster of one point
    rng = np.random.default_rng(0)
    d = 9
    centre = np.zeros((72, d))
    centre[:20, 0] = 1e4
    centre[20:40, 1] = 1e4
    centre[40:50, 0], centre[40:50, 2] = 1e4, 50.0
    r = (centre + 0.01 * rng.standard_normal((72, d))).astype(np.float32)
    far, near = (71, 70) if swap else (70, 71)
    r[far] = r[near] = 0.0
    r[far, 3], r[near, 3] = 103.0, -97.0
    q = np.zeros((1, d), np.float32)
    q[0, 3] = 153.0
    groups = [0] * 20 + [1] * 20 + [2] * 10 + [3] * 20 + [9] * 2
    idx, _, st = knnjoin(q, r, 1, sreps=4, qreps=1, rep_trials=1, lloyd_iters=1,
                         seed=_seed(groups, 4), stats=True)
    assert idx.tolist() == [[far]]
    assert st.dist_evals == 1
