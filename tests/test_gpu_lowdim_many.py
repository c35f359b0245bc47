"""Many queries against few points of few dimensions: one thread a pair of queries,
at the sizes where its tiles, pairs and lists end, and on either side of the line to
one warp a query.  Coordinates are small whole numbers, so every distance is exact
and equal ones abound: the results have to equal the oracle's bit for bit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4

# (ref_nb, query_nb, dim, k)
CASES = [
    (1, 10001, 1, 1), (5, 20000, 2, 5), (16, 12800, 3, 8), (16, 40001, 4, 16), (9, 30011, 4, 9),
    (31, 50003, 1, 16), (64, 99999, 3, 1), (127, 160000, 2, 8), (128, 300001, 3, 7),
    (255, 400000, 4, 8), (399, 600001, 1, 8), (511, 300003, 3, 8), (512, 300002, 2, 8),
    (513, 400001, 3, 6), (699, 800001, 3, 8), (701, 100001, 3, 8), (64, 2000, 3, 8),
    (128, 20000, 4, 16),
]


def _whole(seed, dim, n):
    return np.random.default_rng(seed).integers(0, 30, size=(dim, n)).astype(np.float32)


@pytest.mark.parametrize("case", CASES, ids=["x".join(map(str, c)) for c in CASES])
def test_few_points_equal_oracle(knncuda, oracle, gpu, case):
    n, q, dim, k = case
    ref, query = _whole(n, dim, n), _whole(q, dim, q)
    d, i = knncuda.knn(ref, query, k, "global")
    gt_d, gt_i = oracle.knn_c(ref, query, k, threads=THREADS)
    assert np.array_equal(d.view(np.uint32), gt_d.view(np.uint32))
    assert np.array_equal(i, gt_i)


def test_points_that_are_no_neighbours(knncuda, gpu):
    """Infinite and NaN distances: no neighbours, as in the warp kernel, whose answers
    for the same queries taken a few at a time these are."""
    import torch

    rng = np.random.default_rng(3)
    ref, query = rng.random((3, 40), dtype=np.float32), rng.random((3, 30000), dtype=np.float32)
    ref[1, ::3], ref[2, 1::7], query[0, 5::11] = np.nan, np.inf, 1e30
    r, x = torch.from_numpy(ref).to(gpu), torch.from_numpy(query).to(gpu)
    d, i = knncuda.knn_device(r, x, 16, "global")
    for c in range(0, 30000, 1000):
        xs = x[:, c:c + 1000].contiguous()
        ds, js = knncuda.knn_device(r, xs, 16, "global")
        assert torch.equal(d[:, c:c + 1000], ds) and torch.equal(i[:, c:c + 1000], js)
    assert bool((i == -1).any())
