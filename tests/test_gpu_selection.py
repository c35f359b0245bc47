"""Selection of the fused exact kernel at its edges: k at and around the
sizes of its lists, sets that end inside a tile or hold fewer points than one,
many equal distances (more than a query's buffer holds), and the merges of many
split lists by one and by eight warps.

Coordinates are small whole numbers, so every distance is exact in FP32 and in
the oracle alike: the results have to equal the oracle's bit for bit, indices
included (equal distances in the order of the indices).
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4

CASES = [
    # (ref_nb, query_nb, dim, k, coordinates 0 .. values - 1)
    (31, 3, 5, 31, 4), (128, 65, 6, 128, 3), (255, 7, 5, 32, 50), (256, 7, 5, 33, 50),
    (257, 64, 17, 64, 50), (3000, 70, 16, 65, 9), (3000, 63, 16, 128, 9), (4096, 33, 16, 129, 9),
    (4097, 33, 16, 256, 9), (700, 5, 6, 300, 3), (5000, 66, 5, 32, 1), (5000, 9, 5, 200, 1),
    (6000, 40, 8, 16, 2), (6000, 40, 8, 100, 2),
    (60000, 5, 8, 10, 30), (60000, 5, 8, 50, 30), (60000, 3, 8, 100, 30), (60000, 3, 8, 200, 30),
    (60000, 1500, 8, 40, 30),
    # up to 16 and up to 32 queries: smaller query tiles
    (3000, 16, 9, 50, 9), (3000, 17, 9, 30, 9), (5000, 32, 40, 120, 9), (60000, 30, 8, 64, 30),
    (700, 1, 5, 128, 4),
]


def _whole(seed, dim, n, values):
    return np.random.default_rng(seed).integers(0, values, size=(dim, n)).astype(np.float32)


@pytest.mark.parametrize("case", CASES, ids=[f"n{c[0]}q{c[1]}d{c[2]}k{c[3]}v{c[4]}" for c in CASES])
def test_selection_equals_oracle(knncuda, oracle, gpu, case):
    n, q, dim, k, values = case
    ref, query = _whole(n + k, dim, n, values), _whole(n + k + 1, dim, q, values)
    d, i = knncuda.knn(ref, query, k, "global")
    gt_d, gt_i = oracle.knn_c(ref, query, k, threads=THREADS)
    assert np.array_equal(d.view(np.uint32), gt_d.view(np.uint32))
    assert np.array_equal(i, gt_i)


def test_batched_queries_in_place_and_copied(knncuda, oracle, gpu):
    """One plan with query sets that TMA reads in place and ones it cannot (an
    odd row pitch, a base that is not a multiple of 16 bytes)."""
    import torch

    shapes = [(700, 33, 20, 9, 36, 0), (1500, 65, 16, 40, 65, 0), (900, 10, 33, 64, 16, 1),
              (300, 128, 7, 5, 128, 0)]
    table, want = [], []
    for j, (n, q, dim, k, pitch, shift) in enumerate(shapes):
        ref, query = _whole(j, dim, n, 40), _whole(50 + j, dim, q, 40)
        r = torch.zeros((dim, (n + 3) // 4 * 4), device=gpu)[:, :n]
        x = torch.zeros(dim * pitch + 4, device=gpu)[shift:shift + dim * pitch].view(dim, pitch)
        r.copy_(torch.from_numpy(ref))
        x = x[:, :q]
        x.copy_(torch.from_numpy(query))
        table.append((r, x, k, torch.empty((k, q), device=gpu),
                      torch.empty((k, q), dtype=torch.int32, device=gpu)))
        want.append(oracle.knn_c(ref, query, k, threads=THREADS))
    plan = knncuda.BatchedPlan(knncuda.problems_from(table))
    plan.run()
    assert plan.status() == 0
    for (_, _, _, d, i), (gt_d, gt_i) in zip(table, want):
        assert np.array_equal(d.cpu().numpy().view(np.uint32), gt_d.view(np.uint32))
        assert np.array_equal(i.cpu().numpy(), gt_i)
    plan.close()
