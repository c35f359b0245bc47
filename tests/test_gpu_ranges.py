"""The fused exact kernel where it cuts the tiles of all query tiles into one
range a CTA: ranges that hold parts of two and of three query tiles, of one tile
and of many, last tiles with one point and last query tiles with one query, lists
of every size, and a last stage that is short.

Coordinates are small whole numbers, so every distance is exact in FP32 and in
the oracle alike: the results have to equal the oracle's bit for bit, indices
included (equal distances in the order of the indices).
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4

# (ref_nb, query_nb, dim, k): each is one that 148 SMs run by ranges
CASES = [
    (1025, 9473, 20, 1), (1025, 9473, 100, 128), (1024, 5001, 250, 33), (1154, 9480, 64, 64),
    (16384, 4096, 128, 16), (46859, 1398, 128, 5),
]


def _whole(seed, dim, n):
    return np.random.default_rng(seed).integers(0, 9, size=(dim, n)).astype(np.float32)


@pytest.mark.parametrize("case", CASES, ids=[f"n{c[0]}q{c[1]}d{c[2]}k{c[3]}" for c in CASES])
def test_ranges_equal_oracle(knncuda, oracle, gpu, case):
    n, q, dim, k = case
    ref, query = _whole(n + k, dim, n), _whole(n + k + 1, dim, q)
    d, i = knncuda.knn(ref, query, k, "global")
    gt_d, gt_i = oracle.knn_c(ref, query, k, threads=THREADS)
    assert np.array_equal(d.view(np.uint32), gt_d.view(np.uint32))
    assert np.array_equal(i, gt_i)


def test_ranges_pitched(knncuda, oracle, gpu):
    """Row pitches of both sets and of the outputs."""
    import torch

    n, q, dim, k = 1030, 9473, 36, 30
    ref, query = _whole(7, dim, n), _whole(8, dim, q)
    r = torch.zeros((dim, 1040), device=gpu)[:, :n]
    r.copy_(torch.from_numpy(ref))
    x = torch.zeros((dim, 9500), device=gpu)[:, :q]
    x.copy_(torch.from_numpy(query))
    dist = torch.full((k, 9600), -1.0, device=gpu)
    index = torch.full((k, 9600), -1, dtype=torch.int32, device=gpu)
    knncuda.knn_device(r, x, k, "global", dist=dist[:, :q], index=index[:, :q])
    torch.cuda.synchronize()
    gt_d, gt_i = oracle.knn_c(ref, query, k, threads=THREADS)
    assert np.array_equal(dist[:, :q].cpu().numpy().view(np.uint32), gt_d.view(np.uint32))
    assert np.array_equal(index[:, :q].cpu().numpy(), gt_i)
    assert bool((dist[:, q:] == -1).all()) and bool((index[:, q:] == -1).all())


def test_resident_set_without_room_for_the_lists(knncuda, oracle, gpu):
    """A slot's scratch has no room for two lists of 100 keys a query beside this
    little query set: the grid runs, which needs none."""
    import torch

    n, q, dim, k = 1025, 9473, 20, 100
    ref, query = _whole(9, dim, n), _whole(10, dim, q)
    rs = knncuda.RefSet(ref)
    x = torch.zeros((dim, 9476), device=gpu)[:, :q]
    x.copy_(torch.from_numpy(query))
    d, i = rs.knn(x, k, "global")
    torch.cuda.synchronize()
    gt_d, gt_i = oracle.knn_c(ref, query, k, threads=THREADS)
    assert np.array_equal(d.cpu().numpy().view(np.uint32), gt_d.view(np.uint32))
    assert np.array_equal(i.cpu().numpy(), gt_i)
