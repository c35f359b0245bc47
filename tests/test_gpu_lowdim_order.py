"""The brute force of point clouds on sets in every order: points that come ever nearer
enter the lists 128 at a time, the first ones of a set always do.  Sizes on every
side of the lines between its shapes (queries a warp, warps a query, splits).
Coordinates are small whole numbers, so distances are exact and many are equal: the
results have to equal the oracle's bit for bit."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4

# (ref_nb, query_nb, dim, k)
SIZES = [
    (129, 70, 2, 16), (999, 301, 1, 8), (1000, 299, 3, 7), (1001, 1199, 4, 16), (3001, 4999, 1, 9),
    (3001, 5001, 3, 16), (20000, 1201, 2, 8), (33000, 1300, 3, 8), (40001, 700, 1, 16),
    (140001, 301, 3, 5), (140003, 1201, 1, 1), (262145, 3900, 1, 8),
]
ORDERS = ["random", "near_last", "near_first", "blocks"]


def _arrange(order, ref, rng):
    if order in ("near_last", "near_first"):
        o = np.argsort(ref[0], kind="stable")
        return np.ascontiguousarray(ref[:, o if order == "near_last" else o[::-1]])
    if order == "blocks":   # runs of 100 equal points
        return np.ascontiguousarray(np.repeat(ref, 100, axis=1)[:, :ref.shape[1]])
    return ref


def _noalloc(knncuda, torch, r, x, k):
    d = torch.empty((k, x.shape[1]), device=x.device)
    i = torch.empty((k, x.shape[1]), dtype=torch.int32, device=x.device)
    rc = knncuda.lib().knnb200_knn_device_noalloc(
        r.data_ptr(), r.shape[1], r.stride(0), x.data_ptr(), x.shape[1], x.stride(0), r.shape[0],
        k, d.data_ptr(), i.data_ptr(), d.stride(0),
        ctypes.c_void_p(torch.cuda.current_stream(x.device).cuda_stream))
    assert rc == 0
    return d, i


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
def test_brute_force_in_any_order(knncuda, oracle, gpu, size, order):
    import torch

    n, q, dim, k = size
    rng = np.random.default_rng(n + q)
    ref = _arrange(order, rng.integers(0, 1000, (dim, n)).astype(np.float32), rng)
    query = rng.integers(0, 1400, (dim, q)).astype(np.float32)
    r = torch.zeros((dim, (n + 3) // 4 * 4), device=gpu)[:, :n]
    x = torch.zeros((dim, (q + 3) // 4 * 4), device=gpu)[:, :q]
    r.copy_(torch.from_numpy(ref))
    x.copy_(torch.from_numpy(query))
    d, i = _noalloc(knncuda, torch, r, x, k)
    few = slice(0, q) if n * q < 1e8 else slice(q // 3, q // 3 + 200)   # what the oracle does
    gt_d, gt_i = oracle.knn_c(ref, np.ascontiguousarray(query[:, few]), k, threads=THREADS)
    assert np.array_equal(d[:, few].cpu().numpy().view(np.uint32), gt_d.view(np.uint32))
    assert np.array_equal(i[:, few].cpu().numpy(), gt_i)
    sd, si = knncuda.knn_device(r, x, k, "global")
    assert torch.equal(sd, d) and torch.equal(si, i)
