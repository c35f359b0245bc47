"""Point clouds of which the spatial search answers some queries and leaves others to
the brute force, and a resident one against the allocation-free entry, which has no
scratch for a search."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,k", [(1, 16), (2, 1), (3, 8), (4, 13)])
@pytest.mark.parametrize("inside", [1, 31, 500, 3500, 7000])
def test_queries_left_to_the_brute_force(knncuda, oracle, gpu, dim, k, inside):
    """A fifth of the points in a blob smaller than a grid cell: they are stored in no
    spatial order, so each of the blob's 375 leaves covers it, and a query inside it
    meets more leaves than a search may scan (256); those far from it a few.  The
    former, any number of them, are answered by the brute force, in whose splits the
    reference set is cut by that number."""
    import torch

    n, q = 60000, 7000
    rng = np.random.default_rng(dim * 10000 + inside)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    query[0] += 1.5   # beyond the cloud
    blob = rng.permutation(n)[:n // 5]
    ref[:, blob] = np.float32(1e-6) * rng.random((dim, n // 5), dtype=np.float32)
    at = rng.permutation(q)[:inside]
    query[:, at] = np.float32(1e-6) * rng.random((dim, inside), dtype=np.float32)
    r, x = torch.from_numpy(ref).to(gpu), torch.from_numpy(query).to(gpu)
    d, i = knncuda.knn_device(r, x, k, "global")
    assert knncuda.sync_status() == 0
    bd, bi = torch.empty_like(d), torch.empty_like(i)
    rc = knncuda.lib().knnb200_knn_device_noalloc(
        r.data_ptr(), n, n, x.data_ptr(), q, q, dim, k, bd.data_ptr(), bi.data_ptr(), q,
        ctypes.c_void_p(torch.cuda.current_stream(gpu).cuda_stream))
    assert rc == 0
    assert torch.equal(d, bd) and torch.equal(i, bi)
    some = np.concatenate([at[:40], rng.permutation(q)[:40]])
    gt_d, gt_i = oracle.knn_c(ref, np.ascontiguousarray(query[:, some]), k,
                              threads=os.cpu_count() or 4)
    assert np.allclose(d.cpu().numpy()[:, some], gt_d, rtol=1e-6, atol=0)


@pytest.mark.parametrize("n,q,dim,k", [(100000, 5000, 3, 8), (4000036, 132, 2, 16)])
def test_resident_cloud_equals_brute_force(knncuda, gpu, n, q, dim, k):
    import torch

    rng = np.random.default_rng(3)
    r = torch.from_numpy(rng.random((dim, n), dtype=np.float32)).to(gpu)
    x = torch.from_numpy(rng.random((dim, q), dtype=np.float32)).to(gpu)
    assert knncuda.plan_route(n, q, dim, k) == "cloud_space"
    rs = knncuda.RefSet(r)
    d, i = rs.knn(x, k, "global")
    bd, bi = torch.empty_like(d), torch.empty_like(i)
    rc = knncuda.lib().knnb200_knn_device_noalloc(
        r.data_ptr(), n, n, x.data_ptr(), q, q, dim, k, bd.data_ptr(), bi.data_ptr(), q,
        ctypes.c_void_p(torch.cuda.current_stream(gpu).cuda_stream))
    assert rc == 0
    assert torch.equal(d, bd) and torch.equal(i, bi)
    rs.close()
