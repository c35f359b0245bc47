"""The exact path on scratch that was sized for more queries than a call has left:
a plan for few queries may cut the reference set into more ranges, and so ask for
more lists, than the plan for many did.  The lists are then as many as fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tensors(gpu, *arrays):
    import torch

    out = []
    for a in arrays:
        t = torch.zeros((a.shape[0], (a.shape[1] + 3) // 4 * 4), device=gpu)[:, :a.shape[1]]
        t.copy_(torch.from_numpy(a))
        out.append(t)
    return out


@pytest.mark.parametrize("share", [0.9, 0.93, 0.955, 0.982, 0.995])
@pytest.mark.parametrize("n,q", [(16384, 4096), (40000, 4096), (40000, 2600), (33000, 9300)])
def test_queries_left_over_by_the_tensor_path(knncuda, gpu, n, q, share):
    """More points at one place than a candidate list holds, and most queries there:
    both scans leave those queries to the exact kernel, in the call's scratch."""
    import torch

    dim, k, at = 128, 100, 5000
    rng = np.random.default_rng(q)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    ref[:, rng.permutation(n)[:at]] = 0
    query[:, rng.permutation(q)[:int(q * share)]] = 0
    r, x = _tensors(gpu, ref, query)
    knncuda.lib().knnb200_release_workspace()   # scratch of this call's size, no larger
    d, i = knncuda.knn_device(r, x, k, "cublas")
    assert knncuda.sync_status() == 0
    wd, wi = knncuda.knn_device(r, x, k, "global")
    assert torch.equal(d, wd) and torch.equal(i, wi)


@pytest.mark.parametrize("last", [900, 300, 64, 17, 1])
@pytest.mark.parametrize("k", [100, 300])
def test_small_last_chunk_under_a_memory_cap(knncuda, gpu, k, last):
    n, dim, chunk = 2000, 32, 8448
    q = chunk + last
    rng = np.random.default_rng(last)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    want_d, want_i = knncuda.knn(ref, query, k, "global")
    knncuda.lib().knnb200_release_workspace()
    knncuda.set_memory_cap(knncuda.call_bytes(n, chunk, dim, k, "global", host=True))
    try:
        d, i = knncuda.knn(ref, query, k, "global")
        assert knncuda.last_query_chunks() >= 2
    finally:
        knncuda.set_memory_cap(0)
    assert np.array_equal(d.view(np.uint32), want_d.view(np.uint32))
    assert np.array_equal(i, want_i)


@pytest.mark.parametrize("n,dim,chunk,last", [(9385, 4, 237568, 2), (7955, 4, 232704, 67),
                                              (7970, 3, 302592, 38)])
def test_small_last_chunk_of_a_point_cloud(knncuda, gpu, n, dim, chunk, last):
    """The large chunk needs no lists at all, the last one would like two a query."""
    k, q = 1, chunk + last
    rng = np.random.default_rng(last)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    want_d, want_i = knncuda.knn(ref, query, k, "global")
    knncuda.lib().knnb200_release_workspace()
    knncuda.set_memory_cap(knncuda.call_bytes(n, chunk, dim, k, "global", host=True))
    try:
        d, i = knncuda.knn(ref, query, k, "global")
        assert knncuda.last_query_chunks() == 2
    finally:
        knncuda.set_memory_cap(0)
    assert np.array_equal(d.view(np.uint32), want_d.view(np.uint32))
    assert np.array_equal(i, want_i)
