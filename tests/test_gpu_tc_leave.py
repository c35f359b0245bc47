"""knn_cublas on sets below 32768 points whose data defeats the candidate lists (equal
or nearly equal points, coordinates that overflow, vanish or are not finite, queries
far away): the call goes to the exact kernel after the threshold sample, without the
scans.  With few such queries it stays on the tensor path.  The answers are the
exact kernel's bit for bit either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (ref_nb, query_nb, dim, k)
SIZES = [(16384, 4096, 128, 16), (4096, 8192, 512, 10), (12300, 7001, 260, 256),
         (32767, 3001, 64, 10)]
KINDS = ["constant", "zeros", "far", "tiny", "huge", "inf", "nan"]


def _data(kind, n, q, dim):
    rng = np.random.default_rng(n + dim)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    if kind == "constant":
        ref[:] = 1
    elif kind == "zeros":
        ref[:, rng.permutation(n)[:n // 2]] = 0
        query[:] = 0
    elif kind == "far":
        query += 30000
    elif kind in ("tiny", "huge"):
        scale = np.float32(1e-30 if kind == "tiny" else 1e18)
        ref, query = ref * scale, query * scale
    elif kind in ("inf", "nan"):
        ref[3, 5] = np.float32(kind)
    return ref, query


def _tensors(gpu, *arrays):
    import torch

    out = []
    for a in arrays:
        t = torch.zeros((a.shape[0], (a.shape[1] + 3) // 4 * 4), device=gpu)[:, :a.shape[1]]
        t.copy_(torch.from_numpy(a))
        out.append(t)
    return out


def _equal(torch, got, want):
    return all(torch.equal(g.view(torch.int32), w.view(torch.int32)) for g, w in zip(got, want))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
def test_data_that_defeats_the_lists(knncuda, gpu, size, kind):
    import torch

    n, q, dim, k = size
    ref, query = _data(kind, n, q, dim)
    r, x = _tensors(gpu, ref, query)
    want = knncuda.knn_device(r, x, k, "global")
    got = knncuda.knn_device(r, x, k, "cublas")
    stats = knncuda.last_tc_stats()
    assert knncuda.sync_status() == 0
    assert stats["second_scan"] == 0 and stats["exact"] == q
    assert knncuda.last_tc_kinds() == (None, None)
    assert _equal(torch, got, want)
    d, i = knncuda.knn(ref, query, k, "cublas")
    assert np.array_equal(d.view(np.int32), want[0].cpu().numpy().view(np.int32))
    assert np.array_equal(i, want[1].cpu().numpy())


@pytest.mark.parametrize("share", [0.0, 0.0003, 0.02, 0.04, 0.06, 0.5])
def test_some_queries_that_defeat_them(knncuda, gpu, share):
    import torch

    n, q, dim, k = 16384, 4096, 128, 32
    rng = np.random.default_rng(17)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    ref[:, rng.permutation(n)[:n // 2]] = 0
    query[:, rng.permutation(q)[:int(q * share)]] = 0
    r, x = _tensors(gpu, ref, query)
    want = knncuda.knn_device(r, x, k, "global")
    got = knncuda.knn_device(r, x, k, "cublas")
    stats = knncuda.last_tc_stats()
    # (more than 4.8 % of the queries end a call of this size)
    assert (stats["exact"] == q) == (share > 0.05)
    assert share > 0.05 or stats["exact"] == int(q * share)
    assert _equal(torch, got, want)
