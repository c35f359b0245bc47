"""The spatial search of point clouds (d <= 4) against the brute force.

knnb200_knn_device searches a large cloud in spatial order;
knnb200_knn_device_noalloc, which has no scratch for that, runs the brute-force
kernel.  Both return the k smallest (distance, index) keys, so their results
have to be equal bit for bit -- on uniform clouds and on what a grid handles
badly: clusters, duplicates, lattices (equal distances everywhere), flat and
constant clouds, outliers that stretch the grid so that nearly all points share
a cell (queries then go back to the brute force), points that are not finite.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(kind, rng, dim, n):
    x = rng.random((dim, n), dtype=np.float32)
    if kind == "clusters":
        c = rng.random((dim, 37), dtype=np.float32)
        x = c[:, rng.integers(0, 37, n)] + 1e-3 * rng.standard_normal((dim, n), dtype=np.float32)
    elif kind == "lattice":
        x = np.floor(x * 12)
    elif kind == "constant":
        x[:] = 0.25
    elif kind == "flat":
        x[0] = 1.5
        x *= np.float32(1e-3) if dim == 1 else 1
    elif kind == "outliers":
        x[:, rng.integers(0, n, 5)] = np.float32(1e6) * rng.standard_normal((dim, 5))
    elif kind == "huge":
        x = (x - np.float32(0.5)) * np.float32(3e38)   # distances overflow to inf
    elif kind == "nonfinite":
        bad = rng.integers(0, n, n // 50)
        x[rng.integers(0, dim, n // 50), bad] = rng.choice(
            np.array([np.nan, np.inf, -np.inf], np.float32), n // 50)
    return np.ascontiguousarray(x, dtype=np.float32)


CASES = [(kind, dim, k, n, q)
         for kind, n, q in (("uniform", 100003, 4100), ("clusters", 100003, 4100),
                            ("lattice", 50000, 8200), ("constant", 50000, 8200),
                            ("flat", 70001, 6000), ("outliers", 60000, 7001),
                            ("huge", 60000, 7001), ("nonfinite", 60000, 7001))
         for dim, k in ((1, 16), (2, 1), (3, 8), (4, 13))] + [("uniform", 3, 9, 1000, 400001),
                                                            ("uniform", 2, 16, 4000037, 101)]


@pytest.mark.parametrize("case", CASES, ids=["-".join(map(str, c)) for c in CASES])
def test_space_search_equals_brute_force(knncuda, gpu, case):
    import torch

    kind, dim, k, n, q = case
    rng = np.random.default_rng(n + dim)
    ref, query = _cloud(kind, rng, dim, n), _cloud(kind, rng, dim, q)
    r = torch.zeros((dim, (n + 3) // 4 * 4 + 8), device=gpu)[:, :n]
    x = torch.zeros((dim, (q + 3) // 4 * 4 + 4), device=gpu)[:, :q]
    r.copy_(torch.from_numpy(ref))
    x.copy_(torch.from_numpy(query))
    d, i = knncuda.knn_device(r, x, k, "global")
    bd, bi = torch.zeros_like(d), torch.zeros_like(i)
    step = 1 << 16   # the brute force's scratch holds so many queries
    for c in range(0, q, step):
        e = min(q, c + step)
        rc = knncuda.lib().knnb200_knn_device_noalloc(
            r.data_ptr(), n, r.stride(0), x.data_ptr() + 4 * c, e - c, x.stride(0), dim, k,
            bd.data_ptr() + 4 * c, bi.data_ptr() + 4 * c, bd.stride(0),
            ctypes.c_void_p(torch.cuda.current_stream(gpu).cuda_stream))
        assert rc == 0
    assert knncuda.sync_status() == 0
    assert torch.equal(d, bd) and torch.equal(i, bi)


def test_resident_cloud(knncuda, gpu):
    import torch

    rng = np.random.default_rng(3)
    r = torch.from_numpy(_cloud("uniform", rng, 3, 100000)).to(gpu)
    x = torch.from_numpy(_cloud("uniform", rng, 3, 5000)).to(gpu)
    torch.cuda.synchronize()
    rs = knncuda.RefSet(r)
    d, i = rs.knn(x, 8, "global")
    wd, wi = knncuda.knn_device(r, x, 8, "global")
    assert torch.equal(d, wd) and torch.equal(i, wi)
    rs.close()
