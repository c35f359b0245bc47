"""Requests for the FP8 scan on data that has no FP8 scale: a set of equal points, of
subnormal or non-finite coordinates, queries that are not finite or far out.  Such
a request runs as one for the BF16 scan, in every size range and on a resident set;
its answers are the exact kernel's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ["constant", "inf", "nan", "infinite_query", "nan_query", "far", "tiny", "subnormal",
         "huge"]
SIZES = [(16384, 4096, 128, 16), (40000, 300, 128, 16), (40000, 300, 384, 100)]


def _data(kind, n, q, dim):
    rng = np.random.default_rng(n + dim)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    if kind == "constant":
        ref[:] = 1
    elif kind in ("inf", "nan"):
        ref[3, 5] = np.float32(kind)
    elif kind in ("infinite_query", "nan_query"):
        query[1, 7] = np.float32("inf" if kind == "infinite_query" else "nan")
    elif kind == "far":
        query += 30000
    else:
        scale = np.float32({"tiny": 1e-30, "subnormal": 1e-41, "huge": 1e18}[kind])
        ref, query = ref * scale, query * scale
    return ref, query


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
def test_fp8_request(knncuda, gpu, size, kind):
    import torch

    n, q, dim, k = size
    r, x = (torch.from_numpy(a).to(gpu) for a in _data(kind, n, q, dim))
    wd, wi = knncuda.knn_device(r, x, k, "global")
    d, i = knncuda.knn_device(r, x, k, "fp8")
    assert knncuda.sync_status() == 0
    assert torch.equal(d.view(torch.int32), wd.view(torch.int32)) and torch.equal(i, wi)
    rs = knncuda.RefSet(r)
    try:
        d, i = rs.knn(x, k, "fp8")
        torch.cuda.synchronize()
    finally:
        rs.close()
    assert torch.equal(d.view(torch.int32), wd.view(torch.int32)) and torch.equal(i, wi)


@pytest.mark.parametrize("n,q,dim,k", [(16384, 4096, 128, 16), (32767, 2000, 64, 10)])
def test_small_sets_are_not_scanned_in_fp8(knncuda, gpu, n, q, dim, k):
    """Clusters whose candidates FP8's error bound does not tell apart."""
    import torch

    g = torch.Generator(device=gpu)
    g.manual_seed(n)
    centres = torch.randn((dim, 256), device=gpu, generator=g)
    centres /= centres.norm(dim=0, keepdim=True)

    def points(m):
        of = torch.randint(256, (32768,), device=gpu, generator=g)
        noise = torch.randn((dim, 32768), device=gpu, generator=g)
        return (centres[:, of] + 0.05 * noise)[:, :m]

    r, x = points(n), points(q)
    d, i = knncuda.knn_device(r, x, k, "fp8")
    assert knncuda.last_tc_kinds()[0] == "bf16"
    wd, wi = knncuda.knn_device(r, x, k, "global")
    assert torch.equal(d, wd) and torch.equal(i, wi)
