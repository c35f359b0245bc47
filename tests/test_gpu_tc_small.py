"""knn_cublas on sets below 32768 points that take the tensor path: sizes at the
edges of what it accepts there (256 sample rows), ragged ones, and data whose
candidate lists overflow.  The answers equal the exact kernel's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # (ref_nb, query_nb, dim, k, data)
    (4096, 8192, 512, 10, "uniform"), (4097, 9001, 300, 33, "uniform"),
    (8191, 4099, 256, 102, "uniform"), (8200, 6003, 300, 103, "uniform"),
    (12300, 7000, 260, 256, "uniform"), (20000, 5000, 40, 17, "uniform"),
    (32767, 1500, 96, 100, "uniform"), (16384, 4096, 128, 16, "clusters"),
    (16000, 4100, 128, 16, "duplicates"), (9000, 4100, 200, 20, "far"),
]


def _points(kind, rng, dim, n, base):
    x = rng.random((dim, n), dtype=np.float32)
    if kind == "clusters":
        x = base[:, rng.integers(0, base.shape[1], n)] * 2 - 1
        x = x + np.float32(0.05) * rng.standard_normal((dim, n), dtype=np.float32)
    elif kind == "duplicates":
        x = base[:, rng.integers(0, base.shape[1], n)]
    elif kind == "far":
        x = base[:, rng.integers(0, 4, n)] * 20
        x = x + np.float32(0.01) * rng.standard_normal((dim, n), dtype=np.float32)
    return np.ascontiguousarray(x, dtype=np.float32)


@pytest.mark.parametrize("case", CASES, ids=["-".join(map(str, c)) for c in CASES])
def test_small_sets_on_the_tensor_path(knncuda, gpu, case):
    import torch

    n, q, dim, k, kind = case
    rng = np.random.default_rng(n + q)
    base = rng.random((dim, 50), dtype=np.float32)
    ref, query = _points(kind, rng, dim, n, base), _points(kind, rng, dim, q, base)
    r = torch.zeros((dim, (n + 3) // 4 * 4), device=gpu)[:, :n]
    x = torch.zeros((dim, (q + 3) // 4 * 4), device=gpu)[:, :q]
    r.copy_(torch.from_numpy(ref))
    x.copy_(torch.from_numpy(query))
    dg, ig = knncuda.knn_device(r, x, k, "global")
    dc, ic = knncuda.knn_device(r, x, k, "cublas")
    # the tensor path ran (20000 x 5000 x 40 is left to the exact kernel: at 338 us
    # against 296 by its models the gain is too small)
    assert (knncuda.last_tc_stats()["candidates"] > 0) == (dim != 40)
    assert knncuda.sync_status() == 0
    assert torch.equal(dc, dg) and torch.equal(ic, ig)
    dh, ih = knncuda.knn(ref, query, k, "cublas")
    assert np.array_equal(dh, dg.cpu().numpy()) and np.array_equal(ih, ig.cpu().numpy())


def test_small_set_under_a_memory_cap_runs_as_before(knncuda, gpu):
    """Where the tensor path's memory would not fit, a small set takes the exact
    kernel in one go."""
    rng = np.random.default_rng(5)
    n, q, dim, k = 16384, 4096, 128, 16
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    want_d, want_i = knncuda.knn(ref, query, k, "cublas")
    assert knncuda.last_tc_stats()["candidates"] > 0
    knncuda.set_memory_cap(knncuda.call_bytes(n, q, dim, k, "global", host=True))
    try:
        d, i = knncuda.knn(ref, query, k, "cublas")
        assert knncuda.last_query_chunks() == 1 and knncuda.last_tc_stats()["candidates"] == 0
    finally:
        knncuda.set_memory_cap(0)
    assert np.array_equal(d, want_d) and np.array_equal(i, want_i)
