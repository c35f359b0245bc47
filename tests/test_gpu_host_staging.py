"""Host entries on pageable arrays large enough for the staging buffers: many and
few rows, ragged lengths, more than one buffer's worth, a set whose threshold
sample is many short runs.  The answers are the device entry's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # (ref_nb, query_nb, dim, k, method)
    (400003, 300, 3, 4, "global"), (65537, 40, 70, 5, "global"), (9, 5, 70001, 3, "global"),
    (300001, 262147, 1, 2, "global"), (16385, 4099, 129, 16, "cublas"),
    (262147, 4100, 40, 10, "cublas"), (300005, 70, 100, 33, "cublas"),
]


@pytest.mark.parametrize("case", CASES, ids=["-".join(map(str, c)) for c in CASES])
def test_pageable_input(knncuda, gpu, case):
    import torch

    n, q, dim, k, method = case
    rng = np.random.default_rng(n)
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    r = torch.zeros((dim, (n + 3) // 4 * 4), device=gpu)[:, :n]
    x = torch.zeros((dim, (q + 3) // 4 * 4), device=gpu)[:, :q]
    r.copy_(torch.from_numpy(ref))
    x.copy_(torch.from_numpy(query))
    wd, wi = knncuda.knn_device(r, x, k, "global")
    for _ in range(2):   # the buffers are reused
        d, i = knncuda.knn(ref, query, k, method)
        assert np.array_equal(d, wd.cpu().numpy()) and np.array_equal(i, wi.cpu().numpy())


def test_host_call_waits_for_a_device_call_in_flight(knncuda, gpu):
    """The host and device entries share the workspace's scratch: a host call made
    while a device call still runs on another stream must not touch it."""
    import torch

    rng = np.random.default_rng(9)
    n, q, dim, k = 16385, 4099, 129, 16
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    r = torch.zeros((dim, (n + 3) // 4 * 4), device=gpu)[:, :n]
    x = torch.zeros((dim, (q + 3) // 4 * 4), device=gpu)[:, :q]
    r.copy_(torch.from_numpy(ref))
    x.copy_(torch.from_numpy(query))
    want = [t.cpu() for t in knncuda.knn_device(r, x, k, "global")]
    knncuda.knn(ref, query, k, "cublas")   # the buffers have their sizes now
    side = torch.cuda.Stream()
    for method in ("cublas", "global") * 5:
        with torch.cuda.stream(side):
            outs = [knncuda.knn_device(r, x, k, "global") for _ in range(4)]
        d, i = knncuda.knn(ref, query, k, method)
        torch.cuda.synchronize()
        assert np.array_equal(d, want[0].numpy()) and np.array_equal(i, want[1].numpy())
        for dd, ii in outs:
            assert torch.equal(dd.cpu(), want[0]) and torch.equal(ii.cpu(), want[1])
