"""knn_cublas where the preparation of the reference set splits the dimensions
among warps (512 padded dimensions and more): parts of unequal length, a padded
last one, sets that end inside a block, against the exact kernel bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(33000, 70, 449, 10), (32769, 33, 513, 20),
                                  (33333, 129, 577, 5), (40000, 20, 1023, 50)],
                         ids=lambda c: f"n{c[0]}q{c[1]}d{c[2]}k{c[3]}")
def test_split_preparation(knncuda, gpu, case):
    import torch

    n, q, dim, k = case
    gen = torch.Generator(device=gpu).manual_seed(n + dim)
    ref = torch.randn((dim, (n + 3) // 4 * 4), generator=gen, device=gpu)[:, :n]
    query = torch.randn((dim, (q + 3) // 4 * 4), generator=gen, device=gpu)[:, :q]
    d, i = knncuda.knn_device(ref, query, k, "cublas")
    torch.cuda.synchronize()
    assert knncuda.last_tc_stats()["candidates"] >= k * q
    gd, gi = knncuda.knn_device(ref, query, k, "global")
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy().view(np.uint32), gd.cpu().numpy().view(np.uint32))
    assert torch.equal(i, gi)
