"""Batched plans whose item size is left open, of small batches (items of 64
stages and more) and larger ones, with query sets that leave whole warps of a
query tile without a query, against the same plan with items of 256 stages and
the oracle: whole-number coordinates, so every bit has to be equal."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4

BATCHES = {
    "one": [(30000, 65, 40, 9)],
    "small": [(5000, q, 33, k) for q, k in ((1, 5), (4, 64), (5, 1), (63, 33), (129, 20))],
    "even": [(4000, 200, 64, 10)] * 40,
    "large": [(20000, 700, 64, 30)] * 20,
}


@pytest.mark.parametrize("name", list(BATCHES))
def test_item_size_left_open(knncuda, oracle, gpu, name):
    import torch

    rng = np.random.default_rng(3)
    sets, tables, outs = [], [[], []], [[], []]
    for n, q, dim, k in BATCHES[name]:
        ref = rng.integers(0, 9, size=(dim, n)).astype(np.float32)
        query = rng.integers(0, 9, size=(dim, q)).astype(np.float32)
        r = torch.zeros((dim, (n + 3) // 4 * 4), device=gpu)[:, :n]
        x = torch.zeros((dim, (q + 3) // 4 * 4), device=gpu)[:, :q]
        r.copy_(torch.from_numpy(ref))
        x.copy_(torch.from_numpy(query))
        sets.append((ref, query, k, r, x))
        for table, out in zip(tables, outs):
            d = torch.empty((k, q), device=gpu)
            i = torch.empty((k, q), dtype=torch.int32, device=gpu)
            table.append((r, x, k, d, i))
            out.append((d, i))
    arrays = [knncuda.problems_from(t) for t in tables]
    plans = [knncuda.BatchedPlan(arrays[0]), knncuda.BatchedPlan(arrays[1], item_stages=256)]
    for plan in plans:
        plan.run()
        assert plan.status() == 0
    for j, ((d, i), (d256, i256)) in enumerate(zip(*outs)):
        assert torch.equal(d, d256) and torch.equal(i, i256)
        if j < 5:
            ref, query, k = sets[j][:3]
            gt_d, gt_i = oracle.knn_c(ref, query, k, threads=THREADS)
            assert np.array_equal(d.cpu().numpy().view(np.uint32), gt_d.view(np.uint32))
            assert np.array_equal(i.cpu().numpy(), gt_i)
