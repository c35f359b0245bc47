"""The item size that a batched plan chooses for batches of equal problems: given out to
the SMs, its items end no later than ones of 256 stages would."""
import pytest

pytestmark = pytest.mark.gpu

# (problems, ref_nb, query_nb, dim, k)
BATCHES = [(170, 24000, 64, 256, 10), (150, 48000, 64, 128, 10), (149, 20000, 64, 256, 10),
           (75, 30000, 128, 256, 10), (160, 65536, 64, 256, 32), (300, 16000, 64, 256, 64),
           (148, 20000, 64, 256, 10), (64, 4000, 192, 64, 10)]


@pytest.mark.parametrize("batch", BATCHES, ids=["x".join(map(str, b)) for b in BATCHES])
def test_waves_of_equal_items(knncuda, gpu, batch):
    import torch

    count, n, q, dim, k = batch
    r = torch.rand((dim, n), device=gpu)
    x = torch.rand((dim, q), device=gpu)
    outs = [(torch.empty((k, q), device=gpu), torch.empty((k, q), dtype=torch.int32, device=gpu))
            for _ in range(count)]
    problems = knncuda.problems_from([(r, x, k, d, i) for d, i in outs])
    sms = torch.cuda.get_device_properties(gpu).multi_processor_count
    stages = -(-n // 256) * -(-dim // 16) * (q // 64) * count   # of whole query tiles

    def ends(plan):
        items = plan.items()
        return -(-items // sms) * (stages / items + 14)   # 14: an item's own cost

    plan = knncuda.BatchedPlan(problems)
    plan256 = knncuda.BatchedPlan(problems, item_stages=256)
    assert ends(plan) <= 1.01 * ends(plan256), (plan.config(), plan.items(), plan256.items())
    plan.run()
    assert plan.status() == 0
    wd, wi = knncuda.knn_device(r, x, k, "global")
    for d, i in (outs[0], outs[-1]):
        assert torch.equal(d, wd) and torch.equal(i, wi)
