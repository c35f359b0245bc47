"""The GPU tests of a kernel or a search have to reach it: their sizes, by the plan they
get on 148 SMs (which a machine without a GPU assumes)."""
import pytest

import test_gpu_lowdim_many
import test_gpu_lowdim_order
import test_gpu_ranges
import test_gpu_space


@pytest.mark.parametrize("case", test_gpu_ranges.CASES + [(1030, 9473, 36, 30),
                                                          (1025, 9473, 20, 100)])
def test_ranges(knncuda, case):
    assert knncuda.plan_route(*case) == "ranges"


def test_space(knncuda):
    for kind, dim, k, n, q in test_gpu_space.CASES:
        # (101 queries are too few for 4 million points; 131 are searched in space)
        q = 131 if n > 4000000 else q
        assert knncuda.plan_route(n, q, dim, k) == "cloud_space", (kind, n, q, dim, k)
    assert knncuda.plan_route(100000, 5000, 3, 8) == "cloud_space"
    for dim, k in ((1, 16), (2, 1), (3, 8), (4, 13)):
        assert knncuda.plan_route(60000, 7000, dim, k) == "cloud_space"


def test_brute_force(knncuda):
    routes = [knncuda.plan_route(*c) for c in test_gpu_lowdim_many.CASES]
    assert routes.count("cloud_thread") >= 12 and routes.count("cloud_warp") >= 2
    routes = [knncuda.plan_route(*c) for c in test_gpu_lowdim_order.SIZES]
    assert routes.count("cloud_warp") >= 8


def test_others(knncuda):
    assert knncuda.plan_route(16384, 4096, 5, 16) in ("grid", "ranges")
    assert knncuda.plan_route(1000, 16, 32, 10) == "grid"
    assert knncuda.plan_route(1000, 16, 3, 17) == "grid"
    assert knncuda.plan_route(10, 16, 3, 11) is None
