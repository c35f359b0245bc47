"""The first host calls of a process: small ones before the staging buffers exist, those
that bring them, and larger ones that outgrow them.  Each answer is the device
entry's bit for bit.  (In a process of its own: the buffers stay once they are there.)"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import sys
sys.path.insert(0, {pkg!r})
import numpy as np, torch
import knncuda
rng = np.random.default_rng(1)
for n, q, dim, k, method in [{calls}]:
    ref, query = rng.random((dim, n), dtype=np.float32), rng.random((dim, q), dtype=np.float32)
    r = torch.zeros((dim, (n + 3) // 4 * 4), device="cuda")[:, :n]
    x = torch.zeros((dim, (q + 3) // 4 * 4), device="cuda")[:, :q]
    r.copy_(torch.from_numpy(ref))
    x.copy_(torch.from_numpy(query))
    wd, wi = knncuda.knn_device(r, x, k, "global")
    wd, wi = wd.cpu().numpy(), wi.cpu().numpy()
    d, i = knncuda.knn(ref, query, k, method)
    assert np.array_equal(d, wd) and np.array_equal(i, wi), (n, q, dim)
print("calls ok")
"""

SMALL = "(8192, 1000, 64, 10, 'cublas'), (16384, 4096, 128, 16, 'cublas')"
LARGE = "(262147, 300, 70, 10, 'cublas'), (100003, 500, 300, 10, 'global')"


@pytest.mark.parametrize("calls", [
    ", ".join([SMALL] * 12 + [LARGE] + [SMALL]),   # grow, then outgrow
    ", ".join([LARGE, SMALL, LARGE, LARGE, SMALL]),
    ", ".join(["(9001, 30011, 33, 5, 'global'), (3000, 5000, 100, 3, 'global')"] * 10 + [LARGE]),
], ids=["small_first", "large_first", "queries"])
def test_first_calls(gpu, calls):
    run = subprocess.run(
        [sys.executable, "-c", SCRIPT.format(pkg=os.path.join(ROOT, "knn-cuda_b200"), calls=calls)],
        capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "calls ok" in run.stdout, run.stdout + run.stderr
