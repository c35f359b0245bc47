"""The calls that users of this library make, as cases that can be timed and checked.

A case names an entry point of the Python interface (``knn-cuda_b200/knncuda.py``) and a size:

* ``device``  ``knn_device`` on tensors that are on the GPU already,
* ``host``    ``knn_cuda_global`` / ``knn_cublas`` on numpy arrays, the call that replaces the
              reference's functions in a program of its users,
* ``serve``   ``RefSet.knn``: queries against a set that stays resident,
* ``batch``   ``BatchedPlan.run``: many small problems of uneven sizes in one launch.

``method`` is the caller's choice between the direct FP32 form ("global") and the expansion form
on the tensor cores ("cublas").  Points are ``dim x n``, row-major; ``uniform`` draws U[0,1), and
``mixture`` draws Gaussian clusters (``centres`` of them, unit length or in [-1,1]^dim).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "knn-cuda_b200"))
import knncuda  # noqa: E402
import workloads  # noqa: E402

DEV = "cuda:0"


def _case(kind, method, n, q, d, k, dist="uniform", centres=0, sigma=0.0, unit=True):
    return {"kind": kind, "method": method, "ref_nb": n, "query_nb": q, "dim": d, "k": k,
            "dist": dist, "centres": centres, "sigma": sigma, "unit": unit}


def listed():
    cases = {
        # a few points matched against a small set: launches and host work are all there is
        "small_global": _case("device", "global", 1000, 16, 32, 10),
        # the default problem of the reference's test program, descriptors of one image
        # matched against another's: on the device, and as the program itself calls it
        "readme_global": _case("device", "global", 16384, 4096, 128, 16),
        "readme_host_cublas": _case("host", "cublas", 16384, 4096, 128, 16),
        # neighbours in a 3-D point cloud
        "cloud3_global": _case("device", "global", 1 << 20, 65536, 3, 8),
        # clustered descriptors with many near-ties, on the device and from host arrays
        "mixture128_cublas": _case("device", "cublas", 262144, 16384, 128, 32, "mixture", 256,
                                   0.05, False),
        "mixture128_host_cublas": _case("host", "cublas", 262144, 16384, 128, 32, "mixture", 256,
                                        0.05, False),
        # a million embeddings, k = 100: both forms (the largest problem of the benchmark)
        "mixture256_cublas": _case("device", "cublas", 1 << 20, 16384, 256, 100, "mixture", 1024,
                                   0.1),
        "mixture256_global": _case("device", "global", 1 << 20, 16384, 256, 100, "mixture", 1024,
                                   0.1),
        # high dimension, ragged sizes
        "highdim_cublas": _case("device", "cublas", 100003, 2001, 768, 20, "mixture", 1024, 0.05),
        # a request loop against a resident set: a request of few queries, and a full batch
        "serve_few_cublas": _case("serve", "cublas", 2097152, 13, 128, 10, "mixture", 2048, 0.1),
        "serve_batch_cublas": _case("serve", "cublas", 2097152, 1024, 128, 100, "mixture", 2048,
                                    0.1),
        # 512 independent problems of uneven sizes in one launch
        "batch512": dict(_case("batch", "global", 65536, 2048, 256, 64), count=512, shapes=5),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _points(rng, dim):
    """The distribution of a drawn case."""
    if dim <= 4 or rng.random() < 0.4:
        return {"dist": "uniform", "centres": 0, "sigma": 0.0, "unit": True}
    return {"dist": "mixture", "centres": _log(rng, 64, 2048), "unit": rng.random() < 0.7,
            "sigma": round(rng.uniform(0.05, 1.6 / math.sqrt(dim)) if dim < 256 else 0.05, 3)}


def draw(rng):
    kind = rng.choice(["cloud", "global", "global", "cublas", "cublas", "host", "serve", "batch"])
    if kind == "cloud":
        # point clouds and other sets of few coordinates
        d, k = rng.randint(1, 4), rng.randint(1, 16)
        return dict(_case("device", rng.choice(["global", "cublas"]), _log(rng, 1000, 1 << 20),
                          _log(rng, 16, 65536), d, k))
    if kind == "batch":
        # uneven problems as the benchmark's: 1k-64k points, 16-2048 queries, k to 64
        return dict(_case("batch", "global", 65536, 2048, 256, 64), count=rng.randint(16, 512),
                    shapes=rng.randint(1, 1 << 20))
    if kind == "serve":
        d = rng.randint(32, 256)
        c = _case("serve", "cublas", _log(rng, 1 << 16, 1 << 21), _log(rng, 1, 1024), d,
                  rng.choice([10, 50, 100]))
        return dict(c, **_points(rng, d))
    d = _log(rng, 5 if kind == "global" else 16, 1024)
    n, q = _log(rng, 1000 if kind == "global" else 8192, 1 << 20), _log(rng, 1, 16384)
    if kind == "host":
        n = min(n, max(1000, (1 << 25) // d))
    # no more work than the largest listed case
    most = 1 << (40 if kind == "global" else 41)
    q = max(1, min(q, most // (n * d)))
    k = _log(rng, 1, 300) if kind == "global" else _log(rng, 1, 256)
    c = _case("host" if kind == "host" else "device",
              rng.choice(["global", "cublas"]) if kind == "host" else kind, n, q, d, k)
    return dict(c, **_points(rng, d))


def _generate(case, gen, centres, n, dim):
    """dim x n points on the GPU, the rows 16-byte aligned (a pitch of a multiple of 4)."""
    pitch = (n + 3) // 4 * 4
    x = torch.empty((dim, pitch), device=DEV)
    if case["dist"] == "uniform":
        x.uniform_(generator=gen)
    else:
        x.normal_(std=case["sigma"], generator=gen)
        of = torch.randint(case["centres"], (pitch,), generator=gen, device=DEV)
        for i in range(0, pitch, 1 << 18):
            x[:, i:i + (1 << 18)] += centres[:, of[i:i + (1 << 18)]]
    return x[:, :n]


def _sets(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    centres = None
    if case["dist"] == "mixture":
        centres = torch.empty((case["dim"], case["centres"]), device=DEV)
        if case["unit"]:
            centres.normal_(generator=gen)
            centres /= centres.norm(dim=0)
        else:
            centres.uniform_(-1.0, 1.0, generator=gen)
    ref = _generate(case, gen, centres, case["ref_nb"], case["dim"])
    return ref, _generate(case, gen, centres, case["query_nb"], case["dim"])


def _batch(case, seed):
    """[(ref, query, k)] of a batch: the shapes are the case's, the points the seed's."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    out = []
    for n, q, d, k, _ in workloads.batched_problems(case["count"], case["shapes"]):
        ref = torch.rand((d, (n + 3) // 4 * 4), generator=gen, device=DEV)[:, :n]
        out.append((ref, torch.rand((d, (q + 3) // 4 * 4), generator=gen, device=DEV)[:, :q], k))
    return out


def prepare(case, seed):
    s = dict(case)
    if case["kind"] == "batch":
        s["problems"] = _batch(case, seed)
        size = sum(q.shape[1] * k for _, q, k in s["problems"])
        s["dist_out"] = torch.empty(size, device=DEV)
        s["index_out"] = torch.empty(size, dtype=torch.int32, device=DEV)
        table, at = [], 0
        for ref, query, k in s["problems"]:
            e = at + query.shape[1] * k
            table.append((ref, query, k, s["dist_out"][at:e].view(k, -1),
                          s["index_out"][at:e].view(k, -1)))
            at = e
        s["plan"] = knncuda.BatchedPlan(knncuda.problems_from(table))
        return s
    s["ref"], s["query"] = _sets(case, seed)
    q, k = case["query_nb"], case["k"]
    if case["kind"] == "host":
        s["ref"], s["query"] = (np.ascontiguousarray(s[x].cpu().numpy()) for x in ("ref", "query"))
        s["dist_out"], s["index_out"] = np.empty((k, q), np.float32), np.empty((k, q), np.int32)
        return s
    s["dist_out"] = torch.empty((k, q), device=DEV)
    s["index_out"] = torch.empty((k, q), dtype=torch.int32, device=DEV)
    if case["kind"] == "serve":
        torch.cuda.synchronize()   # the set is copied on a stream of the library's own
        s["refset"] = knncuda.RefSet(s.pop("ref"))
    return s


def run(state):
    s = state
    if s["kind"] == "batch":
        s["plan"].run()
    elif s["kind"] == "serve":
        s["refset"].knn(s["query"], s["k"], s["method"], s["dist_out"], s["index_out"])
    elif s["kind"] == "host":
        ok = knncuda.ENTRY_POINTS[s["method"]](s["ref"], s["ref_nb"], s["query"], s["query_nb"],
                                               s["dim"], s["k"], s["dist_out"], s["index_out"])
        if not ok:
            raise RuntimeError("the call failed")
    else:
        knncuda.knn_device(s["ref"], s["query"], s["k"], s["method"], s["dist_out"],
                           s["index_out"])
    return s["dist_out"], s["index_out"]


def _shapes(case):
    if case["kind"] == "batch":
        return [p[:4] for p in workloads.batched_problems(case["count"], case["shapes"])]
    return [(case["ref_nb"], case["query_nb"], case["dim"], case["k"])]


def work(case):
    """Inputs read once, results written once.  Operations: the direct form subtracts, multiplies
    and adds for each coordinate of each pair; the expansion form multiplies and adds.  A resident
    set is read once too.  In up to 4 dimensions no pair of points has to be looked at for its own
    sake (a set can be searched in the order of its space), so only the bytes count."""
    each = 2 if case["method"] == "cublas" else 3
    b = f = 0
    for n, q, d, k in _shapes(case):
        b += 4 * d * (n + q) + 8 * k * q
        f += 0 if d <= 4 else each * n * q * d
    return {"bytes": b, "flops": f}


def _nearest(ref, query, k):
    """The k smallest distances of each query, ascending, in 64 bits (k x query_nb)."""
    ref, query = ref.double(), query.double()
    r2, q2 = (ref * ref).sum(0), (query * query).sum(0)
    step = max(1, (1 << 27) // ref.shape[1])
    out = []
    for i in range(0, query.shape[1], step):
        d2 = torch.addmm(r2[None, :], query[:, i:i + step].t(), ref, alpha=-2.0)
        d2 = torch.topk(d2, k, dim=1, largest=False, sorted=True).values + q2[i:i + step, None]
        out.append(d2.clamp_(min=0.0).sqrt_().t())
    return torch.cat(out, dim=1)


def exact(case, seed):
    """Distances; the indices have no 64-bit value of their own."""
    if sum(n * q for n, q, _, _ in _shapes(case)) > (1 << 32) - 1:
        return None
    if case["kind"] == "batch":
        return torch.cat([_nearest(*p).reshape(-1) for p in _batch(case, seed)]), None
    dist = _nearest(*_sets(case, seed), case["k"])
    return (dist.cpu().numpy() if case["kind"] == "host" else dist), None
