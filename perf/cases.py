"""Measurement cases of the k-NN / LSH engine: what its users have it do.

A program keeps a resident index over its base vectors and answers query batches with it
(`Index.query_device_async` on buffers in device memory), or makes the one-shot call over
host arrays that the reference's users make (`linear_scans`).  The cases cover the scans
and sketches of the measurement configurations at their sizes -- 1.2M, 1M, 500k and 100k
base vectors of 100 or 128 dimensions, 10,000 or 1,000 queries, k = 32 -- and around them
the smallest requests of the serving loop, odd base, batch and dimension sizes, and the
larger k of its request mix (10, 32, 100).

Every case runs on synthetic data: unit vectors from 1,000 Gaussian clusters (sigma 0.05
a coordinate) for the angular paths, nonnegative rows with 30% Gamma(2, 1) weights for the
Jaccard ones.  All batches of a process go down one stream, as in a program that answers
one batch after another.
"""
from __future__ import annotations

import math

import torch

import lshongpu_gb300 as L

CLUSTERS = 1000
SIGMA = 0.05


def listed():
    return [
        # the headline: a large batch on the 1.2M x 100 base through the tensor-core exact scan
        {"name": "tc_10k", "path": "tc", "n": 1_200_000, "d": 100, "q": 10_000, "k": 32},
        # an ordinary batch on a mid-sized base (the 100k x 100 configuration)
        {"name": "tc_1k", "path": "tc", "n": 100_000, "d": 100, "q": 1000, "k": 32},
        # one interactive lookup in the large base: latency
        {"name": "tc_one_query", "path": "tc", "n": 1_200_000, "d": 100, "q": 1, "k": 10},
        # sizes that fill no tile, and the largest k of the serving mix
        {"name": "tc_ragged", "path": "tc", "n": 333_337, "d": 37, "q": 777, "k": 100},
        # the reference's exact scan, ids and distances bit for bit (100k x 100 configuration)
        {"name": "exact_1k", "path": "exact", "dist": 1, "n": 100_000, "d": 100, "q": 1000, "k": 32},
        # the exact generalized-Jaccard scan: ground truth for the MinHash paths
        {"name": "exact_jaccard", "path": "exact", "dist": 2, "n": 60_013, "d": 100, "q": 129, "k": 10},
        # 1,024-bit SimHash sketches of the large base, 1,024 candidates re-ranked
        {"name": "simhash_10k", "path": "simhash", "n": 1_200_000, "d": 100, "q": 10_000, "k": 32, "words": 32,
         "c": 1024},
        # a small request on the same sketches
        {"name": "simhash_16", "path": "simhash", "n": 1_200_000, "d": 100, "q": 16, "k": 10, "words": 32, "c": 128},
        # cross-polytope LSH tables over 1M vectors padded to 128 dimensions
        {"name": "lsh_10k", "path": "lsh", "n": 1_000_000, "d": 128, "q": 10_000, "k": 32, "tables": 32, "hashes": 2},
        # weighted MinHash, 256 byte samples, the reference's default candidate count (the largest case)
        {"name": "wmh_bytes_10k", "path": "wmh", "n": 500_000, "d": 100, "q": 10_000, "k": 32, "samples": 256,
         "c": 4096},
        # the same base with 256 one-bit samples
        {"name": "wmh_onebit_10k", "path": "wmh1", "n": 500_000, "d": 100, "q": 10_000, "k": 32, "words": 8, "c": 4096},
        # the reference's one-shot call on host arrays: upload, index build, scan, download
        {"name": "call_exact", "path": "call", "impl": 2, "n": 20_011, "d": 100, "q": 257, "k": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any path, base, batch and dimension sizes over their whole range,
    within the listed ones' cost."""
    path = rng.choice(["tc", "tc", "tc", "tc8", "exact", "exact", "simhash", "simhash", "wmh", "wmh1", "cws", "jl",
                       "lsh", "lsh", "call"])
    n = _log_int(rng, 10_000, 1_200_000)
    q = _log_int(rng, 1, 10_000)
    d = rng.randint(16, 128)
    k = rng.choice([1, 5, 10, 32, 32, 64, 100, 128])
    case = {"path": path, "n": n, "d": d, "q": q, "k": k}
    if path == "exact":
        case["dist"] = rng.choice([1, 1, 2, 3])
        cap = 3e11 if case["dist"] == 1 else 1e11
        case["q"] = max(1, min(q, int(cap / (2.0 * n * d))))
    elif path in ("simhash", "wmh1"):
        case["words"] = rng.choice([4, 8, 16, 32]) if path == "simhash" else rng.choice([4, 8])
        case["c"] = rng.choice([128, 256, 1024, 4096])
        if path == "wmh1":
            case["n"] = min(n, 500_000)
    elif path in ("wmh", "cws"):
        case["samples"] = rng.choice([64, 128, 256])
        case["c"] = rng.choice([256, 1024, 4096])
        case["n"] = min(n, 500_000)
        case["q"] = q if q >= 64 else max(1, q // 2)  # below 64 queries each one scans the samples by itself
    elif path == "jl":
        case["sdim"] = rng.choice([16, 32, 64])
        case["c"] = rng.choice([128, 256, 1024])
        case["q"] = max(1, min(q, int(2e10 / (2.0 * n * case["sdim"]))))
    elif path == "lsh":
        case["hashes"] = rng.choice([1, 2, 2])
        case["tables"] = rng.randint(4, 40)
        if case["hashes"] == 1:  # few, full buckets
            case["n"] = min(n, 50_000)
            case["q"] = min(q, 2000)
    elif path == "call":
        case["impl"] = rng.choice([2, 8])
        case["n"] = min(n, 200_000)
        case["q"] = max(1, min(q, int(1e11 / (2.0 * case["n"] * d))))
    return case


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _clustered(rows, centres, g):
    """rows unit vectors around the centres."""
    lab = torch.randint(0, centres.shape[0], (rows,), device="cuda", generator=g)
    v = centres[lab]
    v += SIGMA * torch.randn(v.shape, device="cuda", generator=g)
    return torch.nn.functional.normalize(v, dim=1)


def _sparse_gamma(rows, d, g):
    """Nonnegative rows: 30% of the entries drawn from Gamma(2, 1), at least one a row."""
    u = torch.rand((2, rows, d), device="cuda", generator=g).clamp_min_(1e-7)
    v = -(u[0].log() + u[1].log())
    keep = torch.rand((rows, d), device="cuda", generator=g) < 0.3
    keep.scatter_(1, torch.randint(0, d, (rows, 1), device="cuda", generator=g), True)
    return v * keep


def _inputs(case, seed):
    g = _generator(seed)
    n, q, d = case["n"], case["q"], case["d"]
    if case["path"] in ("wmh", "wmh1", "cws") or case.get("dist") == L.JACCARD:
        return _sparse_gamma(n, d, g), _sparse_gamma(q, d, g)
    centres = torch.nn.functional.normalize(torch.randn((CLUSTERS, d), device="cuda", generator=g), dim=1)
    return _clustered(n, centres, g), _clustered(q, centres, g)


def _index(case, x):
    n, d = x.shape
    path = case["path"]
    at = dict(device_ptr=x.data_ptr(), n=n, d=d)
    if path == "tc":
        return L.Index(implementation=L.IMPL_TC, **at)
    if path == "tc8":
        return L.Index(implementation=L.IMPL_TC_FP8, **at)
    if path == "exact":
        return L.Index(implementation=L.IMPL_EXACT, distanceFunc=case["dist"], **at)
    if path == "lsh":
        p = 1
        while p < d:
            p *= 2
        bits = case["hashes"] * (p.bit_length())  # log2((2p)^hashes)
        return L.Index(implementation=L.IMPL_EXACT, framework=1, keysImplementation=L.KEYS_CROSSPOLY,
                       bucketKeyBits=bits, tables=case["tables"], options=L.make_options(cp_hashes=case["hashes"]), **at)
    opt = L.make_options(candidates=case["c"])
    if path == "simhash":
        return L.Index(implementation=L.IMPL_SIMHASH, sketchDim=case["words"], options=opt, **at)
    if path == "wmh":
        return L.Index(implementation=L.IMPL_WMH, distanceFunc=L.JACCARD, sketchDim=case["samples"], options=opt, **at)
    if path == "wmh1":
        return L.Index(implementation=L.IMPL_WMH_ONEBIT, distanceFunc=L.JACCARD, sketchDim=case["words"], options=opt,
                       **at)
    if path == "cws":
        return L.Index(implementation=L.IMPL_CWS, distanceFunc=L.JACCARD, sketchDim=case["samples"], options=opt, **at)
    if path == "jl":
        return L.Index(implementation=L.IMPL_JL, sketchDim=case["sdim"], options=opt, **at)
    raise ValueError(path)


_stream = None


def _one_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def prepare(case, seed):
    x, q = _inputs(case, seed)
    if case["path"] == "call":
        return {"case": case, "x": x.cpu().numpy(), "q": q.cpu().numpy()}
    torch.cuda.synchronize()  # the index is built on a stream of its own
    out = torch.empty((case["q"], case["k"], 2), dtype=torch.int32, device="cuda")  # (id, distance) pairs
    state = {"case": case, "index": _index(case, x), "q": q, "out": out, "stream": _one_stream().cuda_stream,
             "ids": out[:, :, 0], "distances": out.view(torch.float32)[:, :, 1]}
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["path"] == "call":
        r = L.linear_scans(case["impl"], case["k"], case["d"], case["q"], case["n"], state["x"], state["q"], 0,
                           L.ANGULAR)
        return {"ids": r.ids, "distances": r.distances}
    state["index"].query_device_async(state["q"].data_ptr(), case["q"], case["k"], state["out"].data_ptr(),
                                      stream=state["stream"])
    return {"ids": state["ids"], "distances": state["distances"]}


def work(case):
    """Bytes and operations of one batch: the base (or its sketches), the queries and the
    re-ranked rows read once, the results written once."""
    n, q, d, k, path = case["n"], case["q"], case["d"], case["k"], case["path"]
    ends = 4.0 * q * d + 8.0 * q * k
    if path in ("tc", "tc8", "call"):
        return {"bytes": 4.0 * n * d + ends, "flops": 2.0 * q * n * d}
    if path == "exact":
        # angular: multiply-add; Euclidean: subtract, multiply-add; Jaccard: min, max, two sums
        return {"bytes": 4.0 * n * d + ends, "flops": {1: 2.0, 2: 4.0, 3: 3.0}[case["dist"]] * q * n * d}
    if path == "lsh":
        p = 1 << (d - 1).bit_length()
        keys = 3.0 * p * math.log2(p) * case["tables"] * case["hashes"] * q
        # a bucket of a clustered base holds its cluster's points that agree on the key
        cand = float(q) * case["tables"] * (60 if case["hashes"] == 2 else n / p)
        return {"bytes": min(float(n), cand) * (4.0 * d + 4) + 4.0 * cand + ends, "flops": keys + 2.0 * cand * d}
    c = min(case["c"], n)
    rows = 4.0 * d * min(float(n), float(q) * c)
    if path in ("simhash", "wmh1"):
        bits = 32.0 * case["words"]
        sketch = 2.0 * q * d * bits if path == "simhash" else 0.0
        rank = (2.0 if path == "simhash" else 4.0) * q * c * d
        return {"bytes": n * bits / 8 + rows + ends, "flops": 2.0 * q * n * bits + sketch + rank}
    if path in ("wmh", "cws"):
        return {"bytes": float(n) * case["samples"] + rows + ends,
                "flops": float(q) * n * case["samples"] + 4.0 * q * c * d}
    return {"bytes": 4.0 * n * case["sdim"] + rows + ends, "flops": 3.0 * q * n * case["sdim"] + 2.0 * q * c * d}


def _top(dist, k):
    return torch.topk(dist, k, dim=1, largest=False, sorted=True).values


def exact(case, seed):
    """The k smallest distances of every query in double precision, for the paths that
    return the exact neighbours.  Which ids win among neighbours whose distances differ by
    less than single precision resolves is theirs to say, and the candidates of the
    sketched paths and of the LSH tables follow from the engine's own random projections:
    no value for those."""
    n, q, d, k = case["n"], case["q"], case["d"], case["k"]
    if case["path"] not in ("tc", "exact", "call"):
        return None
    x, qs = (v.double() for v in _inputs(case, seed))
    jaccard = case.get("dist") == L.JACCARD
    # rows a block: 4 GB of distances, or of per-dimension minima
    step = max(1, int(5e8 / n) // (d if jaccard else 1))
    got = []
    if jaccard:
        x = torch.nn.functional.normalize(x, dim=1)
        qs = torch.nn.functional.normalize(qs, dim=1)
        sx = x.sum(dim=1)
    else:
        nx, nq = x.norm(dim=1), qs.norm(dim=1)
    for i in range(0, q, step):
        b = qs[i:i + step]
        if jaccard:
            low = torch.minimum(b[:, None, :], x[None]).sum(dim=2)
            dist = 1 - low / (b.sum(dim=1)[:, None] + sx[None] - low)
        elif case.get("dist") == L.EUCLIDEAN:
            dist = ((nq[i:i + step] ** 2)[:, None] + (nx ** 2)[None] - 2 * (b @ x.T)).clamp_min(0).sqrt()
        else:
            dist = 1 - (b @ x.T) / (nq[i:i + step, None] * nx[None])
        got.append(_top(dist, k))
    return {"ids": None, "distances": torch.cat(got)}
