"""What a user of this library has it do, as timed cases: searches over flat, filtered, inverted-file, int8 and
product-quantised indexes, k-means training, and the encoding of vectors, each through the public Python entry points.

``listed()`` holds the fixed cases, ``draw(rng)`` one more case of the same ranges, ``prepare(case, seed)`` makes the
inputs and the index a program holds before the call, ``run(state)`` is one call, ``work(case)`` the bytes and
operations it cannot do without, ``tolerance(case)`` how far another correct implementation may be off.

All vectors are synthetic: N(0,1) entries (L2-normalised for cosine), uniform in [-1, 1] for Manhattan, and a Gaussian
mixture (centres N(0,1), noise 0.1) wherever structure matters (inverted lists, product quantisation, k-means).
"""
import math

import numpy as np
import torch

import vectorstorekit_b200 as vsk

_DEVICE = []


def _device():
    """One device object for the process, as a program holds it: indexes share its streams and work buffers."""
    if not _DEVICE:
        _DEVICE.append(vsk.CUDAAcceleratorStrategy(0).initialize())
    return _DEVICE[0]


# ---- the cases ---------------------------------------------------------------------------------------------------

def listed():
    return [
        # VectorStore.search on a small store: one host query, every launch and copy counts
        dict(name="flat_one_small", family="flat", metric="euclidean", rows=10_000, dim=128, queries=1, k=10, filtered=False,
             host=True),
        # VectorStore.search on a large store of text embeddings: one host query, bound by the bytes it reads
        dict(name="flat_one_large", family="flat", metric="cosine", rows=1_000_000, dim=768, queries=1, k=10, filtered=False,
             host=True),
        # the small batch of the benchmark's first configuration
        dict(name="flat_small_batch", family="flat", metric="euclidean", rows=100_000, dim=128, queries=1_000, k=10,
             filtered=False, host=False),
        # a ragged filtered batch from host memory: no size is a multiple of a tile, several distinct filters
        dict(name="flat_filtered_ragged", family="flat", metric="dotProduct", rows=300_007, dim=333, queries=777, k=37,
             filtered=True, host=True),
        # the headline batch: exact cosine search over a million embeddings
        dict(name="flat_large_batch", family="flat", metric="cosine", rows=1_000_000, dim=768, queries=10_000, k=100,
             filtered=False, host=False),
        # filtered Manhattan search, the metric without a matrix form
        dict(name="manhattan_filtered", family="flat", metric="manhattan", rows=5_000_000, dim=256, queries=10_000, k=50,
             filtered=True, host=False),
        # IVFIndex.search with the reference's default list and probe counts: one host query
        dict(name="ivf_one", family="ivf", rows=1_000_000, dim=128, nlist=1_024, nprobe=10, queries=1, k=10, host=True),
        # the benchmark's inverted-file batch
        dict(name="ivf_batch", family="ivf", rows=10_000_000, dim=128, nlist=4_096, nprobe=32, queries=10_000, k=10,
             host=False),
        # int8 scalar-quantised batch: one GPU's share of the benchmark's 50 million rows
        dict(name="sq8_batch", family="sq8", metric="dotProduct", rows=6_250_000, dim=384, queries=10_000, k=10, host=False),
        # product-quantised batch searched by asymmetric distance
        dict(name="pq_batch", family="pq", rows=10_000_000, dim=128, segments=16, queries=10_000, k=10, host=False),
        # Lloyd iterations of an inverted-file training run over the whole database
        dict(name="kmeans_train", family="kmeans", rows=10_000_000, dim=128, clusters=4_096, iterations=6, clustered=True),
        # product-quantising a block of new vectors
        dict(name="pq_encode", family="encode", quantizer="pq", rows=1_000_000, dim=128, segments=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_PAIRS = 7.68e12        # (query, row, dimension) triples of the largest contraction listed
_PAIRS_L1 = 6.4e12      # ... and of the Manhattan case (half of the rows pass its filter)


def draw(rng):
    family = rng.choice(["flat", "flat", "flat", "flat", "manhattan", "manhattan", "ivf", "ivf", "sq8", "pq", "kmeans", "encode"])
    queries = rng.choice([1, _log(rng, 1, 64), _log(rng, 64, 10_000), _log(rng, 64, 10_000)])
    host = rng.random() < (0.7 if queries <= 64 else 0.3)
    k = _log(rng, 1, 100)
    if family == "flat":
        dim, rows = _log(rng, 32, 1_536), _log(rng, 1_000, 1_000_000)
        rows = max(1_000, min(rows, int(_PAIRS / (queries * dim))))
        return dict(family="flat", metric=rng.choice(["euclidean", "cosine", "dotProduct"]), rows=rows, dim=dim, queries=queries,
                    k=k, filtered=rng.random() < 0.3, host=host)
    if family == "manhattan":
        dim, rows = _log(rng, 16, 512), _log(rng, 1_000, 5_000_000)
        filtered = rng.random() < 0.5
        rows = max(1_000, min(rows, int(_PAIRS_L1 * (2 if filtered else 1) / (queries * dim))))
        return dict(family="flat", metric="manhattan", rows=rows, dim=dim, queries=queries, k=k, filtered=filtered, host=host)
    if family == "ivf":
        rows = _log(rng, 50_000, 10_000_000)
        nlist = min(_log(rng, 64, 4_096), rows // 32)
        return dict(family="ivf", rows=rows, dim=_log(rng, 32, 256) if rows < 5_000_000 else _log(rng, 32, 128), nlist=nlist,
                    nprobe=min(_log(rng, 1, 64), nlist), queries=queries, k=k, host=host)
    if family == "sq8":
        dim = _log(rng, 32, 768)
        rows = min(_log(rng, 50_000, 6_250_000), int(2.4e9 / dim))
        return dict(family="sq8", metric=rng.choice(["dotProduct", "dotProduct", "euclidean"]), rows=rows, dim=dim, queries=queries,
                    k=k, host=host)
    if family == "pq":
        segments = rng.choice([8, 16, 32])
        return dict(family="pq", rows=_log(rng, 50_000, 10_000_000 * 16 // max(16, segments)), dim=segments * rng.choice([2, 4, 8]),
                    segments=segments, queries=queries, k=k, host=host)
    if family == "kmeans":
        rows = _log(rng, 20_000, 10_000_000)
        clustered = rng.random() < 0.7
        # rows without structure lie between many centroids: rounding grows tenfold per iteration there
        return dict(family="kmeans", rows=rows, dim=_log(rng, 16, 128), clusters=min(_log(rng, 16, 4_096), rows // 16),
                    iterations=6 if clustered else 2, clustered=clustered)
    quantizer = rng.choice(["sq8", "pq"])
    rows = _log(rng, 10_000, 1_000_000)
    if quantizer == "sq8":
        return dict(family="encode", quantizer="sq8", rows=rows, dim=_log(rng, 32, 768), segments=0)
    segments = rng.choice([8, 16, 32])
    return dict(family="encode", quantizer="pq", rows=rows, dim=segments * rng.choice([2, 4, 8]), segments=segments)


# ---- inputs ------------------------------------------------------------------------------------------------------

_PIECE = 1 << 20   # rows made at a time, so that large sets need no second copy of themselves


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, n, d, normalise):
    out = torch.empty((n, d), dtype=torch.float32, device="cuda")
    for b in range(0, n, _PIECE):
        part = out[b:b + _PIECE]
        part.normal_(generator=gen)
        if normalise:
            part /= torch.linalg.vector_norm(part, dim=1, keepdim=True)
    return out


def _uniform(gen, n, d):
    return torch.empty((n, d), dtype=torch.float32, device="cuda").uniform_(-1.0, 1.0, generator=gen)


def _mixture(gen, centres, n):
    out = torch.empty((n, centres.shape[1]), dtype=torch.float32, device="cuda")
    for b in range(0, n, _PIECE):
        part = out[b:b + _PIECE]
        pick = torch.randint(0, centres.shape[0], (part.shape[0],), device="cuda", generator=gen)
        part.normal_(0.0, 0.1, generator=gen)
        part += centres[pick]
    return out


def _masks(gen, n):
    """A uint64 metadata bitmask per row, bits Bernoulli(0.5) (as the int64 tensor with the same bits)."""
    lo = torch.randint(0, 1 << 32, (n,), device="cuda", generator=gen, dtype=torch.int64)
    hi = torch.randint(0, 1 << 32, (n,), device="cuda", generator=gen, dtype=torch.int64)
    return lo | (hi << 32)


def _host(t):
    return t.cpu().numpy()


def prepare(case, seed):
    dev, gen = _device(), _generator(seed)
    family = case["family"]
    s = {"case": case}
    if family == "flat":
        n, d, nq = case["rows"], case["dim"], case["queries"]
        metric = vsk.DistanceMetric(case["metric"])
        if case["metric"] == "manhattan":
            rows, queries = _uniform(gen, n, d), _uniform(gen, nq, d)
        else:
            cosine = case["metric"] == "cosine"
            rows, queries = _normal(gen, n, d, cosine), _normal(gen, nq, d, cosine)
        masks = qmasks = None
        if case["filtered"]:
            masks = _masks(gen, n)
            qmasks = torch.bitwise_left_shift(torch.ones(nq, dtype=torch.int64, device="cuda"),
                                              torch.randint(0, 64, (nq,), device="cuda", generator=gen))
        index = vsk.FlatIndex(dev, d, metric)
        index.add(rows, masks)
        s.update(index=index, k=min(case["k"], n), queries=_host(queries) if case["host"] else queries, qmasks=qmasks)
        if qmasks is not None and case["host"]:
            s["qmasks"] = _host(qmasks).view(np.uint64)
    elif family == "ivf":
        # one mixture component per list, k-means from rows of the sample: lists of very different lengths
        centres = _normal(gen, case["nlist"], case["dim"], False)
        rows = _mixture(gen, centres, case["rows"])
        index = vsk.IVFIndex(dev, case["dim"], case["nlist"], case["nprobe"], maxIterations=8, tolerance=0.0,
                             trainingSampleSize=max(100_000, case["nlist"]))
        sample = rows[: max(64 * case["nlist"], 100_000)]
        index.train(sample, sample[: case["nlist"]])
        index.insert(rows)
        queries = _mixture(gen, centres, case["queries"])
        s.update(index=index, k=case["k"], queries=_host(queries) if case["host"] else queries)
    elif family == "sq8":
        n, d = case["rows"], case["dim"]
        rows = _normal(gen, n, d, False)
        quantizer = vsk.ScalarQuantizer(dev, per_dim=True)
        quantizer.train(rows)
        index = vsk.QuantizedFlatIndex(dev, d, vsk.DistanceMetric(case["metric"]), quantizer.scale, quantizer.offset)
        index.add(quantizer.quantizeBatch(rows))
        del rows
        queries = _normal(gen, case["queries"], d, False)
        s.update(index=index, k=case["k"], queries=_host(queries) if case["host"] else queries)
    elif family == "pq":
        centres = _normal(gen, 4_096, case["dim"], False)
        rows = _mixture(gen, centres, case["rows"])
        quantizer = vsk.ProductQuantizer(dev, case["dim"], case["segments"], trainingIterations=5)
        quantizer.train(rows[:65_536] if case["rows"] > 65_536 else rows)
        index = quantizer.index()
        index.add(quantizer.encodeBatch(rows))
        del rows
        queries = _mixture(gen, centres, case["queries"])
        s.update(index=index, k=case["k"], queries=_host(queries) if case["host"] else queries)
    elif family == "kmeans":
        n, d, c = case["rows"], case["dim"], case["clusters"]
        rows = _mixture(gen, _normal(gen, c, d, False), n) if case["clustered"] else _normal(gen, n, d, False)
        s.update(rows=rows, clusters=c, initial=rows[:c].clone(),
                 trainer=vsk.KMeansClustering(dev, maxIterations=case["iterations"], tolerance=0.0))
    else:
        n, d = case["rows"], case["dim"]
        if case["quantizer"] == "sq8":
            rows = _normal(gen, n, d, False)
            quantizer = vsk.ScalarQuantizer(dev, per_dim=True)
        else:
            rows = _mixture(gen, _normal(gen, 4_096, d, False), n)
            quantizer = vsk.ProductQuantizer(dev, d, case["segments"], trainingIterations=5)
            quantizer.train(rows[:65_536])
        s.update(rows=rows, quantizer=quantizer)
    return s


# ---- one call ----------------------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    family = case["family"]
    if family == "flat":
        return state["index"].batchSearch(state["queries"], state["k"], state["qmasks"])
    if family in ("ivf", "sq8", "pq"):
        return state["index"].batchSearch(state["queries"], state["k"])
    if family == "kmeans":
        centroids, assignments, _, inertia = state["trainer"].cluster(state["rows"], state["clusters"], state["initial"])
        return centroids, assignments, inertia
    if case["quantizer"] == "sq8":
        scale, offset = state["quantizer"].train(state["rows"])
        return scale, offset, state["quantizer"].quantizeBatch(state["rows"])
    return state["quantizer"].encodeBatch(state["rows"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def work(case):
    family, d = case["family"], case["dim"]
    n = case["rows"]
    if family == "kmeans":
        c, it = case["clusters"], case["iterations"]
        return {"bytes": 4.0 * n * d + 4.0 * n + 8.0 * c * d, "flops": 2.0 * n * c * d * it + 1.0 * n * d * it}
    if family == "encode":
        if case["quantizer"] == "sq8":
            return {"bytes": 5.0 * n * d + 8.0 * d, "flops": 4.0 * n * d}
        return {"bytes": 4.0 * n * d + n * case["segments"] + 4.0 * 256 * d, "flops": 2.0 * n * 256 * d}
    nq, k = case["queries"], case["k"]
    io = 4.0 * nq * d + 12.0 * nq * k
    if family == "flat":
        share = 0.5 if case["filtered"] else 1.0
        seen = n * (1.0 - (1.0 - share) ** min(nq, 64))    # rows that some query's filter passes
        masks = 8.0 * (n + nq) if case["filtered"] else 0.0
        return {"bytes": 4.0 * seen * d + masks + io, "flops": (3.0 if case["metric"] == "manhattan" else 2.0) * share * n * nq * d}
    if family == "ivf":
        probed = case["nprobe"] / case["nlist"]
        seen = n * (1.0 - (1.0 - probed) ** nq)
        return {"bytes": 4.0 * seen * d + 4.0 * case["nlist"] * d + io, "flops": 2.0 * nq * d * (probed * n + case["nlist"])}
    if family == "sq8":
        return {"bytes": 1.0 * n * d + 8.0 * d + io, "flops": 2.0 * n * nq * d}
    m = case["segments"]
    return {"bytes": 1.0 * n * m + 4.0 * 256 * d + io, "flops": 1.0 * n * nq * m + 3.0 * nq * 256 * d}


def tolerance(case):
    family = case["family"]
    if family == "encode":
        return {"rel": 1e-6, "differ": 0.0}             # codes are whole numbers, formed with separately rounded operations
    if family == "pq":
        return {"rel": 1e-6, "differ": 0.0}             # sums of table entries in segment order, ties by row
    if family == "kmeans":
        # A row between two centroids may go either way, and every later mean with it.  Against the same iterations in
        # 64 bits: centroids 9e-5 (clustered, six iterations) to 2e-4 (unstructured, two), rows 2e-5.
        return {"rel": 8e-4, "differ": 1e-4}
    # fp32 sums of up to 1 536 terms in any order; rows whose distances agree to that rounding may change places.
    # The direct formulas summed in two different orders differ by at most 3e-7 (norm), 1.4e-6 (largest), 7e-5 (ids).
    return {"rel": 2e-6, "max": 1e-5, "differ": 5e-4}
