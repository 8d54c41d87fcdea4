"""The workloads that this library's speed is judged on, through its Python API.

A case is one call (or one index build) as a program that uses the library makes it: exact, IVF-PQ and HNSW search from
a single query to the benchmark's 10,000-query batches, and the two index constructions.  Every search returns ids,
distances and counts whole.  The library promises the same ids and the same distance bits for the same index and
queries, and byte-identical index files, so every case is compared exactly.
"""
import numpy as np
import torch

import ferrolm_b200 as fv

_ctx = None


def _context():
    """One context per process, as a program keeps it (it stands for the reference's thread pool)."""
    global _ctx
    if _ctx is None:
        _ctx = fv.Context(0)
    return _ctx


# ---------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # one question against the passages of a small document collection (the shape of BEIR SciFact: 5,183 x 384
        # unit-length embeddings), host vectors in, host results out: what the Retriever does per request
        dict(name="flat_one_query", path="flat", data="text", n=5183, dim=384, nq=1, k=10, host=True),
        # a batch of 1,000 against a base that still fits L2: the benchmark's first configuration
        dict(name="flat_100k", path="flat", data="sift", n=100_000, dim=128, nq=1000, k=10, host=False),
        # ground truth for the benchmark's own base: a million descriptors, 10,000 queries
        dict(name="flat_1m", path="flat", data="sift", n=1_000_000, dim=128, nq=10_000, k=10, host=False),
        # embeddings by inner product, no size a multiple of a tile
        dict(name="flat_text", path="flat", data="text", n=200_003, dim=384, nq=2049, k=10, host=False),
        # ground truth with 100 neighbours (recall at 100), rows of an odd length
        dict(name="flat_k100", path="flat", data="sift", n=50_001, dim=100, nq=501, k=100, host=False),
        # the headline: the benchmark's IVF-PQ index and batch, re-ranked
        dict(name="ivfpq_1m", path="ivfpq", data="sift", n=1_000_000, dim=128, nq=10_000, k=10, nlist=1024, m=16,
             nprobe=64, refine=10, host=False),
        # a server's micro-batch on a compressed index, no re-ranking
        dict(name="ivfpq_micro_batch", path="ivfpq", data="sift", n=300_000, dim=128, nq=32, k=10, nlist=512, m=16,
             nprobe=16, refine=0, host=True),
        # embeddings by inner product, 8 components per code byte, re-ranked
        dict(name="ivfpq_text", path="ivfpq", data="text", n=100_000, dim=384, nq=1000, k=10, nlist=256, m=48,
             nprobe=16, refine=4, host=False),
        # a few questions at once against the graph of a small collection
        dict(name="hnsw_few_queries", path="hnsw", data="text", n=5183, dim=384, nq=20, k=10, m=16, ef=64, host=True),
        # the benchmark's graph search
        dict(name="hnsw_200k", path="hnsw", data="sift", n=200_000, dim=128, nq=10_000, k=10, m=16, ef=64, host=False),
        # an index made from scratch: k-means, codebooks, encoding, filing, the file
        dict(name="ivfpq_build", path="ivfpq_build", data="sift", n=100_000, dim=128, sample=25_000, nlist=256, m=16,
             iters=10),
        # a graph made from scratch with the reference's default parameters
        dict(name="hnsw_build", path="hnsw_build", data="text", n=20_000, dim=96, m=16, efc=200),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    path = rng.choice(["flat", "flat", "flat", "ivfpq", "ivfpq", "ivfpq", "hnsw", "hnsw", "ivfpq_build", "hnsw_build"])
    data = rng.choice(["sift", "text"])
    if path == "flat":
        dim = rng.randint(24, 160) if data == "sift" else rng.choice([256, 384, 384, rng.randint(200, 512)])
        nq, n = _log(rng, 1, 10_000), _log(rng, 1000, 1_000_000)
        n = max(1000, min(n, 1_280_000_000_000 // (nq * dim), 250_000_000 // dim))
        return dict(path=path, data=data, n=n, dim=dim, nq=nq, k=rng.choice([1, 10, 10, 10, rng.randint(2, 100)]),
                    host=rng.random() < 0.3)
    if path == "ivfpq":
        m = rng.choice([8, 16, 16, 16, 32])
        dim = m * rng.choice([4, 6, 8]) if data == "sift" else m * rng.choice([8, 12])
        n, nq = _log(rng, 10_000, 400_000), _log(rng, 1, 10_000)
        nlist = max(16, min(1024, n // rng.randint(200, 1200)))
        nprobe = min(nlist, _log(rng, 1, 64))
        return dict(path=path, data=data, n=n, dim=dim, nq=nq, k=rng.choice([1, 10, 10, rng.randint(2, 50)]),
                    nlist=nlist, m=m, nprobe=nprobe, refine=rng.choice([0, 4, 10]), host=rng.random() < 0.3)
    if path == "hnsw":
        dim = rng.randint(32, 128) if data == "sift" else rng.choice([384, rng.randint(96, 400)])
        return dict(path=path, data=data, n=_log(rng, 2000, 100_000), dim=dim, nq=_log(rng, 1, 10_000), k=10,
                    m=rng.choice([8, 16, 16, 24]), ef=_log(rng, 16, 256), host=rng.random() < 0.3)
    if path == "ivfpq_build":
        m = rng.choice([8, 16])
        n = _log(rng, 10_000, 100_000)
        return dict(path=path, data=data, n=n, dim=m * rng.choice([4, 6, 8]), sample=max(5000, n // 4),
                    nlist=rng.randint(16, 256), m=m, iters=rng.randint(3, 10))
    return dict(path=path, data=data, n=_log(rng, 1000, 20_000), dim=rng.randint(32, 96), m=rng.choice([8, 16]),
                efc=rng.choice([100, 200]))


# --------------------------------------------------------------------------------------------------------- inputs
def _rows(kind, seed, part, n, dim):
    """Rows of the benchmark's mixtures, made on the GPU.  sift: 256 centres uniform in [0, 255], sigma 30, clipped and
    rounded (integers, as SIFT's components are); text: 1,000 centres normal * 3, sigma 1, scaled to unit length."""
    g = torch.Generator("cuda")
    g.manual_seed(seed * 7919 + 1)  # the centres are those of the seed, whichever part is drawn
    if kind == "sift":
        centres = torch.rand((256, dim), generator=g, device="cuda") * 255.0
    else:
        centres = torch.randn((1000, dim), generator=g, device="cuda") * 3.0
    g.manual_seed(seed * 7919 + 2 + part)
    at = torch.randint(0, centres.shape[0], (n,), generator=g, device="cuda")
    x = centres[at]
    noise = torch.randn((n, dim), generator=g, device="cuda")
    if kind == "sift":
        return x.add_(noise, alpha=30.0).round_().clamp_(0.0, 255.0)
    return torch.nn.functional.normalize(x.add_(noise), dim=1)


def _metric(case):
    return fv.Metric.L2 if case["data"] == "sift" else fv.Metric.InnerProduct


def prepare(case, seed):
    path, kind, n, dim = case["path"], case["data"], case["n"], case["dim"]
    ctx = _context()
    base = _rows(kind, seed, 0, n, dim)
    if path == "hnsw_build":  # the constructions take host vectors
        return dict(case=case, ctx=ctx, base=base.cpu().numpy())
    if path == "ivfpq_build":
        return dict(case=case, ctx=ctx, base=base.cpu().numpy(), sample=_rows(kind, seed, 2, case["sample"], dim).cpu().numpy())
    queries = _rows(kind, seed, 1, case["nq"], dim)
    if path == "flat":
        index = fv.FlatIndex(ctx, _metric(case), dim)
        index.add(base)
    elif path == "ivfpq":
        sample = base[: max(5000, 25 * case["nlist"])].cpu().numpy()
        index = fv.IvfPq.train(ctx, _metric(case), dim, sample, fv.IvfPqParams(case["nlist"], case["m"], 4, True, 1))
        index.add(base)
    else:
        index = fv.Hnsw.build_batched(ctx, _metric(case), dim, base.cpu().numpy(), fv.HnswParams(case["m"], 200, 1))
    return dict(case=case, index=index, queries=queries.cpu().numpy() if case["host"] else queries)


# ------------------------------------------------------------------------------------------------------- the call
def run(state):
    case = state["case"]
    path = case["path"]
    if path == "ivfpq_build":
        p = fv.IvfPqParams(case["nlist"], case["m"], case["iters"], True, 1)
        index = fv.IvfPq.train(state["ctx"], _metric(case), case["dim"], state["sample"], p)
        index.add(state["base"])
        return np.frombuffer(index.save(), dtype=np.uint8)
    if path == "hnsw_build":
        p = fv.HnswParams(case["m"], case["efc"], 1)
        data = fv.Hnsw.build_batched(state["ctx"], _metric(case), case["dim"], state["base"], p).save()
        # the file's length depends on the links of the upper layers: in an array of one length, with zeros behind it
        out = np.zeros(4 * case["n"] * (fv.padded(case["dim"]) + 4 * case["m"] + 4) + 65536, dtype=np.uint8)
        out[: len(data)] = np.frombuffer(data, dtype=np.uint8)
        return out
    index, queries = state["index"], state["queries"]
    if path == "flat":
        out, counts = index.search_batch(queries, case["k"])
    elif path == "ivfpq":
        out, counts = index.search_batch(queries, case["k"], case["nprobe"], case["refine"])
    else:
        out, counts = index.search_batch(queries, case["k"], case["ef"])
    if case["host"]:
        return dict(ids=out["id"], distances=out["distance"], counts=counts)
    return dict(ids=out[..., 0], distances=out[..., 1].view(torch.float32), counts=counts)


# ----------------------------------------------------------------------------------------------- what is expected
def work(case):
    path, n, dim = case["path"], case["n"], case["dim"]
    if path == "flat":
        nq = case["nq"]
        return dict(bytes=4 * dim * (n + nq) + 8 * nq * case["k"], flops=2 * n * nq * dim)
    if path == "ivfpq":
        nq, m, nlist, nprobe = case["nq"], case["m"], case["nlist"], case["nprobe"]
        rows = nq * nprobe * n // nlist  # (query, row) pairs that are scored
        reranked = nq * case["k"] * case["refine"]
        read = min(1.0, nq * nprobe / nlist) * n * (m + 4) + 4 * dim * (nlist + 256 + nq + min(reranked, n)) + 8 * nq * case["k"]
        return dict(bytes=int(read), flops=2 * nq * dim * (nlist + 256) + rows * m + 2 * reranked * dim)
    if path == "hnsw":
        nq, ef = case["nq"], case["ef"]
        evals = nq * ef * case["m"] // 2  # about half of a node's links are new when it is expanded
        read = min(evals, n) * 4 * dim + min(nq * ef, n) * 4 * (2 * case["m"] + 1) + 4 * dim * nq + 8 * nq * case["k"]
        return dict(bytes=int(read), flops=2 * dim * evals)
    if path == "ivfpq_build":
        s, nlist, m = case["sample"], case["nlist"], case["m"]
        flops = case["iters"] * 2 * s * dim * (nlist + 256) + 2 * n * dim * (nlist + 256)
        return dict(bytes=4 * dim * (n + s) + n * (m + 4 + 4 * dim), flops=flops)
    evals = n * case["efc"] * case["m"] // 2
    return dict(bytes=4 * dim * n * 2 + 4 * n * (2 * case["m"] + 1), flops=2 * dim * evals)


def tolerance(case):
    """Ids, counts and distance bits do not depend on how a search is computed, nor index files on how they are built."""
    return "exact"


def exact(case, seed):
    """Distances of exact search in 64 bits.  What IVF-PQ and HNSW find depends on an index that only this library makes."""
    if case["path"] != "flat":
        return None
    n, dim, nq, k = case["n"], case["dim"], case["nq"], case["k"]
    base, queries = (_rows(case["data"], seed, p, r, dim).double() for p, r in ((0, n), (1, nq)))
    best = torch.empty((nq, min(k, n)), dtype=torch.float64, device="cuda")
    step = max(1, 100_000_000 // n)
    for a in range(0, nq, step):
        q = queries[a : a + step]
        d = -(q @ base.T)
        if case["data"] == "sift":
            d = d.mul_(2.0).add_((base * base).sum(1)[None]).add_((q * q).sum(1)[:, None])
        best[a : a + step] = torch.topk(d, min(k, n), dim=1, largest=False, sorted=True).values
    return dict(ids=None, distances=best.cpu().numpy() if case["host"] else best, counts=None)
