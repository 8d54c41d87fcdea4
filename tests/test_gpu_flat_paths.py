"""Exact search over the paths the library picks by itself: the one-launch scan of a handful of queries, the tensor-core
front end with results longer than 32, and the selection over few rows; against the oracle, ties included."""
import numpy as np
import pytest

from tests.parity import assert_same_neighbours

pytestmark = pytest.mark.gpu

L2, IP = 0, 1


@pytest.fixture(scope="module")
def ctx():
    import ferrolm_b200 as fv

    c = fv.Context(0)
    yield c
    c.close()


def rows(oracle, metric, n, dim, seed):
    x = oracle.testdata(n, dim, seed)
    # coarse grid: many exactly equal distances, ordered by id on both sides
    return np.round(x * 2).astype(np.float32) if metric == L2 else oracle.normalize(x)


def check(oracle, ctx, metric, n, dim, nq, k, what):
    import ferrolm_b200 as fv

    base, q = rows(oracle, metric, n, dim, 1), rows(oracle, metric, nq, dim, 2)
    ix = fv.FlatIndex(ctx, metric, dim)
    ix.add(base)
    o = oracle.FlatIndex(metric, dim)
    o.add(base)
    want, wc = o.search_batch(q, k)
    for mode in (0, 2):
        ix.set_mode(mode)
        got, gc = ix.search_batch(q, k)
        bits, total = assert_same_neighbours(got, gc, want, wc, f"{what}, mode {mode}")
        assert bits == total
    one, oc = ix.search_batch(q[:1], k)
    assert_same_neighbours(one, oc, want[:1], wc[:1], f"{what}, one query")


@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 4095, 4096, 40_001])
@pytest.mark.parametrize("nq,k", [(1, 1), (3, 10), (4, 32), (5, 33), (16, 100), (17, 128), (64, 10), (65, 40)])
def test_few_queries(oracle, ctx, metric, n, nq, k):
    check(oracle, ctx, metric, n, 20 if n % 2 else 72, nq, k, f"{nq} queries of {n} rows, k={k}")


@pytest.mark.parametrize("metric,n,dim,nq,k", [
    (L2, 4096, 24, 700, 33), (L2, 4096, 24, 66, 33), (IP, 4097, 24, 66, 33), (IP, 4100, 130, 257, 64), (L2, 20_000, 100, 300, 100), (IP, 20_000, 64, 129, 128),
    (L2, 20_000, 40, 2700, 33), (IP, 20_000, 40, 2700, 128),  # enough queries for one warp each in the re-rank
    (L2, 9000, 128, 300, 129),  # one beyond the tensor-core path
])
def test_long_results(oracle, ctx, metric, n, dim, nq, k):
    import ferrolm_b200 as fv

    base, q = rows(oracle, metric, n, dim, 1), rows(oracle, metric, nq, dim, 2)
    ix = fv.FlatIndex(ctx, metric, dim)
    ix.add(base)
    o = oracle.FlatIndex(metric, dim)
    o.add(base)
    want, wc = o.search_batch(q, k)
    got, gc = ix.search_batch(q, k)
    st = ctx.stats()
    assert got.tobytes() == want.tobytes() and (gc == wc).all()
    # the scan is one or two launches and the conversions around it; the tensor-core front end has a sample pass, its
    # bounds, the main pass and the re-rank besides.  Of 4,096 rows, a few queries' long results are the scan's.
    assert (st["launches"] >= 6) == (k <= 128 and (n > 4096 or nq > 66)), st
    if metric == IP:  # (the other metric's rows tie by the dozen, and a tie at the bound cannot be certified)
        assert st["uncertified"] <= 0.05 * nq, st
    ix.set_mode(2)
    got, gc = ix.search_batch(q, k)
    assert ctx.stats()["launches"] < 6
    assert got.tobytes() == want.tobytes() and (gc == wc).all()


@pytest.mark.parametrize("n,dim,nq,k", [
    (1, 12, 70, 2), (31, 12, 70, 5), (33, 12, 100, 31), (1025, 12, 300, 2), (2049, 12, 80, 300),
    # eight queries per warp with 128, 64 and 32 rows per block; on either side of four runs of 32 rows per SM, below which
    # two per warp take the rows of short vectors; of long ones, on either side of one block per SM
    (100, 12, 10_000, 33), (576, 12, 1184, 33), (600, 12, 1184, 33), (511, 12, 1184, 33), (512, 12, 1184, 33),
    (160, 260, 1184, 33), (127, 260, 1184, 33), (300, 252, 1000, 10), (300, 256, 1000, 10),
    # on either side of the line beyond which short results are kept in lists (512 + 3 padded dimensions)
    (4095, 12, 400, 33), (2049, 12, 560, 10), (2049, 12, 561, 10), (2048, 12, 561, 10),
])
def test_few_rows(oracle, ctx, n, dim, nq, k):
    check(oracle, ctx, L2, n, dim, nq, k, f"{n} rows x {dim}, k={k}")


def test_a_long_result_is_refused_by_the_forced_tensor_core_mode(oracle, ctx):
    import ferrolm_b200 as fv

    ix = fv.FlatIndex(ctx, L2, 16)
    ix.add(rows(oracle, L2, 5000, 16, 1))
    ix.set_mode(1)
    with pytest.raises(fv.FerrovecError):
        ix.search_batch(rows(oracle, L2, 4, 16, 2), 33)


# as many results as the pinned memory takes, and one query's more: 12,434 queries of 10
@pytest.mark.parametrize("nq", [12_434, 12_435])
def test_host_results_at_the_pinned_limit(oracle, ctx, nq):
    import torch

    import ferrolm_b200 as fv

    base, q = rows(oracle, IP, 3000, 24, 1), rows(oracle, IP, nq, 24, 2)
    flat = fv.FlatIndex(ctx, IP, 24)
    flat.add(base)
    ivf = fv.IvfPq.train(ctx, IP, 24, base[:1000], fv.IvfPqParams(16, 8, 2, True, 1))
    ivf.add(base)
    graph = fv.Hnsw.build_batched(ctx, IP, 24, base, fv.HnswParams(8, 40, 1))
    for search in (lambda x: flat.search_batch(x, 10), lambda x: ivf.search_batch(x, 10, 3, 4), lambda x: graph.search_batch(x, 10, 20)):
        got, gc = search(q)
        out, dc = search(torch.from_numpy(q).cuda())
        assert got.tobytes() == fv.neighbors_from_tensor(out).tobytes() and (gc == dc.cpu().numpy()).all()
        one, oc = search(q[-1:])
        assert one.tobytes() == got[-1:].tobytes() and oc[0] == gc[-1]
