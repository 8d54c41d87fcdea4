"""The per-stage device times that a context records on request: every search fills the first, whichever side its queries
and results are on, and a context that was not asked records none."""
import pytest

pytestmark = pytest.mark.gpu

L2 = 0


@pytest.fixture(scope="module")
def made(oracle):
    import ferrolm_b200 as fv

    ctx = fv.Context(0)
    base = oracle.testdata(6000, 64, 1)
    flat = fv.FlatIndex(ctx, L2, 64)
    flat.add(base)
    ivf = fv.IvfPq.train(ctx, L2, 64, base[:3000], fv.IvfPqParams(32, 16, 3, True, 1))
    ivf.add(base)
    graph = fv.Hnsw.build_batched(ctx, L2, 64, base[:3000], fv.HnswParams(8, 60, 1))
    empty = fv.IvfPq.train(ctx, L2, 64, base[:3000], fv.IvfPqParams(32, 16, 1, True, 1))
    yield ctx, {"flat": lambda q: flat.search_batch(q, 10), "ivfpq": lambda q: ivf.search_batch(q, 10, 16, 4),
                "hnsw": lambda q: graph.search_batch(q, 10, 40), "empty": lambda q: empty.search_batch(q, 10, 16, 4)}
    ctx.close()


@pytest.mark.parametrize("kind", ["flat", "ivfpq", "hnsw", "empty"])
@pytest.mark.parametrize("nq", [1, 300, 14_000])  # 14,000 x 10 results do not fit the pinned memory
def test_stage_times(made, oracle, kind, nq):
    import torch

    ctx, search = made
    host = oracle.testdata(nq, 64, 2)
    for q in (host, torch.from_numpy(host).cuda()):
        ctx.set_timing(True)
        search[kind](q)
        st = ctx.stats()["stage_ms"]
        assert st[0] > 0 and all(0 <= x < 1000 for x in st), st
        ctx.set_timing(False)
        search[kind](q)
        assert not any(ctx.stats()["stage_ms"])
