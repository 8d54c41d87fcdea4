"""Search and construction over the branches of the beam: in registers (up to 32, 64, 128, 256 entries) or in shared
memory, by a team of warps per query (small batches) or a warp per query, visited set within or beyond shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L2, IP = 0, 1
TEAM_MAX = 16 * 148  # a launch of up to 16 searches per SM is run by teams


@pytest.fixture(scope="module")
def setup(oracle):
    import ferrolm_b200 as fv

    ctx = fv.Context(0)
    made = {}

    def graph(metric, n, dim, m, efc):
        key = (metric, n, dim, m, efc)
        if key not in made:
            base = oracle.testdata(n, dim, 5)
            # rows on a coarse grid: many exactly equal distances
            base = np.round(base * 2).astype(np.float32) if metric == L2 else oracle.normalize(base)
            g = fv.Hnsw.build_batched(ctx, metric, dim, base, fv.HnswParams(m, efc, 1), max_batch=8192, divisor=1)
            o = oracle.Hnsw.build_batched(metric, dim, base, m=m, ef_construction=efc, seed=1, max_batch=8192, divisor=1)
            made[key] = g, o
        return made[key]

    yield graph, ctx
    made.clear()
    ctx.close()


@pytest.mark.parametrize("metric,n,dim,m,efc", [
    (L2, 9000, 17, 8, 33),    # the widest batch (4,500 nodes) is inserted by single warps, the others by teams
    (IP, 3000, 104, 40, 100),  # 80 links per node: three runs per expansion
    (L2, 700, 392, 4, 300),   # the found list in shared memory
])
def test_graph_equals_the_oracles(setup, metric, n, dim, m, efc):
    graph, _ = setup
    g, o = graph(metric, n, dim, m, efc)
    assert g.save() == o.save()


@pytest.mark.parametrize("nq", [1, 37, TEAM_MAX, TEAM_MAX + 1])
@pytest.mark.parametrize("ef", [1, 31, 32, 33, 64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("metric,n,dim,m,efc", [(L2, 9000, 17, 8, 33), (IP, 3000, 104, 40, 100)])
def test_search_equals_the_oracle(setup, oracle, metric, n, dim, m, efc, ef, nq):
    if nq > TEAM_MAX and ef > 129 and metric == IP:
        nq = TEAM_MAX + 1 if ef == 257 else 40  # (the oracle's time)
    graph, ctx = setup
    g, o = graph(metric, n, dim, m, efc)
    q = oracle.testdata(nq, dim, 6)
    q = np.round(q * 2).astype(np.float32) if metric == L2 else oracle.normalize(q)
    k = min(10, ef)
    got, gc = g.search_batch(q, k, ef)
    stats = ctx.stats()
    want, wc, work = o.search_batch(q, k, ef, want_work=True)
    if stats["uncertified"] == 0:  # (a tie list that overflowed may resolve later ties differently)
        assert np.array_equal(gc, wc) and np.array_equal(got["id"], want["id"])
        assert np.array_equal(got["distance"].view(np.uint32), want["distance"].view(np.uint32))
        assert stats["dist_evals"] == work[0] and stats["expansions"] == work[1]
    else:
        assert stats["uncertified"] <= 0.01 * nq + 1
