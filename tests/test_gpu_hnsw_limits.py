"""Graph search and construction at the limits of shared memory: long rows, long link lists, long beams; against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L2, IP = 0, 1


@pytest.fixture(scope="module")
def ctx():
    import ferrolm_b200 as fv

    c = fv.Context(0)
    yield c
    c.close()


def same(got, want):
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[0].view(np.uint64), want[0].view(np.uint64))


@pytest.mark.parametrize("metric", [L2, IP])
def test_rows_of_200_kb(oracle, ctx, metric):
    import ferrolm_b200 as fv

    base, q = oracle.testdata(40, 50_000, 1), oracle.testdata(5, 50_000, 2)
    g = fv.Hnsw.build(ctx, metric, 50_000, base, fv.HnswParams(4, 20, 1))
    same(g.search_batch(q, 5, 20), oracle.Hnsw.load(g.save()).search_batch(q, 5, 20))
