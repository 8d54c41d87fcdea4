"""Graph search over whole numbers within 255 of each other, whose distances come from bytes, and over what just fails to qualify,
against the oracle: ids and distance bits, by scouting teams, by teams and by single warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import ferrolm_b200 as fv

    c = fv.Context(0)
    yield c
    c.close()


def whole(n, dim, lo, span, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, span + 1, size=(n, dim))
    x[0], x[1] = 0, span  # both ends are met
    return (x + lo).astype(np.float32)


def check(oracle, ctx, base, queries, ef):
    import ferrolm_b200 as fv

    dim = base.shape[1]
    g = fv.Hnsw.build_batched(ctx, fv.Metric.L2, dim, base, fv.HnswParams(8, 40, 1))
    o = oracle.Hnsw.load(g.save())
    want, wc = o.search_batch(queries, 10, ef)
    for nq in (7, 500, len(queries)):
        got, gc = g.search_batch(queries[:nq], 10, ef)
        assert np.array_equal(gc, wc[:nq])
        assert np.array_equal(got.view(np.uint64), want[:nq].view(np.uint64)), nq


@pytest.mark.parametrize("dim", [5, 8, 16, 17, 64, 100, 128, 129, 200, 248, 256, 260])  # 257 and more are beyond the form
def test_dimensions(oracle, ctx, dim):
    check(oracle, ctx, whole(1500, dim, 0, 255, dim), whole(3000, dim, 0, 255, dim + 1), 40)


@pytest.mark.parametrize("lo,span", [(-128, 255), (0, 90), (5000, 255), (-7, 255), (-1, 256), (100_000, 100)])
def test_ranges(oracle, ctx, lo, span):
    check(oracle, ctx, whole(1500, 36, lo, span, 3), whole(3000, 36, lo, span, 4), 24)


def test_queries_that_do_not_fit(oracle, ctx):
    base, q = whole(2000, 40, 0, 255, 5), whole(3000, 40, 0, 255, 6)
    q[::3] += 0.5
    q[1::7, 39] = 256
    q[2::7, 0] = -3
    check(oracle, ctx, base, q, 70)


def test_values_that_are_not_whole(oracle, ctx):
    base = whole(2000, 40, 0, 255, 7)
    base[1999, 39] += 0.25
    check(oracle, ctx, base, whole(3000, 40, 0, 255, 8), 33)


@pytest.mark.parametrize("lo,span", [(-128, 255), (-7, 255), (-250, 120)])
def test_queries_a_little_off_whole_numbers(oracle, ctx, lo, span):
    # the difference to the rows' lowest value rounds to a whole number where the components are none
    base, q = whole(1500, 40, lo, span, 11), whole(3000, 40, lo, span, 12)
    base[200:240], base[240:280] = -1, 1
    rng = np.random.default_rng(13)
    little = q * np.float32(1 + 2.0**-22)
    little[q == 0] = 5e-6
    at = rng.random(q.shape) < 0.1
    q[at] = little[at]
    q[:, 7] = little[:, 7]
    q[1], q[2], q[3], q[4], q[1000] = 5e-6, 3.0000002, 0.99999994, 1e-6, 1e-6
    check(oracle, ctx, base, q, 24)
