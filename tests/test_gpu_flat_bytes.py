"""Exact search over whole numbers within 255 of each other, whose scores the tensor cores compute in 8-bit integers, and over
what just fails to qualify; against the oracle (ties included: these distances are small whole numbers)."""
import numpy as np
import pytest

from tests.parity import assert_same_neighbours

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
    x[: dim, 0] = 0  # both ends are met
    x[: dim, -1] = span
    return (x + lo).astype(np.float32)


def check(oracle, ctx, parts, queries, k):
    """`parts`: the base, added piece by piece."""
    import ferrolm_b200 as fv

    dim = queries.shape[1]
    ix, o = fv.FlatIndex(ctx, fv.Metric.L2, dim), oracle.FlatIndex(oracle.L2, dim)
    for p in parts:
        ix.add(p)
        o.add(p)
    want, wc = o.search_batch(queries, k)
    got, gc = ix.search_batch(queries, k)
    bits, total = assert_same_neighbours(got, gc, want, wc, f"dim {dim} k {k}")
    assert bits == total


# one k block and two, every number of MMAs in the last one, padded and whole dimensions; 225 is beyond the form
@pytest.mark.parametrize("dim", [4, 8, 31, 32, 33, 64, 65, 96, 100, 127, 128, 129, 160, 161, 200, 217, 224, 225])
def test_dimensions(oracle, ctx, dim):
    check(oracle, ctx, [whole(6001, dim, 0, 255, dim)], whole(300, dim, 0, 255, dim + 1), 10)


@pytest.mark.parametrize("lo,span", [(0, 255), (0, 1), (-128, 255), (-127, 200), (1000, 255), (-3000, 254), (0, 256), (-1, 256), (70000, 255)])
def test_ranges(oracle, ctx, lo, span):
    check(oracle, ctx, [whole(5000, 48, lo, span, 3)], whole(130, 48, lo, span, 4), 10)


@pytest.mark.parametrize("n,nq,k", [(4096, 65, 1), (4097, 256, 10), (4351, 257, 32), (40_000, 66, 33), (33_333, 513, 100), (9000, 2700, 128)])
def test_sizes(oracle, ctx, n, nq, k):
    check(oracle, ctx, [whole(n, 40, 0, 90, 5)], whole(nq, 40, 0, 90, 6), k)


def test_norms_that_do_not_fit(oracle, ctx):
    # components at both ends only: the sum that stands for the norm reaches 128 x 128^2
    rng = np.random.default_rng(7)
    ends = (rng.integers(0, 2, size=(4500, 128)) * 255).astype(np.float32)
    check(oracle, ctx, [ends], ends[:100], 10)


@pytest.mark.parametrize("what", ["half", "below", "above", "infinite"])
def test_queries_that_do_not_fit(oracle, ctx, what):
    base, q = whole(5000, 56, 0, 255, 8), whole(200, 56, 0, 255, 9)
    q[137, 55] = {"half": 3.5, "below": -1.0, "above": 256.0, "infinite": np.inf}[what]
    check(oracle, ctx, [base], q[:137], 10)
    if what != "infinite":
        check(oracle, ctx, [base], q, 10)
        return
    import ferrolm_b200 as fv

    ix = fv.FlatIndex(ctx, fv.Metric.L2, 56)
    ix.add(base)
    got, gc = ix.search_batch(q, 10)
    ix.set_mode(2)
    want, wc = ix.search_batch(q, 10)
    assert np.array_equal(gc, wc) and np.array_equal(got, want)


def test_rows_added_in_pieces(oracle, ctx):
    a, b = whole(4500, 72, 5, 100, 10), whole(901, 72, 5, 100, 11)
    q = whole(128, 72, 5, 100, 12)
    check(oracle, ctx, [a, b, b[:7]], q, 10)                      # the same form throughout
    check(oracle, ctx, [a, whole(300, 72, -100, 90, 13)], q, 10)  # another offset: the old rows are converted again
    check(oracle, ctx, [a, b + 0.25], q, 10)                      # no longer whole numbers
    check(oracle, ctx, [b[:200] + 0.25, a], q, 10)


def test_pieces_added_to_rows_that_do_not_fit(oracle, ctx):
    import ferrolm_b200 as fv

    dark = whole(4500, 128, 0, 100, 14)
    dark[5] = 0  # 128 x 127^2 is beyond the norm's bytes above 0, not above -128
    piece, q = whole(300, 128, 0, 100, 15), whole(200, 128, 0, 100, 16)
    check(oracle, ctx, [dark, piece, piece[:9]], q, 10)
    check(oracle, ctx, [dark, piece, whole(100, 128, -28, 100, 17), piece], q, 10)

    def launches(base):  # of the second and third add: the rows of before are not converted again
        ix = fv.FlatIndex(ctx, fv.Metric.L2, 128)
        ix.add(base)
        before = ctx.stats()["launches"]
        ix.add(piece)
        ix.add(piece)
        return ctx.stats()["launches"] - before

    assert launches(dark) == launches(dark + 0.5)
