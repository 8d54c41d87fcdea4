"""Searches and trainings on a device with little room: a workspace that cannot be had is done without."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L2, IP = 0, 1


@contextlib.contextmanager
def at_most(nbytes):
    from ferrolm_b200._lib import check, lib

    check(lib().fv_debug_alloc_limit(nbytes))
    try:
        yield
    finally:
        check(lib().fv_debug_alloc_limit(0))


@pytest.fixture()
def ctx():
    import ferrolm_b200 as fv

    c = fv.Context(0)  # one per test: workspaces stay with their context
    yield c
    c.close()


@pytest.mark.parametrize("metric,k", [(L2, 10), (IP, 2), (L2, 40)])
def test_search_of_few_rows_without_room_for_every_key(oracle, ctx, metric, k):
    import ferrolm_b200 as fv

    base, q = oracle.testdata(4000, 48, 1), oracle.testdata(3000, 48, 2)
    ix = fv.FlatIndex(ctx, metric, 48)
    ix.add(base)
    with at_most(16 << 20):  # the keys take 96 MB
        got, gc = ix.search_batch(q, k)
    want, wc = ix.search_batch(q, k)
    assert got.tobytes() == want.tobytes() and (gc == wc).all()
    o = oracle.FlatIndex(metric, 48)
    o.add(base)
    assert o.search_batch(q[:100], k)[0].tobytes() == want[:100].tobytes()


def test_search_of_few_rows_in_several_runs(oracle, ctx):
    import ferrolm_b200 as fv

    # the keys of at most 8,388 queries of 4,000 rows are written at a time: two runs
    base, q = oracle.testdata(4000, 24, 1), oracle.testdata(9001, 24, 2)
    ix = fv.FlatIndex(ctx, L2, 24)
    ix.add(base)
    got, gc = ix.search_batch(q, 33)
    o = oracle.FlatIndex(L2, 24)
    o.add(base)
    want, wc = o.search_batch(q, 33)
    assert got.tobytes() == want.tobytes() and (gc == wc).all()


@pytest.mark.parametrize("m,limit", [(16, 2 << 20), (16, 1_800_000), (12, 2_000_000)])
def test_training_without_room_for_all_sub_quantizers(oracle, ctx, m, limit):
    import ferrolm_b200 as fv

    dim = m * 4  # sub-vectors of 4 are padded to 8: together twice the sample's size (3.5 MB at m = 16)
    sample = oracle.testdata(6000, dim, 1)
    p = fv.IvfPqParams(20, m, 2, True, 1)
    with at_most(limit):
        small = fv.IvfPq.train(ctx, L2, dim, sample, p)
    assert small.save() == fv.IvfPq.train(ctx, L2, dim, sample, p).save()


def test_what_cannot_be_done_without_is_an_error(oracle, ctx):
    import ferrolm_b200 as fv
    from ferrolm_b200._lib import FV_ERR_NOMEM

    with at_most(1 << 20), pytest.raises(fv.FerrovecError) as e:
        fv.IvfPq.train(ctx, L2, 64, oracle.testdata(6000, 64, 1), fv.IvfPqParams(20, 16, 2, True, 1))
    assert e.value.status == FV_ERR_NOMEM
    assert len(fv.IvfPq.train(ctx, L2, 64, oracle.testdata(6000, 64, 1), fv.IvfPqParams(20, 16, 2, True, 1))) == 0


@contextlib.contextmanager
def allocations(count):
    from ferrolm_b200._lib import check, lib

    check(lib().fv_debug_alloc_count(count))
    try:
        yield
    finally:
        check(lib().fv_debug_alloc_count(-1))


def rows(oracle, kind, n, seed):
    x = oracle.testdata(n, 40, seed)
    return np.rint(x * 8).clip(-100, 100).astype(np.float32) if kind == "whole" else x


@pytest.mark.parametrize("metric,kind", [(L2, "any"), (L2, "whole"), (IP, "any")])
def test_an_add_that_is_refused_at_any_of_its_allocations(oracle, ctx, metric, kind):
    import ferrolm_b200 as fv
    from ferrolm_b200._lib import FV_ERR_NOMEM

    a, b, q = rows(oracle, kind, 5000, 1), rows(oracle, kind, 6000, 2), rows(oracle, kind, 300, 3)
    o = oracle.FlatIndex(metric, 40)
    o.add(a)
    before, _ = o.search_batch(q, 10)
    o.add(b)
    after, _ = o.search_batch(q, 10)
    for count in range(40):
        ix = fv.FlatIndex(ctx, metric, 40)
        ix.add(a)
        assert ix.search_batch(q, 10)[0].tobytes() == before.tobytes()
        try:
            with allocations(count):
                ix.add(b)
        except fv.FerrovecError as e:
            assert e.status == FV_ERR_NOMEM
            assert len(ix) == 5000 and ix.search_batch(q, 10)[0].tobytes() == before.tobytes(), count
            ix.add(b)
            assert len(ix) == 11000 and ix.search_batch(q, 10)[0].tobytes() == after.tobytes(), count
            continue
        assert count > 5 and ix.search_batch(q, 10)[0].tobytes() == after.tobytes()
        break
    else:
        raise AssertionError("the add was never taken")


def test_an_add_does_without_room_for_bytes(oracle, ctx):
    import ferrolm_b200 as fv

    def taken(kind, count):
        a, b = rows(oracle, kind, 5000, 1), rows(oracle, kind, 6000, 2)
        ix = fv.FlatIndex(ctx, L2, 40)
        ix.add(a)
        try:
            with allocations(count):
                ix.add(b)
        except fv.FerrovecError:
            return None
        return ix, np.concatenate([a, b])

    least = next(count for count in range(40) if taken("any", count))
    q = rows(oracle, "whole", 300, 3)
    for count in range(least, least + 7):  # none to all of the five pieces that the bytes take
        ix, both = taken("whole", count)
        o = oracle.FlatIndex(L2, 40)
        o.add(both)
        assert ix.search_batch(q, 10)[0].tobytes() == o.search_batch(q, 10)[0].tobytes(), count
        more = rows(oracle, "whole", 700, 4)  # with room again
        ix.add(more)
        o.add(more)
        assert ix.search_batch(q, 10)[0].tobytes() == o.search_batch(q, 10)[0].tobytes(), count


@pytest.mark.parametrize("kind", ["any", "whole"])
def test_search_without_room_for_the_samples_minima(oracle, ctx, kind):
    import ferrolm_b200 as fv

    base, q = rows(oracle, kind, 40_000, 5), rows(oracle, kind, 2900, 6)
    ix = fv.FlatIndex(ctx, L2, 40)
    ix.add(base)
    ix.search_batch(q, 100)  # everything but the minima, which are a quarter of those below (a coarser sample)
    with at_most(3_000_000):  # 3,072 queries' minima take 7.9 MB
        got, gc = ix.search_batch(q, 10)
    want, wc = ix.search_batch(q, 10)
    assert got.tobytes() == want.tobytes() and (gc == wc).all()
    o = oracle.FlatIndex(L2, 40)
    o.add(base)
    assert o.search_batch(q[:200], 10)[0].tobytes() == want[:200].tobytes()
