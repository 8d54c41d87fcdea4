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


# a scouting team's room ends first (57,2xx), then a team's visited set; 57,848 is the most that a team has room for
@pytest.mark.parametrize("dim", [50_000, 57_200, 57_800, 57_848])
@pytest.mark.parametrize("metric", [L2, IP])
def test_search_of_long_rows(oracle, ctx, metric, dim):
    import ferrolm_b200 as fv

    base, q = oracle.testdata(40, dim, 1), oracle.testdata(5, dim, 2)
    g = fv.Hnsw.build(ctx, metric, dim, base, fv.HnswParams(4, 20, 1))
    same(g.search_batch(q, 5, 20), oracle.Hnsw.load(g.save()).search_batch(q, 5, 20))


@pytest.mark.parametrize("dim", [28_600, 28_700, 28_832])
def test_construction_of_long_rows(oracle, ctx, dim):
    import ferrolm_b200 as fv

    base = oracle.testdata(30, dim, 3)
    g = fv.Hnsw.build_batched(ctx, L2, dim, base, fv.HnswParams(4, 20, 1), max_batch=4, divisor=4)
    assert g.save() == oracle.Hnsw.build_batched(L2, dim, base, m=4, ef_construction=20, seed=1, max_batch=4, divisor=4).save()
    with pytest.raises(fv.FerrovecError):
        fv.Hnsw.build_batched(ctx, L2, 28_840, np.zeros((30, 28_840), np.float32), fv.HnswParams(4, 20, 1))


def widened(data, m):
    """An FLHNSW01 file with room for 2 m links per node instead of its own."""
    own = int.from_bytes(data[16:20], "little")
    n = int.from_bytes(data[28:36], "little")
    at = 36 + n
    words = np.frombuffer(data, dtype=np.uint32, count=n * (2 * own + 1), offset=at + 8).reshape(n, 2 * own + 1)
    wide = np.zeros((n, 2 * m + 1), np.uint32)
    wide[:, : 2 * own + 1] = words
    return (data[:16] + m.to_bytes(4, "little") + data[20:at] + (n * (2 * m + 1)).to_bytes(8, "little") + wide.tobytes()
            + data[at + 8 + words.nbytes :])


@pytest.mark.parametrize("m", [100, 1000, 4000])
def test_files_with_long_link_lists(oracle, ctx, m):
    import ferrolm_b200 as fv

    base, q = oracle.testdata(600, 24, 4), oracle.testdata(900, 24, 5)
    data = widened(fv.Hnsw.build_batched(ctx, L2, 24, base, fv.HnswParams(8, 40, 1)).save(), m)
    g, o = fv.Hnsw.load(ctx, data), oracle.Hnsw.load(data)
    assert g.save() == data
    for nq, ef in ((3, 20), (900, 20), (20, 300)):
        same(g.search_batch(q[:nq], 10, ef), o.search_batch(q[:nq], 10, ef))


@pytest.mark.parametrize("dim", [1016, 1024])
def test_short_beams_over_long_rows(oracle, ctx, dim):
    # scouting teams up to 1,023 dimensions or from beams of 33 on, teams of eight otherwise
    import ferrolm_b200 as fv

    base, q = oracle.testdata(900, dim, 6), oracle.testdata(40, dim, 7)
    g = fv.Hnsw.build_batched(ctx, IP, dim, base, fv.HnswParams(8, 32, 1))
    assert g.save() == oracle.Hnsw.build_batched(IP, dim, base, m=8, ef_construction=32, seed=1).save()
    o = oracle.Hnsw.load(g.save())
    for ef in (10, 32, 33):
        same(g.search_batch(q, 10, ef), o.search_batch(q, 10, ef))


@pytest.mark.parametrize("metric,m", [(L2, 17), (IP, 24), (L2, 32), (L2, 33)])
def test_links_of_scouting_teams(oracle, ctx, metric, m):
    # 34 to 64 links per node are looked at in two turns, 66 are beyond scouting teams; batches and queries on both sides of two
    # per SM (148 SMs), beams on both sides of registers
    import ferrolm_b200 as fv

    base, q = oracle.testdata(2600, 40, 8), oracle.testdata(297, 40, 9)
    g = fv.Hnsw.build_batched(ctx, metric, 40, base, fv.HnswParams(m, 60, 1), max_batch=600, divisor=4)
    assert g.save() == oracle.Hnsw.build_batched(metric, 40, base, m=m, ef_construction=60, seed=1, max_batch=600, divisor=4).save()
    o = oracle.Hnsw.load(g.save())
    for ef in (20, 100, 256, 257):
        want, wc = o.search_batch(q, 10, ef)
        for nq in (1, 296, 297):
            same(g.search_batch(q[:nq], 10, ef), (want[:nq], wc[:nq]))
