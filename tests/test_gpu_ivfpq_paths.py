"""The per-query IVF-PQ scan over its branches: code loads of 4, 2 and 1 words and of single bytes, results in registers
(up to 32, up to 128 kept) and in the block's buffer, one and several blocks per query; against the oracle."""
import numpy as np
import pytest

from tests.parity import assert_same_neighbours

pytestmark = pytest.mark.gpu

L2, IP = 0, 1


@pytest.fixture(scope="module")
def made(oracle):
    import ferrolm_b200 as fv

    ctx = fv.Context(0)
    cache = {}

    def get(metric, m):
        if (metric, m) not in cache:
            dim = 96
            base = oracle.testdata(5000, dim, 3)
            base[100:140] = base[99]  # rows that tie, at the cut of some queries' lists too
            if metric == IP:
                base = oracle.normalize(base)
            ix = fv.IvfPq.train(ctx, metric, dim, base[:1500], fv.IvfPqParams(20, m, 3, True, 1))
            ix.add(base)
            ix.set_scan_mode(1)
            q = np.concatenate([base[99:100], oracle.testdata(699, dim, 4)])
            cache[metric, m] = ix, oracle.IvfPq.load(ix.save()), oracle.normalize(q) if metric == IP else q
        return cache[metric, m]

    yield get
    cache.clear()
    ctx.close()


@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("m", [6, 4, 8, 16, 24, 48])
@pytest.mark.parametrize("k,refine", [(1, 0), (32, 0), (33, 0), (128, 0), (129, 0), (8, 4), (32, 4), (33, 3), (10, 12), (10, 13), (65, 8)])
def test_scan_equals_the_oracle(made, metric, m, k, refine):
    ix, o, q = made(metric, m)
    for nq, nprobe in ((1, 20), (3, 7), (40, 1), (700, 3)):
        got, gc = ix.search_batch(q[:nq], k, nprobe, refine)
        want, wc = o.search_batch(q[:nq], k, nprobe, refine)
        bits, total = assert_same_neighbours(got, gc, want, wc, f"m={m} nq={nq} nprobe={nprobe}")
        assert bits == total


@pytest.mark.parametrize("k,refine", [(10, 0), (32, 8), (10, 10), (40, 4), (10, 40)])
def test_tensor_pass_finish_equals_the_per_query_scan(made, k, refine):
    ix, _, q = made(L2, 16)
    ix.set_scan_mode(1)
    want, wc = ix.search_batch(q, k, 12, refine)
    for mode in (3, 4):
        ix.set_scan_mode(mode)
        got, gc = ix.search_batch(q, k, 12, refine)
        assert np.array_equal(gc, wc) and np.array_equal(got, want), f"mode {mode}"
    ix.set_scan_mode(1)


# the block finishing kernel: k (refine + 1) keys lie before the query it reads 16 bytes at a time, an odd number here
@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("k,refine,slots", [(33, 4, 0), (35, 2, 0), (31, 10, 0), (7, 10, 80), (1, 4, 8)])
def test_block_finish_of_odd_results(made, metric, k, refine, slots):
    ix, o, q = made(metric, 16)
    want, wc = o.search_batch(q, k, 12, refine)
    ix.set_candidate_slots(slots)  # (few slots: the buffers run over and go to the block kernel too)
    for mode in (2, 3):
        ix.set_scan_mode(mode)
        got, gc = ix.search_batch(q, k, 12, refine)
        bits, total = assert_same_neighbours(got, gc, want, wc, f"mode {mode}")
        assert bits == total
    ix.set_candidate_slots(0)
    ix.set_scan_mode(1)


# the finishing step's queries and selected ids in shared memory: at and beyond the 48 KB a launch has unasked, and
# beyond what an SM has
@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("dim,k,refine", [(1520, 10, 0), (1536, 10, 0), (1536, 10, 4), (1408, 32, 8), (8000, 10, 4)])
def test_table_scan_of_long_vectors(oracle, metric, dim, k, refine):
    import ferrolm_b200 as fv

    ctx = fv.Context(0)
    base, q = oracle.testdata(1500, dim, 3), oracle.testdata(40, dim, 4)
    ix = fv.IvfPq.train(ctx, metric, dim, base[:300], fv.IvfPqParams(8, 16, 1, True, 1))
    ix.add(base)
    want, wc = oracle.IvfPq.load(ix.save()).search_batch(q, k, 4, refine)
    for mode in (1, 2):
        ix.set_scan_mode(mode)
        got, gc = ix.search_batch(q, k, 4, refine)
        bits, total = assert_same_neighbours(got, gc, want, wc, f"mode {mode}")
        assert bits == total
    ctx.close()


@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("k,refine", [(10, 0), (32, 0), (10, 4), (8, 10)])
def test_a_file_that_holds_ids_more_than_once(made, oracle, metric, k, refine):
    import ferrolm_b200 as fv

    ix, _, q = made(metric, 16)
    data = bytearray(ix.save())
    nlist, m, dim = 20, 16, 96
    at = 8 + 5 * 4 + 8 + nlist * dim * 4 + 8 + m * 256 * (dim // m) * 4
    for _ in range(nlist):  # per list: count, ids, bytes of codes, codes; the first 60 rows become copies of the first
        n = int.from_bytes(data[at : at + 8], "little")
        c, d = at + 8 + 4 * n + 8, min(n, 60)
        data[at + 8 : at + 8 + 4 * d] = bytes(data[at + 8 : at + 12]) * d
        data[c : c + m * d] = bytes(data[c : c + m]) * d
        at = c + n * m
    ctx = fv.Context(0)
    dup, o = fv.IvfPq.load(ctx, bytes(data)), oracle.IvfPq.load(bytes(data))
    want, wc = o.search_batch(q, k, 5, refine)
    for mode in (1, 2, 3):
        dup.set_scan_mode(mode)
        got, gc = dup.search_batch(q, k, 5, refine)
        bits, total = assert_same_neighbours(got, gc, want, wc, f"mode {mode}")
        assert bits == total
    ctx.close()


# 4,096 lists and more are looked for by the tensor-core front end: up to 32 probes, and from 33 with its long results
@pytest.mark.parametrize("metric", [L2, IP])
def test_many_probes_of_many_lists(oracle, metric):
    import ferrolm_b200 as fv

    ctx = fv.Context(0)
    base, q = oracle.testdata(9000, 32, 3), oracle.testdata(300, 32, 4)
    if metric == IP:
        base, q = oracle.normalize(base), oracle.normalize(q)
    ix = fv.IvfPq.train(ctx, metric, 32, base, fv.IvfPqParams(4100, 8, 1, True, 1))
    ix.add(base)
    o = oracle.IvfPq.load(ix.save())
    for nprobe in (32, 33, 100, 128, 129):
        got, gc = ix.search_batch(q, 10, nprobe, 4)
        launches = ctx.stats()["launches"]
        want, wc = o.search_batch(q, 10, nprobe, 4)
        bits, total = assert_same_neighbours(got, gc, want, wc, f"{nprobe} probes")
        assert bits == total
        # tables, scan and conversion; the coarse step's passes besides
        assert (launches >= 8) == (nprobe <= 128), launches
    ctx.close()


@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("nq,nprobe", [(341, 3), (1024, 1), (2560, 8), (2561, 8), (4096, 8), (4097, 8), (1725, 19)])
def test_pairs_are_filed_by_one_thread_each_and_by_blocks(made, metric, nq, nprobe):
    # up to 20,480 pairs and beyond; whole and partial blocks
    ix, _, q = made(metric, 16)
    q = np.concatenate([q] * 6)[:nq]
    ix.set_scan_mode(1)
    want, wc = ix.search_batch(q, 10, nprobe, 0)
    ix.set_scan_mode(3)
    got, gc = ix.search_batch(q, 10, nprobe, 0)
    ix.set_scan_mode(1)
    assert np.array_equal(gc, wc) and np.array_equal(got, want)
