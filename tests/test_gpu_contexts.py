"""Several contexts on one GPU, each with its own thread: what a kernel may take of shared memory is a property of the kernel,
not of a context, so calls of different sizes must not get in one another's way."""
import threading

import pytest

pytestmark = pytest.mark.gpu

L2 = 0


def side_by_side(jobs):
    """Runs every job in a thread of its own, all at once; raises what any of them raised."""
    start, failed = threading.Barrier(len(jobs)), []

    def run(job):
        start.wait()
        try:
            job()
        except Exception as e:  # noqa: BLE001 -- reported below
            failed.append(e)

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if failed:
        raise failed[0]


def test_graphs_of_different_dimensions_at_once(oracle):
    import ferrolm_b200 as fv

    # wide batches (a warp per node) and narrow ones (a team): a block takes 53 to 66 KB
    def build(ctx, base):
        return fv.Hnsw.build_batched(ctx, L2, base.shape[1], base, fv.HnswParams(16, 200, 1), max_batch=8192, divisor=1).save()

    bases = [oracle.testdata(6000, d, 1) for d in (24, 96, 200)]
    ctxs = [fv.Context(0) for _ in bases]
    want = [build(c, b) for c, b in zip(ctxs, bases)]
    got = [None] * len(bases)

    def job(i):
        def run():
            for _ in range(4):
                got[i] = build(ctxs[i], bases[i])
        return run

    side_by_side([job(i) for i in range(len(bases))])
    assert got == want
    for c in ctxs:
        c.close()


def test_searches_of_different_dimensions_at_once(oracle):
    import ferrolm_b200 as fv

    made = []
    for dim in (128, 168, 232):
        ctx = fv.Context(0)
        base, q = oracle.testdata(4200, dim, 1), oracle.testdata(2500, dim, 2)
        graph = fv.Hnsw.build_batched(ctx, L2, dim, base[:2000], fv.HnswParams(8, 60, 1))
        flat = fv.FlatIndex(ctx, L2, dim)
        flat.add(base)
        ivf = fv.IvfPq.train(ctx, L2, dim, base, fv.IvfPqParams(16, 8, 1, True, 1))
        ivf.add(base)
        calls = [lambda g=graph, q=q: g.search_batch(q, 10, 64), lambda f=flat, q=q: f.search_batch(q, 10),
                 lambda v=ivf, q=q: v.search_batch(q, 10, 4, 4)]
        made.append((ctx, calls, [c()[0].tobytes() for c in calls]))

    def job(calls, want):
        def run():
            for _ in range(60):
                for c, w in zip(calls, want):
                    assert c()[0].tobytes() == w
        return run

    side_by_side([job(calls, want) for _, calls, want in made])
    for ctx, _, _ in made:
        ctx.close()
