"""Searches of an IVF-PQ index that holds no rows: trained and not yet filled, or loaded from such an index's file.  They
find nothing, whatever the kernel: no vector, code or id exists that could be read."""
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


@pytest.mark.parametrize("metric", [L2, IP])
@pytest.mark.parametrize("m", [4, 6, 16])
@pytest.mark.parametrize("loaded", [False, True])
def test_an_index_without_rows_finds_nothing(oracle, ctx, metric, m, loaded):
    import torch

    import ferrolm_b200 as fv

    dim = 48
    sample, q = oracle.testdata(600, dim, 1), oracle.testdata(300, dim, 2)
    ix = fv.IvfPq.train(ctx, metric, dim, sample, fv.IvfPqParams(20, m, 2, True, 1))
    if loaded:
        ix = fv.IvfPq.load(ctx, ix.save())
    for k, refine in ((10, 0), (10, 4), (32, 4), (40, 4)):  # kept in registers, up to 32 and up to 128 of them, and in the buffer
        for nq, nprobe in ((1, 20), (300, 3)):
            got, counts = ix.search_batch(q[:nq], k, nprobe, refine)
            assert (counts == 0).all() and (got["id"] == 0xFFFFFFFF).all() and np.isinf(got["distance"]).all()
            out, dc = ix.search_batch(torch.from_numpy(q[:nq]).cuda(), k, nprobe, refine)
            assert (dc == 0).all() and (fv.neighbors_from_tensor(out)["id"] == 0xFFFFFFFF).all()
    # the first rows make it an index like any other
    ix.add(sample)
    got, counts = ix.search_batch(sample[:5], 1, 20, 4)
    assert (counts == 1).all()
