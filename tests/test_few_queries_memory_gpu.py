"""The workspace of the few-queries kernel: bounded whatever the number of
references, and no reason for a call to fail."""
import numpy as np
import pytest

from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu

PLAIN_SHAPE = 6      # a forced shape takes tiles


def _fill(leave):
    """Device memory taken so that about `leave` bytes are free."""
    import torch
    torch.cuda.empty_cache()
    hold = []
    for step in (1 << 30, 64 << 20, 2 << 20):
        while torch.cuda.mem_get_info()[0] - leave > step:
            hold.append(torch.empty((torch.cuda.mem_get_info()[0] - leave) // step * step,
                                    dtype=torch.uint8, device="cuda"))
    return hold


# counts of all references at once: 576 MB at K = 24 (the workspace holds 128),
# 102 MB at K = 4, which do not fit 60 MB, where tiles do
@pytest.mark.parametrize("n,nq,K,free_mb", [(100_100, 120, 24, 300), (100_100, 120, 4, 60),
                                            (70_001, 33, 24, 300), (262_657, 100, 5, 300)])
def test_counts_of_many_references_fit(n, nq, K, free_mb):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    kmers = list(range(13, 13 + 2 * K, 2))
    words = torch.randint(0, 16, (n + nq, K, 14), dtype=torch.int64, device="cuda", generator=gen)
    torch.cuda.synchronize()
    with capi.Context(0) as ctx:
        ref = capi.Database(ctx, words.data_ptr(), kmers, 1, n_samples=n)
        qry = capi.Database(ctx, words.data_ptr() + n * K * 14 * 8, kmers, 1, n_samples=nq)
        del words
        got = torch.zeros((n * nq, 2), dtype=torch.float32, device="cuda")
        want = torch.zeros_like(got)
        ctx.set_tile_config(PLAIN_SHAPE)
        capi.dists_dense(ctx, ref, qry, out=want.data_ptr())
        ctx.synchronize()
        ref.close()
        qry.close()
    gen = torch.Generator(device="cuda").manual_seed(n)
    words = torch.randint(0, 16, (n + nq, K, 14), dtype=torch.int64, device="cuda", generator=gen)
    torch.cuda.synchronize()
    with capi.Context(0) as ctx:
        ref = capi.Database(ctx, words.data_ptr(), kmers, 1, n_samples=n)
        qry = capi.Database(ctx, words.data_ptr() + n * K * 14 * 8, kmers, 1, n_samples=nq)
        one = capi.Database(ctx, words.data_ptr(), kmers, 1, n_samples=3)
        capi.dists_dense(ctx, one, one)          # the kernels are loaded
        del words
        hold = _fill(free_mb << 20)
        try:
            capi.dists_dense(ctx, ref, qry, out=got.data_ptr())
            ctx.synchronize()
        finally:
            del hold
            torch.cuda.empty_cache()
        assert torch.equal(got, want)
        for db in (ref, qry, one):
            db.close()


def test_server_slots_hold_no_counts_of_every_reference(gpu_ctx):
    """40,000 references at K = 24: the counts of 120 queries would be 230 MB, a
    slot's own buffers and tiles are 260; results as without a server."""
    import torch
    n, nq, K = 40_003, 120, 24
    gen = torch.Generator(device="cuda").manual_seed(9)
    kmers = list(range(13, 13 + 2 * K, 2))
    words = torch.randint(0, 16, (n + nq, K, 14), dtype=torch.int64, device="cuda", generator=gen)
    torch.cuda.synchronize()
    ref = capi.Database(gpu_ctx, words.data_ptr(), kmers, 1, n_samples=n)
    hq = words[n:].cpu().numpy().view(np.uint64)
    server = capi.Server(gpu_ctx, ref, slots=1, slice_queries=128, kNN=6)
    try:
        assert server.info()["slot_bytes"] < 290 << 20
        t = server.submit(hq)
        server.wait(t)
        idx, dist = server.result(t)[:2]
    finally:
        server.close()
    r, d = capi.query_knn(gpu_ctx, ref, capi.Database(gpu_ctx, hq, kmers, 1), 6)
    np.testing.assert_array_equal(idx, r)
    np.testing.assert_array_equal(dist, d)
