"""The device memory of server slots with coded tiles: bounded without a budget,
and all of it taken at the start."""
import numpy as np
import pytest

from launched import names_during
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu

N, NQ, K, S64 = 30_011, 1024, 10, 156      # a block of 128 queries is 1.5 launches of codes


@pytest.fixture(scope="module")
def references():
    import torch
    kmers = list(range(15, 35, 2))
    words = torch.randint(-2**63, 2**63 - 1, (N, K, S64 * 14), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx = capi.Context(0)
    ref = capi.Database(ctx, words.data_ptr(), kmers, S64, n_samples=N)
    qwords = words[:NQ].cpu().numpy().view(np.uint64)
    del words
    torch.cuda.empty_cache()
    yield ctx, ref, qwords
    ref.close()
    ctx.close()


def test_slots_without_a_budget_leave_the_device_its_memory(references):
    import torch
    ctx, ref, _ = references
    free = torch.cuda.mem_get_info()[0]
    server = capi.Server(ctx, ref, slots=16, slice_queries=256, kNN=3)
    used = free - torch.cuda.mem_get_info()[0]
    server.close()
    assert used < free // 4 + 16 * (600 << 20)


@pytest.mark.parametrize("sizes", [(1024,), (129, 200, 1, 700, 1024)])
def test_slices_allocate_nothing(references, sizes):
    ctx, ref, qwords = references
    server = capi.Server(ctx, ref, slots=1, slice_queries=1024, kNN=3)
    got = []

    def slices():
        for nq in sizes:
            t = server.submit(qwords[:nq])
            server.wait(t)
            got.append((nq, *server.result(t)[:2]))

    try:
        names = names_during(slices, repeats=1)
    finally:
        server.close()
    assert any("dist_items_kernel" in n for n in names)      # the profiler saw the calls
    assert not [n for n in names if n in ("cudaMalloc", "cudaFree")]
    qry = capi.Database(ctx, qwords, list(range(15, 35, 2)), S64)
    r, d = capi.query_knn(ctx, ref, qry, 3)
    qry.close()
    for nq, idx, dist in got:
        np.testing.assert_array_equal(idx, r[:nq])
        np.testing.assert_array_equal(dist, d[:nq])
