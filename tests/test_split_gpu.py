"""Tiles cut into parts: jobs of few tiles (every tile cut), tile edges of both
shapes, narrow and wide sketches, and batches whose tiles differ in cost, all
against the oracle (counts exactly, core/accessory within 1e-6 of its fit)."""
import numpy as np
import pytest

import oracle
from conftest import random_sketches
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,K,s64", [
    (2, None, 8, 156), (63, None, 8, 156), (65, None, 5, 17), (128, None, 1, 1),
    (129, None, 4, 3), (193, None, 3, 64), (70, None, 33, 2), (40, None, 2, 1030),
    (1, 1, 8, 156), (130, 65, 7, 16), (400, 150, 5, 156), (64, 64, 9, 1),
])
def test_cut_tiles_match_oracle(gpu_ctx, n, nq, K, s64):
    w, kmers = random_sketches(n + (nq or 0), K, s64, seed=n + K)
    ref = capi.Database(gpu_ctx, w[:n], kmers, s64)
    qry = None if nq is None else capi.Database(gpu_ctx, w[n:], kmers, s64)
    qw = None if nq is None else w[n:]
    np.testing.assert_array_equal(
        capi.dists_dense(gpu_ctx, ref, qry, out_mode=capi.OUT_COUNTS),
        oracle.dists(w[:n], kmers, s64, query_words=qw, out_mode=2))
    np.testing.assert_allclose(capi.dists_dense(gpu_ctx, ref, qry),
                               oracle.dists(w[:n], kmers, s64, query_words=qw), rtol=0, atol=1e-6)


@pytest.mark.parametrize("shapes", [
    [(300, 12, 312), (500, 4, 16), (60, 8, 156)],             # a few costly tiles among cheap ones
    [(200, 40, 8), (300, 8, 64), (64, 2, 1030), (129, 5, 16)],  # wide and narrow jobs in one launch
])
def test_batch_of_unequal_tiles(gpu_ctx, shapes):
    import torch
    made = []
    for i, (n, K, s64) in enumerate(shapes):
        w, kmers = random_sketches(n, K, s64, seed=50 + i)
        out = torch.zeros((n * (n - 1) // 2, K), dtype=torch.int32, device="cuda")
        made.append((capi.Database(gpu_ctx, w, kmers, s64), out, w, kmers, s64))
    torch.cuda.synchronize()
    b = capi.Batch(gpu_ctx, [(db, None, None, capi.OUT_COUNTS, o.data_ptr())
                             for db, o, *_ in made])
    b.run()
    for _, out, w, kmers, s64 in made:
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32),
                                      oracle.dists(w, kmers, s64, out_mode=2))
    b.close()
