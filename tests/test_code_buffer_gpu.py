"""The buffer a context keeps for coded tiles: calls queued one behind another
that share it, and calls that need its memory for something else."""
import numpy as np
import pytest

from conftest import random_sketches
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu


def test_a_call_from_host_memory_waits_for_the_queued_one():
    """Distances into device memory are only queued; the call from host sketches
    that follows writes its column values to the same buffer from a stream of
    its own, and must not do so while the first call still reads there."""
    import torch
    K, s64 = 8, 64
    w, kmers = random_sketches(3000, K, s64, seed=12)
    v, _ = random_sketches(1800, K, s64, seed=13)
    with capi.Context(0) as ctx:
        db = capi.Database(ctx, w, kmers, s64)
        out = torch.empty((3000 * 2999 // 2, 2), dtype=torch.float32, device="cuda")
        want = capi.dists_dense(ctx, db)
        want_host = capi.query_db(ctx, v, kmers, s64)
        for _ in range(3):
            out.zero_()
            torch.cuda.synchronize()
            for _ in range(20):
                capi.dists_dense(ctx, db, out=out.data_ptr())
            got_host = capi.query_db(ctx, v, kmers, s64)
            ctx.synchronize()
            np.testing.assert_array_equal(out.cpu().numpy(), want)
            np.testing.assert_array_equal(got_host, want_host)
