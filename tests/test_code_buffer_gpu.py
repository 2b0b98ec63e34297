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


def test_memory_kept_for_codes_is_given_back(gpu_ctx):
    """A database, and a server, that fit beside the code buffer's context only
    without the buffer."""
    import torch
    K, s64 = 8, 156
    kmers = list(range(15, 31, 2))
    words = torch.randint(-2**63, 2**63 - 1, (1800, K, s64 * 14), dtype=torch.int64, device="cuda")
    out = torch.empty((1800 * 1799 // 2, 2), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    for use in ("database", "server"):
        with capi.Context(0) as ctx:
            db = capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=1800)
            capi.dists_dense(ctx, db, out=out.data_ptr())
            ctx.synchronize()
            hold = _fill(100 << 20)
            try:
                if use == "database":        # 143 MB
                    more = capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=1000)
                    more.close()
                else:                        # more than that for its one slot
                    server = capi.Server(ctx, db, slots=1, slice_queries=64, kNN=2)
                    server.close()
            finally:
                del hold
                torch.cuda.empty_cache()
            db.close()


def test_codes_do_not_take_the_memory_of_needed_buffers():
    """1,700 samples at K = 24 need 204 MB of counts and, to be coded, 35 MB more:
    in 220 MB the call goes without codes."""
    import torch
    n, K, s64 = 1700, 24, 1
    w, kmers = random_sketches(n, K, s64, seed=15)
    out = torch.empty((n * (n - 1) // 2, 2), dtype=torch.float32, device="cuda")
    with capi.Context(0) as ctx:             # loads every kernel, and the result
        db = capi.Database(ctx, w, kmers, s64)
        ctx.set_tile_config(6)
        want = capi.dists_dense(ctx, db)
        ctx.set_tile_config(0)
        np.testing.assert_array_equal(capi.dists_dense(ctx, db), want)
        db.close()
    with capi.Context(0) as ctx:
        db = capi.Database(ctx, w, kmers, s64)
        torch.cuda.synchronize()
        hold = _fill(220 << 20)
        try:
            capi.dists_dense(ctx, db, out=out.data_ptr())
            ctx.synchronize()
        finally:
            del hold
            torch.cuda.empty_cache()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
        db.close()


def test_blocked_output_at_the_default_budget():
    """13,000 samples to the host, 676 MB, with 1.2 GB of the device free: row
    blocks in half of that."""
    import torch
    n, K, s64 = 13_000, 3, 4
    kmers = [15, 17, 19]
    gen = torch.Generator(device="cuda").manual_seed(3)
    words = torch.randint(0, 2**40, (n, K, s64 * 14), dtype=torch.int64, device="cuda", generator=gen)
    out = torch.empty((n * (n - 1) // 2, 2), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with capi.Context(0) as ctx:
        db = capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=n)
        capi.dists_dense(ctx, db, out=out.data_ptr())
        ctx.synchronize()
        db.close()
    want = out.cpu().numpy()
    del out
    with capi.Context(0) as ctx:
        db = capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=n)
        hold = _fill(1200 << 20)
        try:
            got = capi.dists_dense(ctx, db)
        finally:
            del hold
            torch.cuda.empty_cache()
        db.close()
    np.testing.assert_array_equal(got, want)
