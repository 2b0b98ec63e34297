"""A few queries against every reference (query_kernel.cu): group sizes and
remainders, reference counts around the 4-, 128- and 512-column edges, odd
sketch widths, every output and correction, against the oracle and against the
tiles that a forced shape takes; and the kNN lists over short and long rows."""
import numpy as np
import pytest

import oracle
from conftest import random_sketches
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,n,K,s64", [
    (1, 1, 8, 156), (1, 130, 3, 1), (2, 513, 4, 3), (3, 127, 1, 17), (4, 512, 2, 16),
    (5, 200, 32, 2), (8, 1029, 5, 5), (9, 64, 2, 33), (13, 300, 3, 4), (17, 129, 2, 8),
    (25, 600, 2, 3), (32, 100, 2, 64), (33, 1000, 1, 2), (70, 1100, 2, 3), (100, 1003, 1, 5),
])
def test_counts_match_oracle(gpu_ctx, nq, n, K, s64):
    w, kmers = random_sketches(n + nq, K, s64, seed=nq + n)
    ref = capi.Database(gpu_ctx, w[:n], kmers, s64)
    qry = capi.Database(gpu_ctx, w[n:], kmers, s64)
    got = capi.dists_dense(gpu_ctx, ref, qry, out_mode=capi.OUT_COUNTS)
    np.testing.assert_array_equal(got, oracle.dists(w[:n], kmers, s64, query_words=w[n:],
                                                    out_mode=2))


@pytest.mark.parametrize("mode,semantics", [("none", 0), ("table", 0), ("equal", 0), ("table", 1)])
def test_equals_tiles(mode, semantics):
    n, nq, K, s64 = 1500, 19, 6, 8
    w, kmers = random_sketches(n + nq, K, s64, seed=5)
    rng = np.random.default_rng(6)
    lens = rng.integers(1_000_000, 4_000_000, n + nq).astype(np.uint64)
    cl = rng.integers(0, 3, n + nq).astype(np.uint16)
    with capi.Context(0) as ctx:
        ctx.set_semantics(semantics)
        ref = capi.Database(ctx, w[:n], kmers, s64, cluster=cl[:n], seq_len=lens[:n])
        qry = capi.Database(ctx, w[n:], kmers, s64, cluster=cl[n:], seq_len=lens[n:])
        rnd = None
        if mode == "table":
            rnd = capi.Random(ctx, capi.RANDOM_TABLE, kmers,
                              table=rng.uniform(0, 0.02, (K, 3, 3)).astype(np.float32))
        elif mode == "equal":
            rnd = capi.Random(ctx, capi.RANDOM_EQUAL_BASE, kmers)

        def forms():
            out = [capi.dists_dense(ctx, ref, qry, rnd, out_mode=m)
                   for m in (capi.OUT_CORE_ACC, capi.OUT_JACCARD)]
            out += capi.query_knn(ctx, ref, qry, 7, random=rnd)
            ctx.set_memory_limit(200_000)     # the query side in row blocks too
            out.append(capi.dists_dense(ctx, ref, qry, rnd))
            ctx.set_memory_limit(0)
            return out

        few = forms()
        ctx.set_tile_config(1)
        for a, b in zip(few, forms()):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,knn", [(2, 2), (33, 33), (257, 1), (600, 40), (2100, 300), (900, 800)])
def test_knn_lists(gpu_ctx, n, knn):
    """Self and row lists against a stable sort by (distance, sample)."""
    w, kmers = random_sketches(n + 3, 3, 1, seed=n)     # narrow sketches: many equal distances
    ref = capi.Database(gpu_ctx, w[:n], kmers, 1)
    qry = capi.Database(gpu_ctx, w[n:], kmers, 1)
    sq = np.full((n, n), np.inf, np.float32)
    iu = np.triu_indices(n, 1)
    sq[iu] = sq.T[iu] = capi.dists_dense(gpu_ctx, ref)[:, 0]
    _, j, d = capi.dists_knn(gpu_ctx, ref, knn)
    order = np.argsort(sq, axis=1, kind="stable")[:, :knn]
    np.testing.assert_array_equal(j.reshape(n, knn), order)
    np.testing.assert_array_equal(d.reshape(n, knn), np.take_along_axis(sq, order, 1))
    rows = capi.dists_dense(gpu_ctx, ref, qry)[:, 0].reshape(3, n)
    r, d = capi.query_knn(gpu_ctx, ref, qry, knn)
    order = np.argsort(rows, axis=1, kind="stable")[:, :knn]
    np.testing.assert_array_equal(r, order)
    np.testing.assert_array_equal(d, np.take_along_axis(rows, order, 1))
