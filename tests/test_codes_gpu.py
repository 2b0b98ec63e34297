"""Coded tiles (bin values rewritten as dictionary codes per block of 128 rows)
against the oracle and against the plain planes, which a forced tile shape
without a coded instance still compares: the results are the same integers, so
everything derived from them is the same bits."""
import numpy as np
import pytest

import oracle
from conftest import random_sketches
from sketchlib_b200 import capi, synth

pytestmark = pytest.mark.gpu

PLAIN_SHAPE = 6      # 64 x 64 tiles: no coded instance


def _sketches(kind, n, K, s64, seed):
    rng = np.random.default_rng(seed)
    kmers = np.arange(15, 15 + 2 * K, 2, dtype=np.int32)
    if kind == "tree":
        return random_sketches(n, K, s64, seed)
    if kind == "unrelated":          # up to 128 distinct values in a block: 8 planes
        return rng.integers(0, 2 ** 64, (n, K, s64 * 14), dtype=np.uint64), kmers
    one = rng.integers(0, 2 ** 64, (1, K, s64 * 14), dtype=np.uint64)
    w = np.repeat(one, n, axis=0)    # one value per bin
    if kind == "two":                # or a second one in every third sample
        w[::3] ^= np.uint64(1)
    return w, kmers


@pytest.mark.parametrize("kind", ["tree", "unrelated", "same", "two"])
@pytest.mark.parametrize("n,nq,K,s64", [
    (1700, None, 2, 1), (1793, None, 1, 7), (1921, None, 3, 3),
    (1000, 129, 2, 5), (1153, 257, 1, 2), (1664, 640, 2, 1),
])
def test_coded_counts_match_oracle(gpu_ctx, kind, n, nq, K, s64):
    w, kmers = _sketches(kind, n + (nq or 0), K, s64, seed=n + K)
    ref = capi.Database(gpu_ctx, w[:n], kmers, s64)
    qry = None if nq is None else capi.Database(gpu_ctx, w[n:], kmers, s64)
    got = capi.dists_dense(gpu_ctx, ref, qry, out_mode=capi.OUT_COUNTS)
    want = oracle.dists(w[:n], kmers, s64, query_words=None if nq is None else w[n:], out_mode=2)
    np.testing.assert_array_equal(got, want)


def _forms(ctx, ref, qry, rnd, w, n, kmers, s64):
    """Every entry point that takes the coded path, as arrays."""
    out = [capi.dists_dense(ctx, ref, None, rnd), capi.dists_dense(ctx, ref, qry, rnd),
           capi.dists_dense(ctx, ref, None, rnd, out_mode=capi.OUT_JACCARD)]
    out += capi.dists_knn(ctx, ref, 5, random=rnd)
    out += capi.dists_knn(ctx, ref, 3, dist_col=1, jaccard=True, random=rnd)
    out += capi.query_knn(ctx, ref, qry, 4, dist_col=1, random=rnd)
    out += capi.dists_threshold(ctx, ref, 0, 0.02, random=rnd)
    out.append(capi.query_db(ctx, w[:n], kmers, s64, random=rnd))
    out.append(capi.query_db(ctx, w[:n], kmers, s64, query_words=w[n:], random=rnd))
    ctx.set_memory_limit(2_000_000)          # dense output and kNN in row blocks
    out.append(capi.dists_dense(ctx, ref, None, rnd))
    out += capi.dists_knn(ctx, ref, 5, random=rnd)
    ctx.set_memory_limit(0)
    return out


@pytest.mark.parametrize("mode,semantics", [("none", 0), ("table", 0), ("equal", 0), ("table", 1)])
def test_coded_equals_plain(mode, semantics):
    n, nq, K, s64 = 1800, 300, 5, 4
    w, kmers = random_sketches(n + nq, K, s64, seed=3)
    rng = np.random.default_rng(4)
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
        coded = _forms(ctx, ref, qry, rnd, w, n, kmers, s64)
        ctx.set_tile_config(PLAIN_SHAPE)
        plain = _forms(ctx, ref, qry, rnd, w, n, kmers, s64)
        for i, (a, b) in enumerate(zip(coded, plain)):
            np.testing.assert_array_equal(a, b, err_msg=f"form {i}")


def test_codes_in_several_launches():
    """Codes above the buffer's limit: an all-vs-all in several launches (20 GB
    of codes, 8 GiB kept), and a server slot whose 2 GiB take a row block's
    columns in parts; both against the plain planes."""
    import torch
    kmers = list(range(13, 41, 2))           # K = 14 at 312 words: 36 MB per group
    n, nq, s64 = 8200, 200, 312
    p, t = synth.clade_tree(n + nq, kmers=kmers, seed=11)
    with capi.Context(0) as ctx:
        words = torch.empty((n + nq, len(kmers), s64 * 14), dtype=torch.int64, device="cuda")
        capi.synth_device(ctx, p, t, s64, seed=11, d_words=words.data_ptr())
        torch.cuda.synchronize()
        sub = capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=4200)
        ref = capi.Database(ctx, words.data_ptr(), kmers, s64, n_samples=n)
        qwords = words[n:].cpu().numpy().view(np.uint64)
        qry = capi.Database(ctx, qwords, kmers, s64)
        del words
        server = capi.Server(ctx, ref, slots=1, slice_queries=200, kNN=4)
        ticket = server.submit(qwords)
        server.wait(ticket)
        served = server.result(ticket)[:2]
        server.close()
        coded = [capi.dists_dense(ctx, sub), *capi.query_knn(ctx, ref, qry, 4)]
        ctx.set_tile_config(PLAIN_SHAPE)
        plain = [capi.dists_dense(ctx, sub), *capi.query_knn(ctx, ref, qry, 4)]
        for a, b in zip(coded, plain):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(served[0], plain[1])
        np.testing.assert_array_equal(served[1], plain[2])


def test_coded_batch(gpu_ctx):
    """Coded and plain jobs in one batch, replayed: each equals its own call."""
    import torch
    jobs, keep = [], []
    for i, (n, nq, K, s64) in enumerate([(1900, None, 4, 3), (300, None, 8, 16),
                                         (1500, 200, 3, 5), (100, None, 34, 2)]):
        w, kmers = random_sketches(n + (nq or 0), K, s64, seed=70 + i)
        ref = capi.Database(gpu_ctx, w[:n], kmers, s64)
        qry = None if nq is None else capi.Database(gpu_ctx, w[n:], kmers, s64)
        out = torch.zeros((capi.dists_rows(ref, qry), K), dtype=torch.int32, device="cuda")
        jobs.append((ref, qry, None, capi.OUT_COUNTS, out.data_ptr()))
        keep.append((ref, qry, out))
    torch.cuda.synchronize()
    b = capi.Batch(gpu_ctx, jobs)
    for _ in range(2):
        for *_, out in keep:
            out.zero_()
        torch.cuda.synchronize()
        b.run()
        for ref, qry, out in keep:
            np.testing.assert_array_equal(
                out.cpu().numpy().view(np.uint32),
                capi.dists_dense(gpu_ctx, ref, qry, out_mode=capi.OUT_COUNTS))
    b.close()
