"""Calls of different sizes on several threads at once, each thread with its own
context: every call succeeds and gives what it gives alone."""
import threading

import numpy as np
import pytest

from conftest import random_sketches
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu


def _at_once(jobs, repeats):
    """Runs every job `repeats` times on a thread of its own; their errors."""
    errors, start = [], threading.Barrier(len(jobs))

    def work(job):
        with capi.Context(0) as ctx:
            call, want = job(ctx)
            start.wait()
            try:
                for _ in range(repeats):
                    for a, b in zip(call(), want):
                        np.testing.assert_array_equal(a, b)
            except Exception as e:      # reported by the test below
                errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_knn_lists_of_different_lengths_on_threads():
    """Lists of 25 to 50 entries need different amounts of shared memory."""
    words, kmers = random_sketches(2100, 1, 1, seed=5)

    def job(knn):
        def make(ctx):
            db = capi.Database(ctx, words, kmers, 1)
            call = lambda: capi.dists_knn(ctx, db, knn)
            return call, call()
        return make

    assert _at_once([job(k) for k in (25, 33, 41, 50)], 400) == []


def test_sketches_of_different_widths_on_threads():
    rng = np.random.default_rng(6)
    bases = rng.choice(np.frombuffer(b"ACGT", np.uint8), 20_000)

    def job(s64):
        def make(ctx):
            call = lambda: capi.sketch(ctx, bases, [0, 20_000], [0, 1], [15], s64)[:1]
            return call, call()
        return make

    assert _at_once([job(s) for s in (64, 100, 156, 300)], 400) == []


def test_coded_calls_on_threads():
    """Jobs of different sizes, each coded in its own context's buffer."""
    words, kmers = random_sketches(2300, 3, 8, seed=7)

    def job(n, nq):
        def make(ctx):
            db = capi.Database(ctx, words[:n], kmers, 8)
            qry = capi.Database(ctx, words[n:n + nq], kmers, 8) if nq else None
            call = lambda: [capi.dists_dense(ctx, db, qry)]
            return call, call()
        return make

    assert _at_once([job(1700, 0), job(2300, 0), job(1500, 300), job(1100, 140)], 25) == []
