"""Read sets whose coverage is near min_count (bins left empty by the count from
the low end) and read sets uploaded in several chunks."""
import time

import numpy as np
import pytest

import oracle
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu

LETTERS = np.frombuffer(b"ACGT", np.uint8)


def _read_set(rng, genome, coverage, errors=0.01, length=150):
    g = rng.integers(0, 4, genome)
    n = coverage * genome // length
    r = g[rng.integers(0, genome - length, n)[:, None] + np.arange(length)]
    wrong = rng.random(r.shape) < errors
    r[wrong] = (r[wrong] + 1) % 4
    return LETTERS[r].reshape(-1)


def _offsets(sets, length=150):
    per = [s.size // length for s in sets]
    return (np.arange(sum(per) + 1, dtype=np.int64) * length,
            np.concatenate([[0], np.cumsum(per)]).astype(np.int64))


def _ms(call):
    call()
    call()
    best = []
    for _ in range(9):
        t = time.perf_counter()
        call()
        best.append(time.perf_counter() - t)
    return 1e3 * min(best)


@pytest.mark.parametrize("coverage,min_count", [(2, 5), (3, 5), (2, 3), (3, 3)])
def test_low_coverage_costs_no_more_than_the_full_count(gpu_ctx, coverage, min_count):
    """8 M bases in all.  A width with fewer than 256 windows per bin is counted
    in full; the usual width, counted from the low end, may cost a third more."""
    rng = np.random.default_rng(coverage)
    genome = 4_000_000 // coverage
    sets = [_read_set(rng, genome, coverage) for _ in range(2)]
    off, ss = _offsets(sets)
    bases, kmers = np.concatenate(sets), list(range(15, 31, 2))
    full = int(4_000_000 / 64 / 250)
    assert 4_000_000 >= 256 * 64 * 156 and 4_000_000 < 256 * 64 * full
    low = _ms(lambda: capi.sketch(gpu_ctx, bases, off, ss, kmers, 156, min_count=min_count))
    all_ = _ms(lambda: capi.sketch(gpu_ctx, bases, off, ss, kmers, full, min_count=min_count))
    assert low < 1.35 * all_


@pytest.mark.parametrize("coverage,min_count", [(2, 4), (4, 4), (8, 3)])
def test_rows_rolled_twice_and_rows_counted_in_full_match_the_oracle(gpu_ctx, coverage, min_count):
    """Samples with no, few and most bins left empty, in one call: k of 11 to 61
    and read sets of 300 and more windows per bin."""
    rng = np.random.default_rng(30 + coverage)
    sets = [_read_set(rng, 90_000 // c, c) for c in (coverage, 1, 3 * coverage, coverage)]
    off, ss = _offsets(sets)
    kmers = [11, 21, 41, 61]
    args = (np.concatenate(sets), off, ss, kmers, 4, True, min_count)
    for got, want in zip(capi.sketch(gpu_ctx, *args), oracle.sketch(*args)):
        np.testing.assert_array_equal(got, want)


def test_uploads_in_several_chunks_match_the_oracle(gpu_ctx):
    """Three samples of 9 MB go up one after another while those before them
    are counted; a fourth, small one shares the last chunk."""
    rng = np.random.default_rng(41)
    sets = [_read_set(rng, 900_000, 10) for _ in range(3)] + [_read_set(rng, 3_000, 10)]
    off, ss = _offsets(sets)
    args = (np.concatenate(sets), off, ss, [17, 25], 16, True, 3)
    for got, want in zip(capi.sketch(gpu_ctx, *args), oracle.sketch(*args)):
        np.testing.assert_array_equal(got, want)
