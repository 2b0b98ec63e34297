"""Read sets counted from the low end of their bins (at least 256 windows per
bin): sketches, inverse minhashes and densify flags against the oracle's exact
counter, where bins stay empty after the first roll (few distinct k-mers, a
min_count nothing reaches), where one k-mer floods the lists, and mixed with
samples too small for it."""
import numpy as np
import pytest

import oracle
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu

LETTERS = np.frombuffer(b"ACGT", np.uint8)


def _reads(rng, genome, coverage, errors=0.01, length=100):
    g = LETTERS[rng.integers(0, 4, genome)]
    n = coverage * genome // length
    starts = rng.integers(0, max(1, genome - length), n)
    r = g[(starts[:, None] + np.arange(length)) % genome]
    wrong = rng.random(r.shape) < errors
    r[wrong] = LETTERS[rng.integers(0, 4, int(wrong.sum()))]
    return [x.tobytes() for x in r]


def _samples(kind, rng):
    if kind == "usual":
        return [_reads(rng, 20_000, 12), _reads(rng, 30_000, 6)]
    if kind == "few distinct":            # most bins hold no k-mer near their start
        return [_reads(rng, 300, 400), _reads(rng, 40, 2000, errors=0.0)]
    if kind == "flood":                   # two k-mers make up most of the windows
        return [_reads(rng, 10_000, 10) + [b"A" * 60_000, b"AC" * 40_000]]
    if kind == "nothing":
        return [_reads(rng, 60_000, 1, errors=0.0)]
    return [_reads(rng, 20_000, 10), _reads(rng, 500, 4), [b"ACG"], [b"ACGTN" * 3],
            _reads(rng, 15_000, 30)]


@pytest.mark.parametrize("kind", ["usual", "few distinct", "flood", "nothing", "mixed"])
@pytest.mark.parametrize("s64,min_count,rc,phased", [
    (1, 3, True, False), (2, 2, False, False), (5, 4, True, True), (1, 1, True, False),
])
def test_matches_oracle(gpu_ctx, kind, s64, min_count, rc, phased):
    rng = np.random.default_rng(len(kind) + s64)
    bases, off, ss = capi.pack_sequences(_samples(kind, rng))
    kmers = [15, 21, 31] if not phased else [9, 12]
    got = capi.sketch(gpu_ctx, bases, off, ss, kmers, s64, rc, min_count, codon_phased=phased)
    want = oracle.sketch(bases, off, ss, kmers, s64, rc, min_count, codon_phased=phased)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)
