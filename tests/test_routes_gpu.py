"""Which kernels the entry points launch, from a profiler's record: the results
alone cannot tell, since every special route falls back on a general one with
the same results."""
import numpy as np
import pytest

from conftest import random_sketches
from launched import names_during
from sketchlib_b200 import capi
from test_low_coverage_gpu import _offsets, _read_set

pytestmark = pytest.mark.gpu


def _kernels(call):
    call()
    return " ".join(names_during(call))


def _forms(ctx, ref, qry, few, w, kmers, s64):
    import torch
    out = torch.empty((ref.n * (ref.n - 1) // 2, 2), dtype=torch.float32, device="cuda")

    def blocked():
        ctx.set_memory_limit(2_000_000)
        capi.dists_dense(ctx, ref)
        ctx.set_memory_limit(0)

    def batch():
        b = capi.Batch(ctx, [(ref, None, None, capi.OUT_CORE_ACC, out.data_ptr())])
        b.run()
        b.close()

    def serve(n):
        server = capi.Server(ctx, ref, slots=1, slice_queries=256, kNN=2)
        server.wait(server.submit(w[-n:]))
        server.close()

    return {
        "self": ("code_columns_kernel", lambda: capi.dists_dense(ctx, ref)),
        "query": ("code_columns_kernel", lambda: capi.dists_dense(ctx, ref, qry)),
        "knn": ("code_columns_kernel", lambda: capi.dists_knn(ctx, ref, 3)),
        "threshold": ("code_columns_kernel", lambda: capi.dists_threshold(ctx, ref, 0, 0.01)),
        "host": ("code_columns_kernel", lambda: capi.query_db(ctx, w[:ref.n], kmers, s64)),
        "blocked": ("code_columns_kernel", blocked),
        "batch": ("code_columns_kernel", batch),
        "slice of 200": ("code_columns_kernel", lambda: serve(200)),
        "few": ("few_queries_kernel", lambda: capi.dists_dense(ctx, ref, few)),
        "few kNN": ("few_queries_kernel", lambda: capi.query_knn(ctx, ref, few, 20)),
        "slice of 9": ("few_queries_kernel", lambda: serve(9)),
        "long list": ("knn_select_kernel", lambda: capi.dists_knn(ctx, ref, 17)),
        "short list": ("knn_lists_kernel", lambda: capi.dists_knn(ctx, ref, 16)),
    }


def test_entry_points_take_the_routes_meant_for_them():
    n, K, s64 = 1800, 3, 4
    w, kmers = random_sketches(n + 200, K, s64, seed=23)
    with capi.Context(0) as ctx:
        ref = capi.Database(ctx, w[:n], kmers, s64)
        qry = capi.Database(ctx, w[n:], kmers, s64)
        few = capi.Database(ctx, w[-9:], kmers, s64)
        for name, (kernel, call) in _forms(ctx, ref, qry, few, w, kmers, s64).items():
            assert kernel in _kernels(call), name


# coverage and min_count whose bins are filled at once, rolled again, given up
@pytest.mark.parametrize("coverage,min_count,again,full", [(12, 1, False, False), (3, 5, True, False),
                                                           (1, 5, False, True)])
def test_read_sets_take_the_rolls_meant_for_them(gpu_ctx, coverage, min_count, again, full):
    rng = np.random.default_rng(24)
    sets = [_read_set(rng, 600_000 // coverage, coverage)]
    off, ss = _offsets(sets)
    names = _kernels(lambda: capi.sketch(gpu_ctx, sets[0], off, ss, [15, 17], 16,
                                         min_count=min_count))
    assert "low_roll_kernel<true, false, false>" in names
    assert ("low_roll_kernel<true, false, true>" in names) == again
    assert ("part_kernel" in names) == full
