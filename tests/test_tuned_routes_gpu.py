"""A tuned tile shape chooses among tiles of whole planes only: the kernels a
call launches with an entry in the tuning table, from a profiler's record."""
import numpy as np
import pytest

from conftest import random_sketches
from launched import names_during
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu

K, S64 = 3, 4


def _kernels(call):
    call()
    return " ".join(names_during(call))


@pytest.mark.parametrize("how", ["autotuned", "loaded", "neither"])
def test_tuned_shapes_leave_few_queries_and_codes_alone(tmp_path, how):
    w, kmers = random_sketches(1803, K, S64, seed=17)
    with capi.Context(0) as ctx:
        small = capi.Database(ctx, w[:300], kmers, S64)
        all_ = capi.Database(ctx, w[:1800], kmers, S64)
        qry = capi.Database(ctx, w[1800:], kmers, S64)
        want = [capi.dists_dense(ctx, d, q) for d, q in ((small, None), (all_, None), (all_, qry))]
        if how == "autotuned":
            assert 1 <= capi.autotune(ctx, small, repeats=1) <= len(capi.tile_configs())
        elif how == "loaded":
            (tmp_path / "t").write_text(f"{K} {S64} 4\n")
            ctx.load_tuning(tmp_path / "t")
        assert "few_queries_kernel" in _kernels(lambda: capi.dists_dense(ctx, all_, qry))
        assert "code_columns_kernel" in _kernels(lambda: capi.dists_dense(ctx, all_))
        for kernel in ("few_queries_kernel", "code_columns_kernel"):
            assert kernel not in _kernels(lambda: capi.dists_dense(ctx, small))
        if how == "loaded":                      # shape 4: 8 x 8 pairs per thread
            assert "dist_items_kernel<128, 128, 8, 8" in _kernels(
                lambda: capi.dists_dense(ctx, small))
        for (d, q), x in zip(((small, None), (all_, None), (all_, qry)), want):
            np.testing.assert_array_equal(capi.dists_dense(ctx, d, q), x)


def test_a_batch_of_mostly_coded_work_is_coded_whatever_is_tuned(tmp_path):
    import torch
    w, kmers = random_sketches(1800, K, S64, seed=18)
    (tmp_path / "t").write_text(f"{K} {S64} 4\n")
    with capi.Context(0) as ctx:
        ctx.load_tuning(tmp_path / "t")
        dbs = [capi.Database(ctx, w[:n], kmers, S64) for n in (1800, 200)]
        outs = [torch.empty((d.n * (d.n - 1) // 2, 2), dtype=torch.float32, device="cuda") for d in dbs]
        b = capi.Batch(ctx, [(d, None, None, capi.OUT_CORE_ACC, o.data_ptr()) for d, o in zip(dbs, outs)])
        assert b.info()["tile_config"] == 1
        b.run()
        for d, o in zip(dbs, outs):
            np.testing.assert_array_equal(o.cpu().numpy(), capi.dists_dense(ctx, d))
        b.close()
