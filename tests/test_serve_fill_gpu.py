"""Rows that a slice computes anyway are filled with queries of larger requests,
and no others: a small request does not wait for more than that."""
import numpy as np
import pytest

from conftest import random_sketches
from launched import names_during
from sketchlib_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small,group", [(10, 12), (3, 4), (20, 12)])
def test_a_small_slice_takes_its_group_of_queries(small, group):
    n, nq, K, s64 = 4000, 1500, 4, 64
    w, kmers = random_sketches(n + 64, K, s64, seed=19)
    q = np.concatenate([w[n:]] * 24)[:nq]
    with capi.Context(0) as ctx:
        ref = capi.Database(ctx, w[:n], kmers, s64)
        server = capi.Server(ctx, ref, slots=1, slice_queries=128, kNN=2)
        first = server.submit(q)
        server.wait(first)                       # the kernels are loaded
        tickets = []

        def both():
            tickets[:] = [server.submit(q), server.submit(q[:small])]
            for t in tickets:
                server.wait(t)

        names = {x for x in names_during(both) if "few_queries_kernel" in x}
        large, ticket = tickets
        got, whole = server.result(ticket)[:2], server.result(large)[:2]
        server.close()
        ref.close()
    assert any(f"few_queries_kernel<{group}>" in x for x in names)
    for a, b in zip(got, whole):
        np.testing.assert_array_equal(a, b[:small])
