"""The exact modes' bounded heap (ICH, PMS) against the oracle at the sizes where its shape
changes: one node, a last position that is a left or a right child, full and barely started
last levels, up to a path of 14 nodes.  Durations in {1, 2} make most keys tie, so the
order libstdc++ leaves among equals decides the next level."""
import numpy as np
import pytest

from beamsearch_jssp_gpu_gb300 import synthetic_instance
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["ich", "pms"])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 31, 33, 64, 127, 128, 129, 500, 1023, 1025])
def test_heap_sizes_match_oracle(ctx, mode, K):
    n, m = (7, 4) if K > 200 else (9, 5)
    mc, du = synthetic_instance(n, m, K)
    for d in (du, (du % 2 + 1).astype(np.int32)):
        want = O.solve(mc, d, mode, K, 17)
        got = ctx.solve(mc, d, mode, K, 17)
        for k in ("makespan", "found", "expanded", "levels"):
            assert got[k] == want[k], (k, mode, K)
        assert np.array_equal(got["seq"], want["seq"]), (mode, K)


@pytest.mark.parametrize("mode,n,m,K", [("ich", 5, 4, 8191), ("pms", 12, 3, 8192), ("pms", 100, 2, 300),
                                        ("ich", 128, 1, 20)])
def test_heap_wide_and_long_lists(ctx, mode, n, m, K):
    mc, du = synthetic_instance(n, m, 3)
    want = O.solve(mc, du, mode, K, 2**32 - 5)
    got = ctx.solve(mc, du, mode, K, 2**32 - 5)
    assert got["makespan"] == want["makespan"] and got["expanded"] == want["expanded"]
    assert np.array_equal(got["seq"], want["seq"])
