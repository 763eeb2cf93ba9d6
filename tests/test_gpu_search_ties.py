"""The resident search on durations whose scores tie, or lie in another unit than 1 .. 99, against
the oracle; and tied levels stay in it: the one-block routes, which a level takes whose bins do
not fit the blocks' buffers, show as "bucket", "radix" or "large" for levels of this size."""
import numpy as np
import pytest

from beamsearch_jssp_gpu_gb300 import BeamSpec, synthetic_instance
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DURATIONS = {
    "one": lambda du: np.ones_like(du),
    "one or two": lambda du: du % 2 + 1,
    "small": lambda du: du % 5 + 1,
    "quarter hours": lambda du: 15 * (du % 6 + 1),
    "x1000": lambda du: du * 1000,
    "outlier": lambda du: np.where(np.arange(du.size).reshape(du.shape) == 3, 300000, du),
    "some zero": lambda du: np.where(du % 3 == 0, 0, du % 4),
    "zero": lambda du: np.zeros_like(du),
}


def _solve(ctx, mc, du, mode, K, bk):
    want = O.solve(mc, du, mode, K, 77, best_known=bk)
    plan = ctx.plan([(mc, du)], [BeamSpec(mode, K, bk, 77, 0, -1)])
    try:
        plan.run()
        got, routes = plan.results()[0], plan.select_routes()
    finally:
        plan.close()
    for k in ("makespan", "found", "expanded", "slots", "levels"):
        assert got[k] == want[k], (k, mode, mc.shape, K, bk)
    assert np.array_equal(got["seq"], want["seq"]), (mode, mc.shape, K, bk)
    return got, routes


@pytest.mark.parametrize("mode", ["v1", "v2", "clean"])
@pytest.mark.parametrize("name", list(DURATIONS))
def test_durations_match_oracle(ctx, mode, name):
    for n, m, K in ((10, 5, 64), (15, 7, 256), (20, 5, 700), (30, 4, 2500)):
        mc, du = synthetic_instance(n, m, n)
        du = DURATIONS[name](du).astype(np.int32)
        got, _ = _solve(ctx, mc, du, mode, K, 2**31 - 2)
        for bk in (got["makespan"] + 1, got["makespan"], max(1, got["makespan"] * 3 // 4)):
            _solve(ctx, mc, du, mode, K, bk)


@pytest.mark.parametrize("name", ["one", "one or two", "small", "quarter hours"])
@pytest.mark.parametrize("n,m,K", [(60, 6, 1000), (50, 5, 4096)])
def test_tied_levels_stay_resident(ctx, name, n, m, K):
    mc, du = synthetic_instance(n, m, 4)
    _, routes = _solve(ctx, mc, DURATIONS[name](du).astype(np.int32), "v2", K, 500000)
    assert not routes & {"bucket", "radix"}, routes


@pytest.mark.parametrize("mode,n,m", [("v2", 20, 3), ("clean", 30, 3), ("v1", 24, 4)])
def test_wide_tied_levels_leave_one_block(ctx, mode, n, m):
    # a wide beam whose early levels fit no bins goes on with tie bins: it does not stay with one block
    # (a v1 beam's stale states score by their own number of operations, tie bins by the level's)
    mc, du = synthetic_instance(n, m, n + m)
    _, routes = _solve(ctx, mc, DURATIONS["small"](du).astype(np.int32), mode, 16384, 500000)
    assert "tie_bins" in routes and (mode == "v1" or "one_block" not in routes), routes
