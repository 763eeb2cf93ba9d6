"""32-bit order keys of the exact modes' heap: (makespan, noise index) pairs order as the
fp64 scores do up to 1 000 operations (CPU), and the searches equal the oracle on both sides
of each line: level 1 000 and a total duration of 4 294 966 (GPU; one context, so a plan is
reused with the other kind of instance)."""
import numpy as np
import pytest

from beamsearch_jssp_gpu_gb300 import synthetic_instance
from oracle import oracle as O

LIMIT = 4294966


def _scores(cc, k, ns):
    return cc / np.float64(ns) + k / np.float64(1000000.0)


@pytest.mark.parametrize("ns", [1, 2, 3, 7, 64, 300, 640, 997, 999, 1000])
@pytest.mark.parametrize("lo", [0, 1, 4095, 499998, 1 << 21, 4194303, LIMIT - 3])
def test_pms_pairs_order_as_scores(ns, lo):
    cc = np.repeat(np.arange(lo, lo + 4, dtype=np.int64), 1000)
    k = np.tile(np.arange(1000, dtype=np.int64), 4)
    key = cc * 1000 + k
    assert key[cc <= LIMIT].max() < 2**32
    assert np.all(np.diff(_scores(cc.astype(np.float64), k, ns)) > 0)   # strictly, in key order


def test_pms_pairs_do_not_order_later_scores():
    assert _scores(1000.0, 999, 1200) > _scores(1001.0, 0, 1200)


def _with_total(n, m, seed, total):
    mc, du = synthetic_instance(n, m, seed)
    du = du.astype(np.int64) * (total // int(du.sum()))
    du.flat[-1] += total - int(du.sum())
    assert int(du.sum()) == total and du.max() < 2**24
    return mc, du.astype(np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["ich", "pms"])
def test_total_duration_limit(ctx, mode):
    for total in (LIMIT, LIMIT + 1, LIMIT - 20000):
        mc, du = _with_total(30, 20, 4, total)   # makespans below the 500 000 of "none found"
        want = O.solve(mc, du, mode, 40, 11)
        got = ctx.solve(mc, du, mode, 40, 11)
        assert want["found"]
        for f in ("makespan", "found", "expanded", "levels"):
            assert got[f] == want[f], (f, mode, total)
        assert np.array_equal(got["seq"], want["seq"]), (mode, total)


@pytest.mark.gpu
def test_levels_past_one_thousand(ctx):
    mc, du = synthetic_instance(51, 20, 2)   # 1 020 levels
    want = O.solve(mc, du, "pms", 37, 5)
    got = ctx.solve(mc, du, "pms", 37, 5)
    for f in ("makespan", "found", "expanded", "levels"):
        assert got[f] == want[f], f
    assert np.array_equal(got["seq"], want["seq"])
