"""The resident search (one cluster of thread blocks per beam, all levels in one kernel)
against the oracle, bit for bit.

Sizes at the edges of what it splits: beam widths around the shares at which the lanes per
survivor and the blocks per beam change, lists of 32, 40, 64 and 128 jobs (the words a lane
compares), two machines (half of a parent's children on the pivot machine, lists beyond the
shared-memory capacity), several rounds per block, and a single survivor.  Durations of 1
tie nearly every score, so bins exceed the blocks' buffers and the one-block selection
takes the level; bounds prune children, so v1 / v2 fillers and empty clean levels occur.
"""
import numpy as np
import pytest

from beamsearch_jssp_gpu_gb300 import BeamSpec, synthetic_instance
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MODES = ["v1", "v2", "clean"]
SHAPES = [  # (n, m, K)
    (1, 2, 3), (2, 2, 1), (9, 3, 64), (9, 3, 65), (12, 4, 128), (12, 4, 129), (15, 5, 256), (15, 5, 257),
    (32, 3, 513), (33, 3, 512), (40, 2, 700), (41, 2, 700), (64, 2, 300), (65, 2, 300), (128, 2, 100),
    (6, 64, 40), (11, 4, 2049), (7, 5, 4096), (8, 4, 16384),
]


def _check(ctx, mc, du, mode, K, seed, bk=500000):
    want = O.solve(mc, du, mode, K, seed, best_known=bk)
    plan = ctx.plan([(mc, du)], [BeamSpec(mode, K, bk, seed, 0, -1)])
    try:
        for wide in (True, False):
            plan.set_select_cluster(wide)
            plan.run()
            got = plan.results()[0]
            what = (mode, mc.shape, K, seed, bk, wide)
            for k in ("makespan", "found", "expanded", "slots", "levels"):
                assert got[k] == want[k], (k, what)
            assert np.array_equal(got["seq"], want["seq"]), what
        assert plan.launches == 3, what   # the search, the lineage runs and the finalisation
    finally:
        plan.close()


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,m,K", SHAPES)
def test_search_matches_oracle(ctx, mode, n, m, K):
    mc, du = synthetic_instance(n, m, n + m)
    _check(ctx, mc, du, mode, K, 2**32 - K)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("n,m,K", [(10, 4, 3000), (40, 2, 2000), (70, 2, 900), (8, 4, 16384)])
def test_search_tied_scores(ctx, mode, n, m, K):
    mc, _ = synthetic_instance(n, m, 3)
    _check(ctx, mc, np.ones((n, m), np.int32), mode, K, 5)


@pytest.mark.parametrize("mode", MODES)
def test_search_bounds(ctx, mode):
    mc, du = synthetic_instance(10, 5, 21)
    for K in (64, 600):
        base = O.solve(mc, du, mode, K, 3)["makespan"]
        for bk in (base + 30, base + 1, base, base - 20, 1):
            _check(ctx, mc, du, mode, K, 3, bk)


def test_search_many_beams_of_mixed_classes(ctx):
    """Beams of every mode, uneven sizes and widths in one plan: the searches run as one
    launch per class beside the level kernels of the exact modes and of m = 1."""
    insts = [synthetic_instance(12, 4, 1), synthetic_instance(66, 2, 2), synthetic_instance(9, 1, 3),
             synthetic_instance(20, 6, 4)]
    beams = [BeamSpec(mode, K, 500000, 100 + i, i % 4, -1)
             for i, (mode, K) in enumerate([("v2", 64), ("clean", 100), ("v1", 50), ("ich", 16), ("v1", 700),
                                            ("pms", 8), ("clean", 257), ("v2", 1200), ("v1", 300), ("v2", 33)])]
    plan = ctx.plan(insts, beams)
    try:
        for _ in range(2):
            plan.run()
            for b, r in zip(beams, plan.results()):
                mc, du = insts[b.instance]
                want = O.solve(mc, du, b.mode, b.beam_width, b.seed)
                assert r["makespan"] == want["makespan"], b
                assert np.array_equal(r["seq"], want["seq"]), b
                assert r["expanded"] == want["expanded"], b
    finally:
        plan.close()
