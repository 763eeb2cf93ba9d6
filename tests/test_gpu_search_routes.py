"""What bsj_plan_select_routes reports of the resident search: that it ran and with how many thread
blocks per beam in either form, which of its routes a level took, and levels that one block
had to select (several thousand tied scores, or survivors close to the buffers' size); each
search equals the oracle."""
import numpy as np
import pytest

from beamsearch_jssp_gpu_gb300 import BeamSpec, synthetic_instance
from oracle import oracle as O

pytestmark = pytest.mark.gpu

BLOCKS = {"blocks_1", "blocks_2", "blocks_4", "blocks_8", "blocks_12", "blocks_16"}
OWN = BLOCKS | {"resident", "recount", "tie_bins", "window_sort", "one_block"}


def _routes(ctx, beams, insts, wide=True, flags=(), chunk=0):
    plan = ctx.plan(insts, beams)
    try:
        plan.set_select_cluster(wide)
        plan.set_select_route(*flags)
        if chunk:
            plan.chunk = chunk
        plan.run()
        got, routes = plan.results(), plan.select_routes()
    finally:
        plan.close()
    for b, g in zip(beams, got):
        want = O.solve(*insts[b.instance], b.mode, b.beam_width, b.seed)
        for k in ("makespan", "found", "expanded", "levels"):
            assert g[k] == want[k], (k, b)
        assert np.array_equal(g["seq"], want["seq"]), b
    return routes


@pytest.mark.parametrize("n,m,K,wide,narrow", [
    (10, 5, 64, "blocks_1", {"blocks_1"}), (15, 6, 256, "blocks_4", {"blocks_4"}),
    (20, 6, 4096, "blocks_16", {"blocks_4", "blocks_8"}), (100, 2, 2048, "blocks_16", {"blocks_4", "blocks_8"})])
def test_blocks_per_beam(ctx, n, m, K, wide, narrow):
    inst = synthetic_instance(n, m, 2)
    beam = BeamSpec("v2", K, 500000, 3, 0, -1)
    got = _routes(ctx, [beam], [inst])
    assert "resident" in got and got & BLOCKS == {wide}, got
    got = _routes(ctx, [beam], [inst], wide=False)
    assert "resident" in got and len(got & BLOCKS) == 1 and got & BLOCKS <= narrow, got


def test_level_kernels_report_none_of_it(ctx):
    inst, one = synthetic_instance(12, 4, 2), synthetic_instance(12, 1, 2)
    for mode in ("v1", "v2", "clean"):
        beam = BeamSpec(mode, 200, 500000, 3, 0, -1)
        assert not _routes(ctx, [beam], [inst], flags=("no_direct",)) & OWN
        assert not _routes(ctx, [beam], [inst], chunk=16) & OWN
        assert not _routes(ctx, [beam], [one]) & OWN
    assert not _routes(ctx, [BeamSpec("pms", 30, 500000, 3, 0, -1)], [inst]) & OWN


@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("mode,n,m,K,dmax", [("v1", 16, 3, 16384, 2), ("v2", 16, 3, 16384, 99)])
def test_one_block_levels(ctx, mode, n, m, K, dmax, wide):
    mc, du = synthetic_instance(n, m, 3)
    if dmax < 99:
        du = (du % dmax + 1).astype(np.int32)
    got = _routes(ctx, [BeamSpec(mode, K, 500000, 5, 0, -1)], [(mc, du)], wide)
    assert {"resident", "recount", "one_block"} <= got, got


def test_plain_levels_take_no_detour(ctx):
    got = _routes(ctx, [BeamSpec("v2", 256, 500000, 3, 0, -1)], [synthetic_instance(15, 15, 1)])
    assert not got & {"one_block", "bucket", "radix", "large"}, got


@pytest.mark.parametrize("n,m,K,resident", [
    (32, 4, 5000, True), (40, 8, 5120, False), (40, 3, 5120, True), (50, 5, 4096, False), (50, 10, 4096, True),
    (64, 6, 8191, True), (64, 8, 7000, False), (64, 6, 8192, True), (80, 2, 2560, False), (80, 5, 2560, True),
    (128, 2, 2048, True), (128, 3, 2049, False), (100, 9, 4096, False), (100, 8, 6144, True)])
def test_v1_beams_by_size(ctx, n, m, K, resident):
    # v1 writes every scored child: beams of many children go to the level kernels (v2 and clean never)
    inst = synthetic_instance(n, m, 2)
    got = _routes(ctx, [BeamSpec("v1", K, 500000, 3, 0, -1)], [inst])
    assert ("resident" in got) == resident, got
