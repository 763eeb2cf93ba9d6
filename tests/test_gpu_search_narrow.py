"""The narrow form of the resident search: beams that stay at four blocks and beams whose
long lists take eight, against the oracle, alone and mixed in one plan."""
import numpy as np
import pytest

from beamsearch_jssp_gpu_gb300 import BeamSpec, synthetic_instance
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beams", [[("v2", 100, 2, 4096)], [("clean", 128, 2, 2500)], [("v1", 20, 3, 512)],
                                   [("v2", 100, 2, 4096), ("v2", 20, 3, 512), ("clean", 64, 2, 3000), ("v1", 65, 2, 2048)]])
def test_narrow_form_matches_oracle(ctx, beams):
    inst = [synthetic_instance(n, m, i) for i, (_, n, m, _) in enumerate(beams)]
    plan = ctx.plan(inst, [BeamSpec(mode, K, 500000, 3 + i, i) for i, (mode, _, _, K) in enumerate(beams)])
    try:
        plan.set_select_cluster(False)
        plan.run()
        got = plan.results()
        assert "cluster" not in plan.select_routes()
    finally:
        plan.close()
    for i, (mode, _, _, K) in enumerate(beams):
        want = O.solve(*inst[i], mode, K, 3 + i)
        for f in ("makespan", "found", "expanded", "slots", "levels"):
            assert got[i][f] == want[f], (f, beams[i])
        assert np.array_equal(got[i]["seq"], want["seq"]), beams[i]


@pytest.mark.parametrize("first", [True, False])
def test_narrow_form_is_no_wider(ctx, first):
    # so many beams that the rule gives each one block: the narrow form, which trades latency for
    # SM time, gives them no more, and the form asked for first does not stand in for the other
    inst = [synthetic_instance(100, 2, 1)]
    want = O.solve(*inst[0], "v2", 4096, 3)
    plan = ctx.plan(inst, [BeamSpec("v2", 4096, 500000, i, 0, -1) for i in range(140)])
    try:
        for wide in (first, not first):
            plan.set_select_cluster(wide)
            plan.run()
            got = plan.results()
            assert {r for r in plan.select_routes() if r.startswith("blocks")} == {"blocks_1"}, wide
            assert got[3]["makespan"] == want["makespan"] and np.array_equal(got[3]["seq"], want["seq"]), wide
    finally:
        plan.close()
