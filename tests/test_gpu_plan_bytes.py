"""Device memory of a plan of the resident search: a second key region only where a block's candidate
list can outgrow its shared memory."""
import pytest

from beamsearch_jssp_gpu_gb300 import BeamSpec, synthetic_instance

pytestmark = pytest.mark.gpu


def _regions(n, m, K):
    """Bytes of one v2 beam: two snapshot buffers, one key region, history, branch positions, masks,
    survivors and the ranks' chunk counts."""
    N, snap = n * m, ((4 * m + 6 * n + 3) // 4 * 4 + n + 15) // 16 * 16 + 16
    return 2 * K * snap + 8 * n * ((K + 31) // 32 * 32) + 4 * N * K + 2 * K * n + 4 * K * ((n + 31) // 32) + 4 * K + 2 * K


SMALL = 32 << 10   # descriptors, states, tables, operations, alignment


@pytest.mark.parametrize("n,m,K,spills", [(100, 2, 64, False), (50, 5, 512, False), (128, 3, 4096, True)])
def test_key_regions(ctx, n, m, K, spills):
    inst = synthetic_instance(n, m, 1)
    got = ctx.estimate([inst], [BeamSpec("v2", K, 500000, 1, 0, -1)]) - _regions(n, m, K)
    assert (got > 8 * n * K - SMALL) == spills and got <= SMALL + (8 * n * K if spills else 0), got
