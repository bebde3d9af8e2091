"""A re-test queue that overflows at level 1: the run gives the oracle's skeleton."""
import numpy as np
import pytest

import heterogpc as hg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

N, ALPHA = 400, 0.05


@pytest.mark.parametrize("max_level", [1, 2])
def test_captured_queue_only_kernel_is_not_replayed_after_an_overflow(max_level):
    rng = np.random.default_rng(3)
    X = (rng.uniform(0.2, 0.9, (40, 1)) * rng.standard_normal((1, N)) + rng.standard_normal((40, N))).astype(np.float32)
    want = orc.run(orc.correlation(X.astype(np.float64)), N, ALPHA, max_level)
    sk = hg.SkeletonCalculator(40, N, alpha=ALPHA, max_level=max_level, precision=hg.PREC_MIXED_TC, retest_margin=0.3)
    sk.add_observations(X)
    sk.run()
    assert sk.level_stats[1]["retests"] > 16
    assert hg.lib().hpc_debug_set_retest_queue(sk.handle, 16) == 0
    for _ in range(3):  # captured and overflowing, rerun, replayed
        sk.reset()
        sk.run()
        assert np.array_equal(sk.adjacency(), want.adj)
    sk.close()
