"""A re-test queue that overflows at level 1: the run gives the oracle's skeleton, and what it changes
ends with the data that caused it."""
import numpy as np
import pytest

import heterogpc as hg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

P, N, ALPHA = 321, 400, 0.05


def _correlation(seed, spread):
    rng = np.random.default_rng(seed)
    X = rng.uniform(*spread, (P, 1)) * rng.standard_normal((1, N)) + rng.standard_normal((P, N))
    return orc.correlation(X)


def _launches(sk):
    before = sk.timings()["launches"]
    sk.reset()
    sk.run()
    return sk.timings()["launches"] - before


def test_deferral_beside_a_matrix_returns_with_new_data():
    """Mixed precision beside an FP64 matrix: data with many undecided tests run inline, later data
    queue them again (a launch more)."""
    many = _correlation(1, (0.2, 0.9))
    few = 0.6 * np.ones((P, P)) + 0.4 * np.eye(P)  # every test of level 1 far above the critical value
    L = hg.lib()
    sk = hg.SkeletonCalculator(P, N, alpha=ALPHA, max_level=1, retest_margin=0.5)
    sk.add_correlation_matrix(few)
    sk.run()
    assert L.hpc_debug_set_retest_queue(sk.handle, 64) == 0
    deferred = [_launches(sk) for _ in range(2)][-1]
    want = orc.run(many, N, ALPHA, 1)
    sk.add_correlation_matrix(many)
    for _ in range(3):
        inline = _launches(sk)
        assert np.array_equal(sk.adjacency(), want.adj)
        assert sk.level_stats[1]["retests"] > 64
    assert inline == deferred - 1
    assert L.hpc_debug_set_order_active(sk.handle) == 1
    sk.add_correlation_matrix(few)
    again = [_launches(sk) for _ in range(2)][-1]
    assert again == deferred
    assert sk.edge_count() == P * (P - 1) // 2
    sk.close()


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
