"""Which kernels levels 1 and 2 run, read from the tests that a level executes: on a complete graph
that loses no edge at level 1 the ordinary kernels run every test from both of its rows, the
kernel for wide rows once."""
import ctypes as C
import re

import numpy as np
import pytest

import heterogpc as hg

pytestmark = pytest.mark.gpu

# equicorrelation 1/2: 1/3 given one variable, 1/4 given two; the critical value lies between them,
# so level 1 keeps every edge and every test of level 2 removes its edge
N_OBS, ALPHA = 100, 0.0033


def _equicorrelation(p):
    return 0.5 * np.ones((p, p)) + 0.5 * np.eye(p)


def _context(p, max_level, verbose=False):
    sk = hg.SkeletonCalculator(p, N_OBS, alpha=ALPHA, max_level=max_level, verbose=verbose)
    sk.add_correlation_matrix(_equicorrelation(p))
    return sk


def _level1(sk):
    """executed / potential tests of level 1 in one more run"""
    sk.reset()
    st = sk.run()[1]
    assert st["edges_after"] == st["edges_before"] == sk.p * (sk.p - 1) // 2
    return st["executed_tests"] / st["potential_tests"]


def _set_wide(sk, l1, l2):
    assert hg.lib().hpc_debug_set_wide(sk.handle, l1, l2) == 0


def test_autotune_times_the_kernels_that_read_the_policies(capfd):
    hg.tune_clear()
    sk = _context(1200, 1, verbose=True)
    assert _level1(sk) == 0.5  # wide rows by the rule
    C.CDLL(None).fflush(None)
    capfd.readouterr()
    sk.autotune([{"tile_cap": 16, "tiles_per_lane": 4, "edge_lanes": 32, "l1_prefetch": 0},
                 {"tile_cap": 64, "tiles_per_lane": 8, "edge_lanes": 32, "l1_prefetch": 1}], reps=2)
    C.CDLL(None).fflush(None)
    runs = re.findall(r"level 1: .* tests (\d+) of (\d+)", capfd.readouterr().out)
    assert len(runs) == 4 and all(done == potential for done, potential in runs)
    assert _level1(sk) == 0.5  # and wide again after it
    sk.close()
    hg.tune_clear()


def test_autotune_leaves_the_queue_in_use():
    """The candidates' kernels run every re-test from both rows and overflow a queue that the wide level 1
    does not fill: they are timed with it off, the context keeps it."""
    p, n = 1200, 2000
    rng = np.random.default_rng(9)
    X = (rng.standard_normal((1, n)) + rng.standard_normal((p, n))).astype(np.float32)
    hg.tune_clear()
    sk = hg.SkeletonCalculator(p, n, alpha=0.05, max_level=1, precision=hg.PREC_MIXED_TC, retest_margin=4.5)
    sk.add_observations(X)
    assert _level1(sk) == 0.5
    retests = sk.level_stats[1]["retests"]
    assert retests > 100
    assert hg.lib().hpc_debug_set_retest_queue(sk.handle, retests * 3 // 2) == 0
    sk.autotune([{"tile_cap": 64, "tiles_per_lane": 4, "edge_lanes": 32, "l1_prefetch": 0}], reps=1)
    assert hg.lib().hpc_debug_set_order_active(sk.handle) == 1
    for _ in range(2):
        assert _level1(sk) == 0.5 and sk.level_stats[1]["retests"] == retests
    assert hg.lib().hpc_debug_set_order_active(sk.handle) == 1
    sk.close()
    hg.tune_clear()


def test_no_room_for_level_2_leaves_level_1_alone():
    L = hg.lib()
    sk = _context(1600, 2)
    _set_wide(sk, 0, 0)
    assert _level1(sk) == 1.0
    _set_wide(sk, -1, -1)
    live = L.hpc_debug_live_allocations()
    L.hpc_debug_fail_allocation(3)  # after level 1's snapshot and level 2's queue: level 2's scratch
    try:
        assert _level1(sk) == 0.5
    finally:
        L.hpc_debug_fail_allocation(0)
    assert sk.edge_count() == 0  # level 2 on the ordinary kernel
    assert L.hpc_debug_live_allocations() == live + 1  # the snapshot; the queue went back
    for _ in range(2):
        assert _level1(sk) == 0.5 and sk.edge_count() == 0
    assert L.hpc_debug_live_allocations() == live + 1
    sk.close()


def test_no_level_2_buffers_below_level_2():
    L = hg.lib()
    live = []
    for p in (1000, 1600):  # too few items for wide rows by the rule; enough
        base = L.hpc_debug_live_allocations()
        sk = _context(p, 1)
        sk.run()
        assert _level1(sk) == (1.0 if p == 1000 else 0.5)
        live.append(L.hpc_debug_live_allocations() - base)
        sk.close()
    assert live[1] == live[0] + 1  # level 1's snapshot


def test_executed_tests_are_those_run():
    """Every test of level 2 removes its edge, so an edge end is run by the warp that comes to it first
    (seldom by a second one at the same time): about an eighth of the tests of a row's eight warps, not
    those of every warp that once found it live."""
    p = 64
    sk = _context(p, 2)
    _set_wide(sk, 1, 1)
    sk.run()
    for _ in range(3):
        sk.reset()
        st = sk.run()[2]
        assert st["edges_before"] == p * (p - 1) // 2 and st["edges_after"] == 0
        d = p - 1
        per_warp = sum(d - a for a in range(1, 33)) / 8  # a warp's tests of one edge end, on average
        assert 0 < st["executed_tests"] <= 2 * per_warp * p * d
    sk.close()
