"""A single instance at the edge of what every block scans for itself (5,119 rows) and one row beyond it,
and at the edges of a thread's run of rows: the oracle's skeleton."""
import numpy as np
import pytest

import heterogpc as hg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [255, 256, 257, 513, 5119, 5120])
def test_oracle(p):
    n, alpha = 300, 1e-4
    X = hg.sem_generate(p, n, hg.GRAPH_ER, 6.0, 2, 0.3, 1.0, seed=p).astype(np.float32)
    want = orc.run(orc.correlation(X.astype(np.float64)), n, alpha, 4)
    for precision in (hg.PREC_MIXED_TC, hg.PREC_FP64):  # set order from level 3 on; edge order
        sk = hg.SkeletonCalculator(p, n, alpha=alpha, max_level=4, precision=precision)
        sk.add_observations(X)
        for _ in range(2):
            sk.reset()
            st = sk.run()
            assert np.array_equal(sk.adjacency(), want.adj)
        for s, lv in zip(st[-5:], want.levels):
            assert (s["level"], s["edges_after"], s["potential_tests"]) == (lv["level"], lv["edges_after"],
                                                                         lv["potential_tests"])
        sk.close()
