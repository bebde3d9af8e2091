"""The FP64 re-tests of the tensor-core mode with few items (entries cut into parts), some
(entry by entry) and many (by columns at levels 1-4): the retest margin sets how many. The
oracle's skeleton, and separation sets that re-test as independent."""
import numpy as np
import pytest

import heterogpc as hg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("margin", [1e-3, 0.05, 0.5])
@pytest.mark.parametrize("p,n,factors", [(14, 40, 2), (14, 4097, 2), (40, 515, 4)])
def test_oracle(p, n, factors, margin):
    rng = np.random.default_rng(p + n)
    F = rng.standard_normal((factors, n))
    X = (0.3 * rng.standard_normal((p, factors)) @ F + rng.standard_normal((p, n))).astype(np.float32)
    Cm = orc.correlation(X.astype(np.float64))
    top = 5 if p == 14 else 3
    want = orc.run(Cm, n, 0.05, top)
    sk = hg.SkeletonCalculator(p, n, alpha=0.05, max_level=top, precision=hg.PREC_MIXED_TC, retest_margin=margin)
    sk.add_observations(X)
    for _ in range(2):
        sk.reset()
        sk.run()
        assert np.array_equal(sk.adjacency(), want.adj)
    assert orc.verify_sepsets(Cm, n, 0.05, sk.sepset_records()).all()
    sk.close()


@pytest.mark.parametrize("entries", [None, 16])
@pytest.mark.parametrize("p,margin", [(260, 1e-3), (321, 0.05)])
def test_level_1_deferred_beside_a_matrix(p, margin, entries):
    """Mixed precision with an FP64 matrix and millions of level-1 tests: the re-tests go through the
    queue, and inline where it is too small."""
    n = 400
    rng = np.random.default_rng(p)
    X = rng.uniform(0.2, 0.9, (p, 1)) * rng.standard_normal((1, n)) + rng.standard_normal((p, n))
    Cm = orc.correlation(X)
    want = orc.run(Cm, n, 0.05, 1)
    sk = hg.SkeletonCalculator(p, n, alpha=0.05, max_level=1, retest_margin=margin)
    sk.add_correlation_matrix(Cm)
    sk.run()
    if entries:
        assert hg.lib().hpc_debug_set_retest_queue(sk.handle, entries) == 0
    for _ in range(3):  # eager (or overflowing), captured, replayed
        sk.reset()
        sk.run()
        assert np.array_equal(sk.adjacency(), want.adj)
    assert orc.verify_sepsets(Cm, n, 0.05, sk.sepset_records()).all()
    sk.close()
