"""Levels 1 and 2 on the kernels for wide rows, forced on at sizes around their tiles
(32-variable words, 16-row groups, 128 second members, 256-neighbour slices, 1024-variable
chunks): the oracle's skeleton, or the ordinary kernels' where the oracle would take long."""
import numpy as np
import pytest

import heterogpc as hg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ALPHA = 0.05


def _dense(p, n, seed, missing=0.0):
    """Nearly complete graph after level 0: a few shared factors of uneven strength, some
    variables almost equal to a factor (ill-conditioned tests)."""
    rng = np.random.default_rng(seed)
    F = rng.standard_normal((3, n))
    A = rng.uniform(-1.0, 1.0, (p, 3)) * rng.choice([0.2, 1.0], (p, 1))
    noise = np.where(rng.random(p) < 0.05, 0.05, 1.0)
    X = A @ F + noise[:, None] * rng.standard_normal((p, n))
    if missing:
        X[rng.random((p, n)) < missing] = np.nan
    return X


def _run(X, precision, levels, wide):
    p, n = X.shape
    sk = hg.SkeletonCalculator(p, n, alpha=ALPHA, max_level=levels, precision=precision)
    assert hg.lib().hpc_debug_set_wide(sk.handle, wide, wide) == 0
    sk.add_observations(X)
    for _ in range(3):  # eager, captured, replayed
        sk.reset()
        sk.run()
    recs = sk.sepset_records()
    out = sk.adjacency(), [(s["edges_after"], s["potential_tests"]) for s in sk.level_stats], recs
    sk.close()
    return out


@pytest.mark.parametrize("precision", [hg.PREC_MIXED, hg.PREC_MIXED_TC])
@pytest.mark.parametrize("p", [3, 17, 33, 64, 97])
def test_against_oracle(p, precision):
    X = _dense(p, 500, p, missing=0.01 if p == 33 else 0.0)
    if precision == hg.PREC_MIXED_TC:
        X = X.astype(np.float32)
    Cm = orc.correlation(X.astype(np.float64))
    want = orc.run(Cm, X.shape[1], ALPHA, 2)
    adj, levels, recs = _run(X, precision, 2, 1)
    assert np.array_equal(adj, want.adj)
    shared = min(len(levels), len(want.levels))
    assert [e for e, _ in levels][:shared] == [lv["edges_after"] for lv in want.levels][:shared]
    assert orc.verify_sepsets(Cm, X.shape[1], ALPHA, recs).all()


@pytest.mark.parametrize("p,n,precision", [(259, 1000, hg.PREC_MIXED_TC), (300, 1500, hg.PREC_MIXED),
                                           (530, 900, hg.PREC_MIXED_TC), (1030, 700, hg.PREC_MIXED_TC)])
@pytest.mark.parametrize("dense", [False, True])
def test_against_ordinary_kernels(p, n, precision, dense):
    if dense and p > 530:
        pytest.skip("the ordinary level-2 kernel takes minutes")
    X = _dense(p, n, p) if dense else hg.sem_generate(p, n, hg.GRAPH_PA, w_lo=0.2, seed=p)
    X = X.astype(np.float32)
    adj, levels, recs = _run(X, precision, 2, 1)
    adj0, levels0, recs0 = _run(X, precision, 2, 0)
    assert np.array_equal(adj, adj0)
    assert levels == levels0
    assert {r[:3] for r in recs} == {r[:3] for r in recs0}  # the same edges, each at the same level
    Cm = orc.correlation(X.astype(np.float64))
    assert orc.verify_sepsets(Cm, n, ALPHA, recs).all()


def test_batch_of_uneven_problems():
    ps, ns = [5, 300, 40, 129], [200, 600, 400, 500]
    Xs = [_dense(p, n, p).astype(np.float32) for p, n in zip(ps, ns)]
    got = []
    for wide in (1, 0):
        b = hg.SkeletonBatch(ps, ns, [ALPHA] * 4, max_level=2)
        assert hg.lib().hpc_debug_set_wide(b._h, wide, wide) == 0
        b.add_observations(b.pack(Xs))
        for _ in range(3):  # eager, captured, replayed
            b.reset()
            b.run()
        got.append([b.adjacency(k) for k in range(4)])
        b.close()
    for a, c in zip(*got):
        assert np.array_equal(a, c)
