"""Levels 1 and 2 on wide rows with the values that their filter must not decide on: NaN (a constant
variable, missing entries of a given matrix), |r| = 1 (copies of a variable), entries just below 1."""
import numpy as np
import pytest

import heterogpc as hg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ALPHA = 0.05


def _factor_data(p, n, seed):
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1.0, 1.0, (p, 3)) * rng.choice([0.2, 1.0], (p, 1))
    return A @ rng.standard_normal((3, n)) + rng.standard_normal((p, n))


def _run(sk, wide, levels):
    assert hg.lib().hpc_debug_set_wide(sk.handle, wide, wide) == 0
    for _ in range(2):
        sk.reset()
        sk.run()
    return sk.adjacency(), [(s["edges_after"], s["potential_tests"]) for s in sk.level_stats[-levels - 1:]]


@pytest.mark.parametrize("precision", [hg.PREC_MIXED, hg.PREC_MIXED_TC])
@pytest.mark.parametrize("p", [40, 97])
@pytest.mark.parametrize("what", ["nan", "copies", "nearly"])
def test_matrix_values(p, precision, what):
    n = 500
    Cm = orc.correlation(_factor_data(p, n, p))
    rng = np.random.default_rng(p)
    if what == "nan":  # entries and a whole variable
        for _ in range(12):
            i, j = rng.integers(0, p, 2)
            if i != j:
                Cm[i, j] = Cm[j, i] = np.nan
        Cm[7, :] = Cm[:, 7] = np.nan
        Cm[7, 7] = 1.0
    else:  # variables 3k, 3k + 1 alike, exactly or up to 1e-4
        for i in range(0, p - 1, 3):
            Cm[i + 1, :] = Cm[i, :]
            Cm[:, i + 1] = Cm[:, i]
            Cm[i, i + 1] = Cm[i + 1, i] = 1.0 if what == "copies" else 1.0 - 1e-4
            Cm[i, i] = Cm[i + 1, i + 1] = 1.0
    for levels in (1, 2):
        sk = hg.SkeletonCalculator(p, n, alpha=ALPHA, max_level=levels, precision=precision)
        sk.add_correlation_matrix(Cm)
        adj, stats = _run(sk, 1, levels)
        adj0, stats0 = _run(sk, 0, levels)
        sk.close()
        assert np.array_equal(adj, adj0) and stats == stats0
        if levels == 1:
            assert np.array_equal(adj, orc.run(Cm, n, ALPHA, 1).adj)


@pytest.mark.parametrize("precision,dtype", [(hg.PREC_MIXED, np.float64), (hg.PREC_MIXED_TC, np.float32)])
def test_constant_variables(precision, dtype):
    p, n = 70, 400
    X = _factor_data(p, n, 5).astype(dtype)
    X[[0, 31, 69]] = 1.5
    sk = hg.SkeletonCalculator(p, n, alpha=ALPHA, max_level=2, precision=precision)
    sk.add_observations(X)
    adj, stats = _run(sk, 1, 2)
    adj0, stats0 = _run(sk, 0, 2)
    sk.close()
    assert np.array_equal(adj, adj0) and stats == stats0
    assert not adj[[0, 31, 69]].any()
