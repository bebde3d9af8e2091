"""The FP64-accurate correlation by digits: the same entries whatever the split of the samples over a
cluster, and its error bound on data where one sample outweighs all others."""
import numpy as np
import pytest

import heterogpc as hg

pytestmark = pytest.mark.gpu


def _correlation(X):
    sk = hg.SkeletonCalculator(X.shape[0], X.shape[1], max_level=0)
    sk.add_observations(X)
    out = sk.correlation()
    sk.close()
    return out


def _data(p, n, heavy, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((p, n)) + 0.5 * rng.standard_normal((1, n))
    if heavy:
        X[np.arange(p), rng.integers(0, n, p)] = 1e3 * rng.choice([-1.0, 1.0], p)
    return X


@pytest.mark.parametrize("heavy", [False, True])
@pytest.mark.parametrize("n", [999, 5000, 8191])
def test_entries_do_not_depend_on_the_split(n, heavy):
    X = _data(1800, n, heavy, n)
    whole = _correlation(X)            # 120 tiles, a block each
    for p in (256, 515, 900):          # 3, 15 and 36 tiles: up to 8, 8 and 4 blocks each
        assert np.array_equal(_correlation(X[:p]), whole[:p, :p]), p


@pytest.mark.parametrize("p,n", [(257, 2000), (257, 32768), (1700, 32768)])
@pytest.mark.parametrize("heavy", [False, True])
def test_error_bound(p, n, heavy):
    X = _data(p, n, heavy, p + n)
    got = _correlation(X)
    pick = np.r_[0:40, p - 40:p]
    D = X[pick].astype(np.longdouble)
    D = D - D.mean(1, keepdims=True)
    Z = D / np.sqrt((D * D).sum(1, keepdims=True) / (n - 1))
    want = np.array([[(Z[a] * Z[b]).sum() for b in range(len(pick))] for a in range(len(pick))]) / (n - 1)
    e = np.exp2(np.floor(np.log2(np.abs(Z).max(1).astype(np.float64))) + 1)  # 2^e_v > max |z_v|
    ea, eb = e[:, None], e[None, :]
    # digits of 49 bits; dropped digit pairs, at most 6 * 2^12 of weight 2^-63 a sample (and a 2^-6th
    # of that behind them); the rounding of the sum to 2^-47; and the standardisation in FP64
    bound = 2.0 ** -50 * (ea + eb) + ea * eb * (2.0 ** -48.3 * n / (n - 1) + 2.0 ** -48 / (n - 1))
    bound += 2 * (n + 16) * 2.0 ** -52
    err = np.abs((got[np.ix_(pick, pick)] - want).astype(np.float64))
    assert (err <= bound).all()
