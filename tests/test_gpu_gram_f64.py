"""The FP64 Gram at the edges of its 8 x 8 tiles, its 64-sample stages and its cluster
split (8 blocks a tile for small problems, fewer with more tiles), against NumPy FP64."""
import ctypes as C

import numpy as np
import pytest

import heterogpc as hg

pytestmark = pytest.mark.gpu


def _expect(X):
    D = X - X.mean(1, keepdims=True)
    Z = D / np.sqrt((D * D).sum(1, keepdims=True) / (X.shape[1] - 1))
    return Z @ Z.T / (X.shape[1] - 1)


def _tol(n):
    # a sum of n products of |z_a z_b|, whose total is at most n - 1 (Cauchy-Schwarz), in any
    # order: n ulps at most, on either side, plus a few for the standardisation
    return 2 * (n + 16) * 2.0 ** -52


@pytest.mark.parametrize("p", [1, 7, 8, 9, 33, 97, 140, 280])  # 280: 630 tiles, no split
@pytest.mark.parametrize("n", [4, 63, 64, 65, 511, 513])
def test_edges(p, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1000 * p + n)
    X = rng.standard_normal((p, n)) + rng.standard_normal((p, 1))
    Xd, Cd = torch.from_numpy(X).cuda(), torch.full((p, p), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    st = hg.lib().hpc_correlation_noalloc_f64(C.c_void_p(Xd.data_ptr()), n, p, 0, C.c_void_p(Cd.data_ptr()), None)
    assert st == 0
    torch.cuda.synchronize()
    got = Cd.cpu().numpy()
    assert np.array_equal(got, got.T)
    assert np.abs(got - _expect(X)).max() <= _tol(n)


def test_uneven_batch():
    ps, ns = [5, 64, 17, 33], [70, 64, 1000, 129]
    rng = np.random.default_rng(5)
    Xs = [rng.standard_normal((p, n)) for p, n in zip(ps, ns)]
    b = hg.SkeletonBatch(ps, ns, precision=hg.PREC_FP64)
    b.add_observations(b.pack(Xs, np.float64))
    out = np.empty(int(b.cor_off[-1]))
    assert hg.lib().hpc_get_correlation(b._h, C.c_void_p(out.ctypes.data)) == 0
    for k, X in enumerate(Xs):
        got = out[b.cor_off[k]:b.cor_off[k + 1]].reshape(ps[k], ps[k])
        assert np.abs(got - _expect(X)).max() <= _tol(ns[k])
    b.close()
